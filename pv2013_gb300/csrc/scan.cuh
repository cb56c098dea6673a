// Order-preserving prefix sums and stream compaction (hand-written, three
// passes: per-tile totals, a single-block scan of the totals, per-tile
// rescan and write).  Used by the set-up kernels: boundary-point lists,
// node numbering, run-table construction.  Tiles are 256 threads x 16 items.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#include "internal.h"

namespace lbm {
namespace scan {

constexpr int kThreads = 256;
constexpr int kItems = 16;
constexpr int64_t kTile = (int64_t)kThreads * kItems;

__device__ __forceinline__ int64_t warp_incl_scan(int64_t v) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        int64_t t = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += t;
    }
    return v;
}

// Exclusive block scan of one value per thread; returns the exclusive prefix
// and writes the block total to *total (all threads).
__device__ __forceinline__ int64_t block_excl_scan(int64_t v, int64_t* total) {
    __shared__ int64_t warp_sums[kThreads / 32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    int64_t inc = warp_incl_scan(v);
    if (lane == 31) warp_sums[wid] = inc;
    __syncthreads();
    if (wid == 0) {
        int64_t s = lane < kThreads / 32 ? warp_sums[lane] : 0;
        s = warp_incl_scan(s);
        if (lane < kThreads / 32) warp_sums[lane] = s;
    }
    __syncthreads();
    int64_t before = wid > 0 ? warp_sums[wid - 1] : 0;
    *total = warp_sums[kThreads / 32 - 1];
    __syncthreads();
    return before + inc - v;
}

// Nonzero mask of a thread's kItems bytes at base: one 16-byte load where the
// tile is whole (268 MB of flags counted in 73 us, 149 us with 16 byte loads a thread).
static_assert(kItems == 16, "a thread's bytes are one 16-byte word");
__device__ __forceinline__ uint32_t nonzero_bits(const uint8_t* __restrict__ in, int64_t base, int64_t n) {
    uint32_t bits = 0;
    if (base + kItems <= n) {
        const uint4 q = *reinterpret_cast<const uint4*>(in + base);
        const uint32_t w[4] = {q.x, q.y, q.z, q.w};
        if ((q.x | q.y | q.z | q.w) == 0u) return 0u;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            // 0x01 per nonzero byte, gathered into four bits
            const uint32_t m = __vcmpne4(w[i], 0u) & 0x01010101u;
            bits |= ((m * 0x10204080u) >> 28) << (4 * i);
        }
        return bits;
    }
    for (int i = 0; i < kItems; ++i)
        if (base + i < n && in[base + i] != 0) bits |= 1u << i;
    return bits;
}

template <class T>
__global__ void tile_totals(const T* __restrict__ in, int64_t n, int64_t* __restrict__ tile_sum, bool nonzero) {
    int64_t base = blockIdx.x * kTile + (int64_t)threadIdx.x * kItems;
    int64_t s = 0;
    bool done = false;
    if constexpr (sizeof(T) == 1) {                  // (bytes: device allocations, base a multiple of 16)
        if (nonzero) {
            s = __popc(nonzero_bits(reinterpret_cast<const uint8_t*>(in), base, n));
            done = true;
        }
    }
    if (!done) {
#pragma unroll
        for (int i = 0; i < kItems; ++i) {
            int64_t idx = base + i;
            if (idx < n) s += nonzero ? (in[idx] != 0 ? 1 : 0) : (int64_t)in[idx];
        }
    }
    int64_t tot;
    block_excl_scan(s, &tot);
    if (threadIdx.x == 0) tile_sum[blockIdx.x] = tot;
}

// Single block: exclusive scan of ntiles totals in place; grand total to *total.
static __global__ void scan_totals(int64_t* __restrict__ tile_sum, int64_t ntiles, int64_t* __restrict__ total) {
    int64_t per = (ntiles + kThreads - 1) / kThreads;
    int64_t b = threadIdx.x * per, e = min(ntiles, b + per);
    int64_t s = 0;
    for (int64_t i = b; i < e; ++i) s += tile_sum[i];
    int64_t tot;
    int64_t off = block_excl_scan(s, &tot);
    for (int64_t i = b; i < e; ++i) {
        int64_t v = tile_sum[i];
        tile_sum[i] = off;
        off += v;
    }
    if (threadIdx.x == 0) *total = tot;
}

// Exclusive scan of counts into out.
template <class T, class O>
__global__ void tile_scan_write(const T* __restrict__ in, int64_t n, const int64_t* __restrict__ tile_off,
                                O* __restrict__ out) {
    int64_t base = blockIdx.x * kTile + (int64_t)threadIdx.x * kItems;
    int64_t v[kItems];
    int64_t s = 0;
#pragma unroll
    for (int i = 0; i < kItems; ++i) {
        int64_t idx = base + i;
        v[i] = idx < n ? (int64_t)in[idx] : 0;
        s += v[i];
    }
    int64_t tot;
    int64_t off = block_excl_scan(s, &tot) + tile_off[blockIdx.x];
#pragma unroll
    for (int i = 0; i < kItems; ++i) {
        int64_t idx = base + i;
        if (idx < n) out[idx] = (O)off;
        off += v[i];
    }
}

// Writes the indices of nonzero entries, in order.
template <class T>
__global__ void tile_compact_write(const T* __restrict__ in, int64_t n, const int64_t* __restrict__ tile_off,
                                   int64_t* __restrict__ out) {
    int64_t base = blockIdx.x * kTile + (int64_t)threadIdx.x * kItems;
    uint32_t bits = 0;
    if constexpr (sizeof(T) == 1) {
        bits = nonzero_bits(reinterpret_cast<const uint8_t*>(in), base, n);
    } else {
#pragma unroll
        for (int i = 0; i < kItems; ++i) {
            int64_t idx = base + i;
            if (idx < n && in[idx] != 0) bits |= 1u << i;
        }
    }
    const int64_t s = __popc(bits);
    int64_t tot;
    int64_t off = block_excl_scan(s, &tot) + tile_off[blockIdx.x];
#pragma unroll
    for (int i = 0; i < kItems; ++i)
        if (bits & (1u << i)) out[off++] = base + i;
}

// Set bits of words: totals per tile, and the exclusive prefix of each word.
__device__ __forceinline__ int load_words(const uint32_t* __restrict__ in, int64_t base, int64_t n, uint32_t* v) {
    int s = 0;
    if (base + kItems <= n) {
#pragma unroll
        for (int i = 0; i < kItems; i += 4) {
            const uint4 q = *reinterpret_cast<const uint4*>(in + base + i);
            v[i] = q.x; v[i + 1] = q.y; v[i + 2] = q.z; v[i + 3] = q.w;
        }
    } else {
#pragma unroll
        for (int i = 0; i < kItems; ++i) v[i] = base + i < n ? in[base + i] : 0u;
    }
#pragma unroll
    for (int i = 0; i < kItems; ++i) s += __popc(v[i]);
    return s;
}
static __global__ void word_totals(const uint32_t* __restrict__ in, int64_t n, int64_t* __restrict__ tile_sum) {
    uint32_t v[kItems];
    const int s = load_words(in, blockIdx.x * kTile + (int64_t)threadIdx.x * kItems, n, v);
    int64_t tot;
    block_excl_scan(s, &tot);
    if (threadIdx.x == 0) tile_sum[blockIdx.x] = tot;
}
static __global__ void word_prefix(const uint32_t* __restrict__ in, int64_t n, const int64_t* __restrict__ tile_off,
                                   uint32_t* __restrict__ out) {
    const int64_t base = blockIdx.x * kTile + (int64_t)threadIdx.x * kItems;
    uint32_t v[kItems];
    const int s = load_words(in, base, n, v);
    int64_t tot;
    uint32_t off = (uint32_t)(block_excl_scan(s, &tot) + tile_off[blockIdx.x]);
#pragma unroll
    for (int i = 0; i < kItems; ++i) {
        if (base + i < n) out[base + i] = off;
        off += __popc(v[i]);
    }
}

// Workspace for one scan of n elements.
struct Workspace {
    int64_t* tiles = nullptr;
    int64_t* total = nullptr;
    int64_t ntiles = 0;
    cudaStream_t st = 0;
};

#define LBM_SCAN_TRY(x)                 \
    do {                                \
        lbm_status s_ = (x);            \
        if (s_ != LBM_OK) return s_;    \
    } while (0)

inline lbm_status ws_alloc(Workspace& w, int64_t n, cudaStream_t st) {
    w.ntiles = (n + kTile - 1) / kTile;
    if (w.ntiles < 1) w.ntiles = 1;
    LBM_SCAN_TRY(dev_alloc(reinterpret_cast<void**>(&w.tiles), sizeof(int64_t) * (w.ntiles + 1), st, "scan workspace"));
    w.total = w.tiles + w.ntiles;
    w.st = st;
    return LBM_OK;
}
inline void ws_free(Workspace& w) {
    if (w.tiles) dev_free(w.tiles, w.st);
    w.tiles = nullptr;
}

// Exclusive scan of n counts; *h_total receives the sum (synchronises stream).
template <class T, class O>
lbm_status exclusive_scan(const T* d_in, int64_t n, O* d_out, int64_t* h_total, cudaStream_t st) {
    Workspace w;
    lbm_status s = ws_alloc(w, n, st);
    if (s != LBM_OK) return s;
    tile_totals<T><<<(unsigned)w.ntiles, kThreads, 0, st>>>(d_in, n, w.tiles, false);
    scan_totals<<<1, kThreads, 0, st>>>(w.tiles, w.ntiles, w.total);
    tile_scan_write<T, O><<<(unsigned)w.ntiles, kThreads, 0, st>>>(d_in, n, w.tiles, d_out);
    cudaError_t e = cudaMemcpyAsync(h_total, w.total, sizeof(int64_t), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    ws_free(w);
    if (e != cudaSuccess) return fail(LBM_ERR_CUDA, "exclusive_scan: %s", cudaGetErrorString(e));
    return LBM_OK;
}

// Set bits of n words (synchronises), and their exclusive prefix per word where
// d_prefix is not null (valid when the total fits 32 bits).
inline lbm_status bit_ranks(const uint32_t* d_in, int64_t n, uint32_t* d_prefix, int64_t* h_total, cudaStream_t st) {
    Workspace w;
    lbm_status s = ws_alloc(w, n, st);
    if (s != LBM_OK) return s;
    word_totals<<<(unsigned)w.ntiles, kThreads, 0, st>>>(d_in, n, w.tiles);
    scan_totals<<<1, kThreads, 0, st>>>(w.tiles, w.ntiles, w.total);
    if (d_prefix) word_prefix<<<(unsigned)w.ntiles, kThreads, 0, st>>>(d_in, n, w.tiles, d_prefix);
    cudaError_t e = cudaMemcpyAsync(h_total, w.total, sizeof(int64_t), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    ws_free(w);
    if (e != cudaSuccess) return fail(LBM_ERR_CUDA, "bit_ranks: %s", cudaGetErrorString(e));
    return LBM_OK;
}

// Ordered indices of nonzero entries into *d_out (allocated here from the
// stream-ordered pool on st, count in *h_count).
template <class T>
lbm_status compact(const T* d_in, int64_t n, int64_t** d_out, int64_t* h_count, cudaStream_t st) {
    Workspace w;
    lbm_status s = ws_alloc(w, n, st);
    if (s != LBM_OK) return s;
    tile_totals<T><<<(unsigned)w.ntiles, kThreads, 0, st>>>(d_in, n, w.tiles, true);
    scan_totals<<<1, kThreads, 0, st>>>(w.tiles, w.ntiles, w.total);
    cudaError_t e = cudaMemcpyAsync(h_count, w.total, sizeof(int64_t), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) { ws_free(w); return fail(LBM_ERR_CUDA, "compact: %s", cudaGetErrorString(e)); }
    s = dev_alloc(reinterpret_cast<void**>(d_out), sizeof(int64_t) * (*h_count > 0 ? *h_count : 1), st, "compacted indices");
    if (s != LBM_OK) { ws_free(w); return s; }
    tile_compact_write<T><<<(unsigned)w.ntiles, kThreads, 0, st>>>(d_in, n, w.tiles, *d_out);
    e = cudaStreamSynchronize(st);
    ws_free(w);
    if (e != cudaSuccess) return fail(LBM_ERR_CUDA, "compact: %s", cudaGetErrorString(e));
    return LBM_OK;
}

}  // namespace scan
}  // namespace lbm
