// Launchers of the step kernel instantiations (internal).  One translation
// unit per storage format so they compile in parallel; the FP64 one is built
// with -fmad=false.
#pragma once
#include <cuda_runtime.h>

#include "device.cuh"
#include "internal.h"
#include "launch_plan.h"

namespace lbm {

struct Partials;

// LaunchPlans::blocks for kernel `k` on the current device; `twin` (or null) is
// launched by the same plans.  Fails where no block fits on an SM.
inline lbm_status resident_blocks(LaunchPlans& plans, const void* k, const void* twin, int wpb, size_t smem, int* blocks) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess || dev < 0 || dev >= LaunchPlans::kDevices)
        return fail(LBM_ERR_CUDA, "step kernel: device %d not supported", dev);
    const int n = plans.blocks(
        dev, wpb, smem,
        [&](size_t bytes) {
            e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
            if (e == cudaSuccess && twin)
                e = cudaFuncSetAttribute(twin, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
            return e == cudaSuccess;
        },
        [&] {
            int per_sm = 0, sms = 0;
            e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, 32 * wpb, smem);
            if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
            return e == cudaSuccess ? per_sm * sms : 0;
        });
    if (n < 1) {
        cudaGetLastError();
        return fail(LBM_ERR_CUDA, "step kernel, %d warps a block, %zu B shared: %s", wpb, smem,
                    e != cudaSuccess ? cudaGetErrorString(e) : "does not fit on an SM");
    }
    *blocks = n;
    return LBM_OK;
}

lbm_status launch_step_f64(int Q, int mode, bool dry, int ra, const StepArgs& a, const Partials& p, int wpb,
                           cudaStream_t st);
lbm_status launch_step_f32(int Q, int mode, bool dry, int ra, const StepArgs& a, const Partials& p, int wpb,
                           cudaStream_t st);
lbm_status launch_step_f16s(int Q, int mode, bool dry, int ra, const StepArgs& a, const Partials& p, int wpb,
                            cudaStream_t st);
lbm_status launch_step_bf16s(int Q, int mode, bool dry, int ra, const StepArgs& a, const Partials& p, int wpb,
                             cudaStream_t st);

// TMA-staged pipeline (non-dry launches only); err receives 1 if a bounded wait gave up.
lbm_status launch_tma_f64(int Q, int mode, int ra, const StepArgs& a, int32_t* err, int wpb, cudaStream_t st);
lbm_status launch_tma_f32(int Q, int mode, int ra, const StepArgs& a, int32_t* err, int wpb, cudaStream_t st);
lbm_status launch_tma_f16s(int Q, int mode, int ra, const StepArgs& a, int32_t* err, int wpb, cudaStream_t st);
lbm_status launch_tma_bf16s(int Q, int mode, int ra, const StepArgs& a, int32_t* err, int wpb, cudaStream_t st);

// Paired kernel (two adjacent nodes per lane; non-dry launches, FP32 and
// 16-bit storage); a.chunks must be the paired chunk table.
lbm_status launch_pair_f32(int Q, int mode, int ra, const StepArgs& a, int wpb, cudaStream_t st);
lbm_status launch_pair_f16s(int Q, int mode, int ra, const StepArgs& a, int wpb, cudaStream_t st);
lbm_status launch_pair_bf16s(int Q, int mode, int ra, const StepArgs& a, int wpb, cudaStream_t st);

// Wall shear stress of every wall lane (one-node-per-lane chunk table):
// wss[out_pos] = |mu grad u| from the node velocities u (3 per output
// position); wall_flag[out_pos] = 1 when wall_flag is not null.
lbm_status launch_wss(int Q, int ra, const Chunk* chunks, int64_t nchunks, const uint32_t* mmask,
                      const int32_t* out_pos, const InstParam* insts, const double* u, double* wss,
                      uint8_t* wall_flag, cudaStream_t st);

}  // namespace lbm
