// Reads a file in blocks on several threads, each block copied on while the next
// is read.  Each reader has two blocks of pinned memory, or of ordinary memory
// where pinning is refused (the copies are slower then, the result is the same); a
// reader that can have neither, or cannot open its link, leaves the blocks to the
// others.
//
// Link is one reader's way to the destination; a status of 0 is success:
//   int open()                                   before the first block
//   char* pin(size_t n), void unpin(char*)       pinned memory, or null
//   int copy(int64_t at, const char* block, size_t n, int b)   starts copying block b
//   int wait(int b)                              the copy from block b has left it
//   void close()
#pragma once
#include <algorithm>
#include <atomic>
#include <cerrno>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <thread>
#include <vector>

#include <unistd.h>

namespace lbm {

// (52 MB file: pinning a buffer of its size, one read and one copy took 8.9 of the
// reader's 10.2 ms; with blocks the whole call takes 2.9 ms)
constexpr int kReaders = 4;
constexpr size_t kReadBlock = size_t(1) << 19;

struct ReadState {
    std::atomic<int64_t> next{0}, done{0};     // bytes claimed, bytes handed to a copy
    std::atomic<int> io{0}, link{0}, nul{0};   // short read; status of a failed copy; a NUL byte was seen
    std::atomic<int> closed{0};                // status of a link that did not open
};

template <class Link>
void read_blocks(int fd, int64_t L, Link link, ReadState* R) {
    const size_t size = std::min<size_t>(kReadBlock, (size_t)L);
    char* block[2] = {nullptr, nullptr};
    bool pinned[2] = {false, false}, used[2] = {false, false};
    const int opened = link.open();
    if (opened != 0) R->closed = opened;
    int e = 0;
    for (int b = 0; b < 2 && opened == 0; ++b) {
        block[b] = link.pin(size);
        pinned[b] = block[b] != nullptr;
        if (!block[b]) block[b] = (char*)std::malloc(size);
    }
    for (int b = 0; e == 0 && block[0] && block[1] && !R->io && !R->link; b ^= 1) {
        const int64_t off = R->next.fetch_add((int64_t)kReadBlock);
        if (off >= L) break;
        const size_t n = (size_t)std::min<int64_t>((int64_t)kReadBlock, L - off);
        if (used[b] && (e = link.wait(b)) != 0) break;
        size_t got = 0;
        while (got < n) {
            const ssize_t k = pread(fd, block[b] + got, n - got, (off_t)(off + (int64_t)got));
            if (k < 0 && errno == EINTR) continue;
            if (k <= 0) break;
            got += (size_t)k;
        }
        if (got != n) { R->io = 1; break; }
        if (std::memchr(block[b], 0, n)) R->nul = 1;
        e = link.copy(off, block[b], n, b);
        used[b] = true;
        R->done += (int64_t)n;
    }
    if (e != 0) R->link = e;
    for (int b = 0; b < 2; ++b) {
        if (used[b]) link.wait(b);
        if (pinned[b]) link.unpin(block[b]);
        else std::free(block[b]);
    }
    link.close();
}

// The whole file through up to kReaders readers, each with its own copy of link;
// every byte has been handed on when R->done is L.
template <class Link>
void read_file(int fd, int64_t L, const Link& link, ReadState* R) {
    const int n = (int)std::min<int64_t>(kReaders, (L - 1) / (int64_t)kReadBlock + 1);
    std::vector<std::thread> th;
    th.reserve(kReaders);                  // (no growth with a running thread in it)
    for (int i = 1; i < n; ++i) {
        try {
            th.emplace_back(read_blocks<Link>, fd, L, link, R);
        } catch (...) {
            break;                         // fewer readers, the same result
        }
    }
    read_blocks<Link>(fd, L, link, R);
    for (std::thread& t : th) t.join();
}

}  // namespace lbm
