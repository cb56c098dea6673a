// The block reader with a destination in host memory that refuses what a device
// may refuse: pinned memory (of every reader, of some), a reader's set-up, a copy.
#include "block_reader.h"

#include <cstdio>
#include <mutex>
#include <string>

#include <fcntl.h>

using namespace lbm;

struct Fake {
    std::string dst;
    std::atomic<int> pins{0}, pinned{0}, opens{0}, copies{0};
    int pins_allowed = 1 << 30, open_fails_from = 1 << 30, copy_fails_at = 1 << 30;
};
struct FakeLink {
    Fake* f;
    int open() { return f->opens++ >= f->open_fails_from ? 7 : 0; }
    char* pin(size_t n) {
        if (f->pins++ >= f->pins_allowed) return nullptr;
        ++f->pinned;
        return (char*)std::malloc(n);
    }
    void unpin(char* p) { --f->pinned; std::free(p); }
    int copy(int64_t at, const char* block, size_t n, int) {
        if (f->copies++ >= f->copy_fails_at) return 9;
        std::memcpy(&f->dst[(size_t)at], block, n);
        return 0;
    }
    int wait(int) { return 0; }
    void close() {}
};

static int bad = 0;
#define CHECK(x) do { if (!(x)) { std::printf("line %d: %s (size %zu)\n", __LINE__, #x, size); ++bad; } } while (0)

int main(int argc, char** argv) {
    const std::string path = std::string(argv[1]) + "/f.bin";
    for (size_t size : {size_t(1), size_t(1000), kReadBlock - 1, kReadBlock, kReadBlock + 1, 3 * kReadBlock, 9 * kReadBlock + 17}) {
        std::string text(size, 'x');
        for (size_t i = 0; i < size; ++i) text[i] = (char)(1 + (i * 2654435761u >> 7) % 250);
        FILE* fh = std::fopen(path.c_str(), "wb");
        std::fwrite(text.data(), 1, size, fh);
        std::fclose(fh);
        const int fd = open(path.c_str(), O_RDONLY);
        for (int allowed : {1 << 30, 0, 1, 2, 3}) {          // pinned blocks there are
            Fake f;
            f.dst.assign(size, 0);
            f.pins_allowed = allowed;
            ReadState R;
            read_file(fd, (int64_t)size, FakeLink{&f}, &R);
            CHECK(!R.io && !R.link && !R.nul && R.done == (int64_t)size && f.dst == text && f.pinned == 0);
        }
        {
            Fake f;                                          // a copy is refused: its status comes back
            f.dst.assign(size, 0);
            f.copy_fails_at = (int)(size / kReadBlock / 2);
            ReadState R;
            read_file(fd, (int64_t)size, FakeLink{&f}, &R);
            CHECK(R.link == 9 && f.pinned == 0);
        }
        {
            Fake f;                                          // no reader has a device
            f.dst.assign(size, 0);
            f.open_fails_from = 0;
            ReadState R;
            read_file(fd, (int64_t)size, FakeLink{&f}, &R);
            CHECK(R.closed == 7 && !R.link && R.done == 0 && f.pinned == 0);
        }
        {
            Fake f;                                          // only the first one there has
            f.dst.assign(size, 0);
            f.open_fails_from = 1;
            ReadState R;
            read_file(fd, (int64_t)size, FakeLink{&f}, &R);
            CHECK(!R.io && !R.link && R.done == (int64_t)size && f.dst == text && f.pinned == 0);
        }
        {
            Fake f;                                          // the file is shorter than it was
            f.dst.assign(size + 5, 0);
            ReadState R;
            read_file(fd, (int64_t)size + 5, FakeLink{&f}, &R);
            CHECK(R.io && f.pinned == 0);
        }
        close(fd);
    }
    {
        const size_t size = 0;                               // a directory, of whatever size it claims
        const int fd = open(argv[1], O_RDONLY);
        for (int64_t claimed : {int64_t(4096), INT64_MAX}) {
            Fake f;
            ReadState R;
            read_file(fd, claimed, FakeLink{&f}, &R);
            CHECK(R.io && R.done == 0 && f.copies == 0 && f.pinned == 0);
        }
        close(fd);
    }
    std::printf(bad ? "failed\n" : "block reader ok\n");
    return bad ? 1 : 0;
}
