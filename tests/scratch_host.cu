// The run buffers of csrc/scratch.hpp over a counting allocator that hands out
// addresses and no memory.
#include "../3dalm_b200/csrc/scratch.hpp"

namespace {
size_t held, peak, calls;
char *at;
struct Counter {
    static void *allocate(size_t bytes) {
        held += bytes;
        peak = held > peak ? held : peak;
        calls++;
        void *p = at;
        at += (bytes + (1 << 20)) / 512 * 512;
        return p;
    }
    static void release(void *) { calls--; }
};
}  // namespace

// n buffers of `bytes` with a small one after every `every`-th: addresses to
// `out`, bytes allocated in all returned, *most allocations; *open: allocations
// still held at the end
extern "C" long long scratch_run(long long bytes, int n, int every, long long *out,
                                 long long *most, long long *open) {
    held = peak = calls = 0;
    at = (char *)(1 << 20);
    {
        dalm::Scratch<Counter> S((size_t)n, (size_t)bytes);
        for (int q = 0; q < n; q++) {
            out[q] = (long long)S.get<char>((size_t)bytes);
            if (every && q % every == 0) S.get<double>(3);
        }
        *most = (long long)calls;
    }
    *open = (long long)calls;
    return (long long)peak;
}
