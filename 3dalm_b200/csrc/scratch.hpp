// Buffers of one run, cut from few allocations and freed together.
#pragma once

#include <algorithm>
#include <cstddef>
#include <vector>

namespace dalm {

// Mem: allocate(bytes) and release(pointer), static.  Buffers of up to
// OWN_BYTES are cut one after the other from chunks of `chunk` bytes; what is
// left of a chunk when the next buffer does not fit is lost, at most a
// sixteenth of the 256 MB that a chunk has at most.  Larger buffers are
// allocations of their own: a call takes some tens of microseconds, which a
// run on such a grid does not feel, while two of them seldom fill a chunk.
template <typename Mem>
class Scratch {
  public:
    static constexpr size_t CHUNK_BYTES = 256u << 20, OWN_BYTES = 16u << 20;

    // n buffers of `bytes` each, and up to a megabyte of smaller ones
    Scratch(size_t n, size_t bytes)
        : chunk(std::min((bytes > OWN_BYTES ? 0 : n * bytes) + (1u << 20), CHUNK_BYTES)) {}
    Scratch(const Scratch &) = delete;
    Scratch &operator=(const Scratch &) = delete;
    ~Scratch() {
        for (void *p : ptrs) Mem::release(p);
    }
    template <typename T>
    T *get(size_t n) {
        const size_t bytes = (std::max<size_t>(n, 1) * sizeof(T) + 255) / 256 * 256;
        if (bytes > OWN_BYTES) return (T *)add(bytes);
        if (bytes > left) {
            left = std::max(chunk, bytes);
            next = (char *)add(left);
        }
        T *r = (T *)next;
        next += bytes;
        left -= bytes;
        return r;
    }

  private:
    void *add(size_t bytes) {
        ptrs.push_back(nullptr);  // (first, so that no allocation is lost to a failing push)
        return ptrs.back() = Mem::allocate(bytes);
    }
    size_t chunk, left = 0;
    char *next = nullptr;
    std::vector<void *> ptrs;
};

}  // namespace dalm
