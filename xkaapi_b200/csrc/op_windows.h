// Ops of a batch, numbered by ints on the device: how many a batch may have, and the windows in which
// the resolver's bitmap sort passes over them. Plain C++, compiled by the CPU tests too.
#pragma once
#include <climits>
#include <cstdint>

#ifdef __CUDACC__
#define XKB_HD __host__ __device__ __forceinline__
#else
#define XKB_HD inline
#endif

namespace xkb {

// Ops of one domain in one batch at most: their indices stay inside an int, with room for the step past
// the end that a loop over them by all threads of a grid takes.
constexpr uint64_t RESOLVE_MAX_OPS = (uint64_t) INT_MAX - (1u << 20);

// The ops [first, last) of a window; `words` words of 32 ops each, the last window cut at nops.
struct OpWindow {
    int first, last;
    // the window after one that ends at `at` (0: the first); none is left when at == nops
    static XKB_HD OpWindow from(int at, int words, int nops)
    {
        const int room = nops - at;                        // (no sum of `at` and a window may pass INT_MAX)
        return OpWindow{at, room / 32 < words ? nops : at + words * 32};
    }
    XKB_HD bool holds(int op) const { return op >= first && op < last; }
};

} // namespace xkb
