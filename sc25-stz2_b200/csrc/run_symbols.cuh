// Decomposition of a run of centre codes into run symbols (device code).
#pragma once
#include <cstdint>

#include <cuda_runtime.h>

#include "stz_internal.h"

namespace stz {

// Symbols of a run of r centre codes (none for r = 0), in order: while
// r > D, 2^k (the largest power of two <= r, k <= J) when k > LD, else D
// codes; then the symbol of the remaining 2..D codes, or the centre code.
template <class F>
__device__ __forceinline__ void run_symbols(uint32_t r, uint32_t R, uint32_t base, uint32_t J, uint32_t D, uint32_t LD,
                                            F&& f)
{
    while (r > D) {
        const uint32_t k = min((uint32_t)(31 - __clz(r)), J);
        if (k > LD) {
            f(base + D - 1 + (k - LD - 1));
            r -= 1u << k;
        } else {
            f(base + D - 2);
            r -= D;
        }
    }
    if (r >= 2) f(base + r - 2);
    else if (r) f(R);
}

}  // namespace stz
