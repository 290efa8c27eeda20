// fma_add.cuh -- 32-bit addition on the FMA pipe.
//
// The ALU pipe (logic, shifts, additions) and the FMA pipe (multiply-adds) each
// issue 64 lanes per SM and clock.  In a hash function the logic and the
// rotates can run on the ALU pipe only, so a + b is written as a * 1 + b; the 1
// is read from constant memory, where the compiler cannot fold it back into an
// addition.
#pragma once

namespace wg {

static __constant__ unsigned FMA_ONE = 1;

__device__ __forceinline__ unsigned fma_add(unsigned a, unsigned b) {
    unsigned r;
    asm("mad.lo.u32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(FMA_ONE), "r"(b));
    return r;
}

}  // namespace wg
