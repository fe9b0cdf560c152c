// gl_w.h -- multiplication by the Fp3 non-residue W without a general product.
//
// F64Ext3 is Fp[X]/(X^3 - W) with W = 0xFFFFFFF800000001 = 2^64 - 2^35 + 1
// (the crate's from_raw(7): 7 * 2^-64 mod p).  Since 2^64 = 2^32 - 1 (mod p),
// W = 2^32 - 1 - 2^35 + 1 = -7 * 2^32 (mod p), so W x needs no 64 x 64
// product.  With x = x0 + x1 2^32 and 2^64 = 2^32 - 1:
//   x 2^32 = (x0 + x1) 2^32 - x1
//   7 (x0 + x1) = sl + sh 2^32                       (sh < 16)
//   7 (x0 + x1) 2^32 = (sl + sh) 2^32 - sh           (2^64 = 2^32 - 1)
//   sl + sh = t + c 2^32, (sl + sh) 2^32 = (t + c) 2^32 - c
//   W x = (7 x1 + sh + c) - (t + c) 2^32 = A - T 2^32
// with A < 2^36 and T < 2^32, so A - T 2^32 lies in (-p, p): one subtraction
// with p added on a borrow is the canonical residue, for any 64-bit x.
// Three multiply-adds and nine adds, half of what the shift form (8x - x, two
// folds, a compare) takes.
// Plain C, shared by the kernels and the host tests.
#pragma once
#include <stdint.h>

#if defined(__CUDACC__)
#define GLW_FN __host__ __device__ __forceinline__
#else
#define GLW_FN static inline
#endif

// W x = *a - (*t << 32) mod p.
GLW_FN void gl_mul_w_parts(uint64_t x, uint64_t* a, uint32_t* t) {
    const uint32_t x0 = (uint32_t)x, x1 = (uint32_t)(x >> 32);
    const uint64_t b = 7 * ((uint64_t)x0 + x1);
    const uint32_t sh = (uint32_t)(b >> 32);
    const uint64_t u = (uint64_t)(uint32_t)b + sh;
    const uint32_t c = (uint32_t)(u >> 32);
    *t = (uint32_t)u + c;
    *a = 7 * (uint64_t)x1 + (sh + c);
}

#if !defined(__CUDACC__)
GLW_FN uint64_t gl_mul_w(uint64_t x) {
    uint64_t a;
    uint32_t t;
    gl_mul_w_parts(x, &a, &t);
    const uint64_t b = (uint64_t)t << 32;
    return a >= b ? a - b : a - b + 0xFFFFFFFF00000001ULL;
}
#endif
