// 32-bit products on the tensor cores.
//
// A number is a sum of two that the tensor cores take (11 bits each; the second, of at most 12, loses its last one), and a product three of
// theirs: what is left out is 2^-21 of it at most (the product of both second parts and the two last bits), 2^-24 in the mean.  So a single product is further off than one
// multiply-add, which rounds it by 2^-24.  Sums of 16 products go through the tensor cores, which cut off what does not fit
// where the 32-bit adders round, and are added in those; the products with second parts go first, so that little is cut off.  Against 64 bits
// a chain of 64 or 128 such multiply-adds is no further off than one of the FMA pipe's, unless its terms grow towards its end.
// (Three parts of 8 bits and six products are exact and take the tensor cores as long, but more instructions: the same error, the delta
// rule's chain 104 us with them and 83 so.  The conversion instruction for these formats runs at an eighth of the adders' rate: 142 us.)
#pragma once
#include "common.cuh"

namespace {

struct Two {
    unsigned hi, lo;
};
__device__ __forceinline__ unsigned long long packed(float x, float y) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
    return r;
}
__device__ __forceinline__ unsigned nearest(float x) { return (__float_as_uint(x) + 0x1000u) & 0xFFFFE000u; }
// (the tensor cores ignore the last 13 bits; what is no number stays in the second part)
__device__ __forceinline__ void two(float x, float y, Two& a, Two& b) {
    a.hi = nearest(x);
    b.hi = nearest(y);
    unsigned long long d;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(packed(x, y)), "l"(packed(__uint_as_float(a.hi), __uint_as_float(b.hi))));
    asm("mov.b64 {%0, %1}, %2;" : "=r"(a.lo), "=r"(b.lo) : "l"(d));
}
// (one number: where the parts of a pair do not become neighbouring registers, moving them costs more than the second subtraction)
__device__ __forceinline__ Two apart(float x) {
    Two r;
    r.hi = nearest(x);
    r.lo = __float_as_uint(x - __uint_as_float(r.hi));
    return r;
}
__device__ __forceinline__ void add_to(float (&acc)[4], const float (&c)[4]) {
#pragma unroll
    for (int i = 0; i < 4; i += 2) {
        unsigned long long d;
        asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(packed(acc[i], acc[i + 1])), "l"(packed(c[i], c[i + 1])));
        asm("mov.b64 {%0, %1}, %2;" : "=f"(acc[i]), "=f"(acc[i + 1]) : "l"(d));
    }
}
// c = a b (first) or c += a b.  a: (row g, k t'), (g + 8, t'), (g, t''), (g + 8, t'') with g = lane / 4; b: (k t', column g), (t'', g): t' and t'' are
// the lane's two k of eight, the same for both.
__device__ __forceinline__ void mma8(float (&c)[4], bool first, unsigned a0, unsigned a1, unsigned a2, unsigned a3, unsigned b0, unsigned b1) {
    if (first)
        asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
            : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
    else
        asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
            : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// c = a b over 16 of k, eights of it in a[0], b[0] and a[1], b[1]: the i-th of six products
__device__ __forceinline__ void mma6_part(float (&c)[4], int i, const Two (&a)[2][4], const Two (&b)[2][2]) {
    const int h = i < 4 ? i >> 1 : i - 4;
    if (i == 0 || i == 2) mma8(c, i == 0, a[h][0].lo, a[h][1].lo, a[h][2].lo, a[h][3].lo, b[h][0].hi, b[h][1].hi);
    else if (i < 4) mma8(c, false, a[h][0].hi, a[h][1].hi, a[h][2].hi, a[h][3].hi, b[h][0].lo, b[h][1].lo);
    else mma8(c, false, a[h][0].hi, a[h][1].hi, a[h][2].hi, a[h][3].hi, b[h][0].hi, b[h][1].hi);
}
__device__ __forceinline__ void mma6(float (&c)[4], const Two (&a)[2][4], const Two (&b)[2][2]) {
#pragma unroll
    for (int i = 0; i < 6; ++i) mma6_part(c, i, a, b);
}

}  // namespace
