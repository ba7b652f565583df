// Products of floats on the tensor cores: a float is the sum of three bfloat16 parts (24 bits), and six of the nine products of two
// floats' parts are taken; the other three lie below a float's last bit.  The leading product has an accumulator of its own, so
// that the roundings of the others' sums count 2^-8 of it.  The tensor cores cut a sum's last bits off instead of rounding it, which over
// many steps draws an accumulator towards zero (measured: 1.4e-7 of a state over four steps of 16).  So long sums start the leading
// product of every step from zero and add it with an addition that rounds (parts_mma6_round: 4 additions to 6 products); a few
// steps accumulate (parts_mma6).  mma.sync m16n8k16 runs at 550 TFLOP/s here (measured), a float product so at 92, against 74 for the
// pairs of float multiply-adds, and takes a fraction of their operands from shared memory.
#pragma once
#include "common.cuh"

// The three bfloat16 parts of two floats, packed (the first in the low half).
__device__ __forceinline__ void parts_cut(float a, float b, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
    auto pack = [](float x, float y) {
        const __nv_bfloat162 v = __floats2bfloat162_rn(x, y);
        return *reinterpret_cast<const uint32_t*>(&v);
    };
    hi = pack(a, b);
    a -= __uint_as_float(hi << 16); b -= __uint_as_float(hi & 0xffff0000u);
    mid = pack(a, b);
    a -= __uint_as_float(mid << 16); b -= __uint_as_float(mid & 0xffff0000u);
    lo = pack(a, b);
}

__device__ __forceinline__ void parts_mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// c += the product, which starts from zero
__device__ __forceinline__ void parts_mma_add(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    float d[4];
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
#pragma unroll
    for (int x = 0; x < 4; ++x) c[x] += d[x];
}
__device__ __forceinline__ void parts_load4(uint32_t (&r)[4], uint32_t at) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(at));
}
__device__ __forceinline__ void parts_load4_trans(uint32_t (&r)[4], uint32_t at) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(at));
}
// s += the products of parts but the leading one, over the parts a[3], b of the fragment pair starting at b[.][i]
__device__ __forceinline__ void parts_mma5(float (&s)[4], const uint32_t (&a)[3][4], const uint32_t (&b)[3][4], int i) {
    parts_mma(s, a[2], b[0][i], b[0][i + 1]);
    parts_mma(s, a[0], b[2][i], b[2][i + 1]);
    parts_mma(s, a[1], b[1][i], b[1][i + 1]);
    parts_mma(s, a[1], b[0][i], b[0][i + 1]);
    parts_mma(s, a[0], b[1][i], b[1][i + 1]);
}
// c (leading parts) and s (the rest) += A B
__device__ __forceinline__ void parts_mma6(float (&c)[4], float (&s)[4], const uint32_t (&a)[3][4], const uint32_t (&b)[3][4], int i) {
    parts_mma(c, a[0], b[0][i], b[0][i + 1]);
    parts_mma5(s, a, b, i);
}
__device__ __forceinline__ void parts_mma6_round(float (&c)[4], float (&s)[4], const uint32_t (&a)[3][4], const uint32_t (&b)[3][4], int i) {
    parts_mma_add(c, a[0], b[0][i], b[0][i + 1]);
    parts_mma5(s, a, b, i);
}
