// float32 as the exact sum of three bfloat16 values, for float32 products on the tensor cores (the scheme of Henry, Tang and Heinecke,
// "Leveraging the bfloat16 artificial intelligence datatype for higher-precision computations", 2019).
//
// x = h + m + l: h is x rounded to bfloat16, m what is left rounded, l the rest, which bfloat16 holds exactly (24 bits are 8 and two
// times 8 with a sign; below 2^-110 the last bits of l go).  Of the nine products of two such sums the six largest are taken, h h', h m',
// m h', m m', h l', l h'; the other three are at most 2^-26 of x x' together, less than one rounding of a float32 product.  (Cut
// instead of rounded, the parts leave out up to 2^-21, always to the same side: a product of 2,048 elements was off by 2.0e-7 instead of
// 1.3e-7.)  Where one side holds bfloat16 values (its m and l are zero) three products are exact.  An infinity, a NaN or what rounds
// to an infinity leaves a NaN in m: a caller that must tell them apart looks at the result.
#pragma once
#include "common.cuh"

struct TqSplit4 { uint2 h, m, l; };      // four neighbours: bfloat16 pairs (first in the low half)

// two neighbours rounded to a bfloat16 pair, and what is left of them
__device__ __forceinline__ uint32_t tq_part2(float& a, float& b) {
    uint32_t p;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(p) : "f"(b), "f"(a));
    a -= __uint_as_float(p << 16);
    b -= __uint_as_float(p & 0xffff0000u);
    return p;
}
__device__ __forceinline__ void tq_split2(float a, float b, uint32_t& h, uint32_t& m, uint32_t& l) {
    h = tq_part2(a, b);
    m = tq_part2(a, b);
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(l) : "f"(b), "f"(a));
}
__device__ __forceinline__ TqSplit4 tq_split4(float4 v) {
    TqSplit4 s;
    tq_split2(v.x, v.y, s.h.x, s.m.x, s.l.x);
    tq_split2(v.z, v.w, s.h.y, s.m.y, s.l.y);
    return s;
}

// ---- mma.sync on parts in shared memory ---------------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t tq_smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void tq_ldm4(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void tq_ldm4t(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
// c (+)= a b, 16 x 8 x 16
template <bool FIRST> __device__ __forceinline__ void tq_mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    if (FIRST)
        asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
                     : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
    else
        asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                     : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// Six products of 16 rows and N groups of eight columns over 16 elements: h h' to `big`, the rest to `small`; a[part], b[part][two groups].
// The tensor cores cut bits off at every addition: sums of h h' are kept short and added up in rounded float32.  With four groups
// a sum is met again after four products, about as many as its latency.
template <int N, bool FIRST_BIG, bool FIRST>
__device__ __forceinline__ void tq_six(float (*big)[4], float (*small)[4], const uint32_t (&a)[3][4], const uint32_t (&b)[3][N / 2][4]) {
#define TQ_ALL(FIRST_, to, pa, pb)                                                                                       \
    _Pragma("unroll") for (int u = 0; u < N; ++u) tq_mma<FIRST_>(to[u], a[pa], b[pb][u >> 1][2 * (u & 1)], b[pb][u >> 1][2 * (u & 1) + 1]);
    TQ_ALL(FIRST_BIG, big, 0, 0)
    TQ_ALL(FIRST, small, 2, 0)
    TQ_ALL(false, small, 1, 1)
    TQ_ALL(false, small, 0, 2)
    TQ_ALL(false, small, 1, 0)
    TQ_ALL(false, small, 0, 1)
#undef TQ_ALL
}
// Rows of N bfloat16 in shared memory, their 16-byte pieces shuffled by the row's lowest three bits: eight neighbouring rows' pieces
// of one column, and a row's pieces, lie in different banks.
template <int N> __device__ __forceinline__ uint32_t tq_piece(int row, int c) { return (uint32_t)(row * (N * 2) + ((c ^ (row & 7)) << 4)); }
// four neighbours of such a row, d a multiple of four; the three parts lie `part` bytes apart
template <int N>
__device__ __forceinline__ void tq_put4(uint32_t at, int part, int row, int d, float4 v) {
    const TqSplit4 s = tq_split4(v);
    const uint32_t a = at + tq_piece<N>(row, d >> 3) + (d & 4) * 2;
    asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(a), "r"(s.h.x), "r"(s.h.y) : "memory");
    asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(a + part), "r"(s.m.x), "r"(s.m.y) : "memory");
    asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(a + 2 * part), "r"(s.l.x), "r"(s.l.y) : "memory");
}
// two neighbours, d even
template <int N>
__device__ __forceinline__ void tq_put2(uint32_t at, int part, int row, int d, float x, float y) {
    uint32_t h, m, l;
    tq_split2(x, y, h, m, l);
    const uint32_t a = at + tq_piece<N>(row, d >> 3) + (d & 7) * 2;
    asm volatile("st.shared.b32 [%0], %1;" ::"r"(a), "r"(h) : "memory");
    asm volatile("st.shared.b32 [%0], %1;" ::"r"(a + part), "r"(m) : "memory");
    asm volatile("st.shared.b32 [%0], %1;" ::"r"(a + 2 * part), "r"(l) : "memory");
}
