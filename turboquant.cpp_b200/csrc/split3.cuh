// float32 as the exact sum of three bfloat16 values, for float32 products on the tensor cores.
//
// x = h + m + l: h is x without its lower 16 bits, m the same of what is left, l the rest; 3 x 8 bits hold the 24 of a
// float32, so nothing is lost (below 2^-110 the last bits of l go; they are less than 2^-133).  Of the nine products of two
// such sums the six largest are taken, h h', h m', m h', m m', h l', l h'; the other three are at most 2^-21 and on average
// 2^-24 of x x' together, what one rounding of a float32 product costs.  Where one side holds bfloat16 values (its m and l are
// zero) three products are exact.  An infinity or a NaN leaves a NaN in m: a caller that must tell them apart looks at the result.
#pragma once
#include "common.cuh"

struct TqSplit4 { uint2 h, m, l; };      // four neighbours: bfloat16 pairs (first in the low half)

__device__ __forceinline__ uint32_t tq_tops(uint32_t a, uint32_t b) { return __byte_perm(a, b, 0x7632); }
__device__ __forceinline__ void tq_split(float x, uint32_t& h, uint32_t& m, uint32_t& l) {
    h = __float_as_uint(x) & 0xffff0000u;
    const float r = x - __uint_as_float(h);
    m = __float_as_uint(r) & 0xffff0000u;
    l = __float_as_uint(r - __uint_as_float(m));
}
// two values: their parts as bfloat16 pairs
__device__ __forceinline__ void tq_split2(float a, float b, uint32_t& h, uint32_t& m, uint32_t& l) {
    uint32_t ha, ma, la, hb, mb, lb;
    tq_split(a, ha, ma, la);
    tq_split(b, hb, mb, lb);
    h = tq_tops(ha, hb);
    m = tq_tops(ma, mb);
    l = tq_tops(la, lb);
}
__device__ __forceinline__ TqSplit4 tq_split4(float4 v) {
    TqSplit4 s;
    tq_split2(v.x, v.y, s.h.x, s.m.x, s.l.x);
    tq_split2(v.z, v.w, s.h.y, s.m.y, s.l.y);
    return s;
}
