// The matrix memory over runs of many tokens in chunks of 64 as float32 matrix products on the tensor cores, operands as three bfloat16
// values each (split3.cuh).  A state S [dk, dv] per head with a decay and a write per token,
//   S_t = a_t S_(t-1) + b_t k_t v_t^T,   y_t = S_t^T q_t       (a = e^gate0, b = e^gate1; n is one more column whose value is one)
// is linear in the state it starts from: with D[t][s] = a_(s+1) ... a_t (products in token order; D[t][t] = 1) and
// A_t = a_first ... a_t, inside a chunk that starts from S_0
//   y_t = A_t S_0^T q_t + sum over s <= t of (q_t . k_s) D[t][s] b_s v_s
//   S_last = A_last S_0 + sum over s of D[last][s] b_s k_s v_s^T.
// Three launches: every chunk's own sum (the second formula from zero) side by side; the states the chunks start from, one chunk
// after the other but every element by itself; every chunk's outputs side by side.  A long step does this for a group of chunks after
// the other, the kept state going from group to group, so that the chunks' states take a bounded buffer.  Token by token (csrc/ssm.cu)
// a walk does 2 multiply-adds an element of the state and token, a chain of its tokens with a shuffle tree each, and long runs are
// walked twice to fill the GPU; in chunks it is 2 + 64 (1 / dk + 1 / dv) of them, all in products.
// Everything is kept and added up in float32; products are six bfloat16 ones whose largest are summed over at most 64 elements.
// 682 + 1,366 tokens, 16 heads of 128 x 129: 33 us for the chunks' sums, 17 for the starts and 56 for the outputs (as products on the
// fp32 units 37, 16 and 79, bound by what they read of shared memory; token by token 289).  With one CTA an SM the outputs take 89; what bounds
// either kernel with two is a warp's own chain of loads, splitting and products, the tensor cores are active 41 to 42 % of the time.
// An element of a value that is not finite takes no part in earlier tokens' outputs; the token's own and all later ones are NaN in its
// column, and in no other.
// Part of csrc/ssm.cu's library.
#pragma once
#include "split3.cuh"
#include "chunks.cuh"

namespace tq_recurrence {

constexpr int THREADS = 128;

template <int DK, int DV>
struct MemoryCfg {
    static constexpr int K_PART = L * DK * 2, V_PART = L * DV * 2;
    static constexpr int ENDS_BYTES = 3 * (K_PART + V_PART);
    static constexpr int SQ_PART = 32 * DK * 2, VQ_PART = L * 32 * 2;                // 32 columns of a state and of the values
    static constexpr int WORK = 3 * (K_PART > SQ_PART + VQ_PART ? K_PART : SQ_PART + VQ_PART);
    static constexpr int OUT_BYTES = 3 * K_PART + WORK + L * LD * 4;
};

// Rows of 32 bfloat16, their four 16-byte pieces shuffled by bits 1 and 2 of the row: eight neighbouring rows' pieces of one column lie in
// different banks
__device__ __forceinline__ uint32_t piece32(int row, int c) { return (uint32_t)(row * 64 + ((c ^ ((row >> 1) & 3)) << 4)); }

// ---- a chunk's own sum, of the group from chunk0 on: ends [chunk - chunk0][head][dv + 1][dk] (the last row n), last [..][head] ----
template <int DK, int DV>
__global__ void __launch_bounds__(THREADS, 2)
memory_ends_kernel(const float* __restrict__ rows, int C, int k_off, int v_off, const float2* __restrict__ gates, int heads, int chunk0,
                   const int* __restrict__ cu_seqlens, int n_seqs, float* __restrict__ ends, float* __restrict__ last) {
    tq_grid_wait();                    // everything below may read what the previous kernel wrote
    tq_grid_launch_dependents();       // the next kernel's CTAs may move in as SMs free up
    using F = MemoryCfg<DK, DV>;
    extern __shared__ __align__(128) uint8_t smem[];
    const uint32_t sk = tq_smem_u32(smem), sv = sk + 3 * F::K_PART;                // K; V times the weight of its token
    __shared__ Chunk s_chunk;
    __shared__ float s_w[L], s_half;
    const int h = blockIdx.y;
    const Chunk c = find_chunk(chunk0 + blockIdx.x, cu_seqlens, n_seqs, &s_chunk);
    if (c.n == 0) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const Lane ln(lane);
    const float* tok = rows + (size_t)c.t0 * C;
    if (tid < L) {                     // D[last][s] b_s: what is left of token s at the chunk's end
        const float2 g = tid < c.n ? gates[(size_t)(c.t0 + tid) * heads + h] : make_float2(0.f, -INFINITY);
        float a = expf(g.x), down = a;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) { const float v = __shfl_down_sync(0xffffffffu, down, o); if (lane + o < 32) down *= v; }
        float after = __shfl_down_sync(0xffffffffu, down, 1);
        if (lane == 31) after = 1.f;
        s_w[tid] = after * expf(g.y);
        if (tid == L / 2) s_half = down;
        if (tid == 0) last[(size_t)blockIdx.x * heads + h] = down;         // the first half's; completed below
    }
    constexpr int KQ = DK / 4, VQ = DV / 4, KN = L * KQ / THREADS, VN = L * VQ / THREADS;
    float4 v4[VN];                     // on their way while K is split
    {
        float4 k4[KN];
#pragma unroll
        for (int i = 0; i < KN; ++i) {
            const int t = (i * THREADS + tid) / KQ;
            k4[i] = t < c.n ? *reinterpret_cast<const float4*>(tok + (size_t)t * C + k_off + h * DK + tid % KQ * 4) : zero4();
        }
#pragma unroll
        for (int i = 0; i < VN; ++i) {
            const int t = (i * THREADS + tid) / VQ;
            v4[i] = t < c.n ? *reinterpret_cast<const float4*>(tok + (size_t)t * C + v_off + h * DV + tid % VQ * 4) : zero4();
        }
#pragma unroll
        for (int i = 0; i < KN; ++i) tq_put4<DK>(sk, F::K_PART, (i * THREADS + tid) / KQ, tid % KQ * 4, k4[i]);
    }
    __syncthreads();
    if (tid < L / 2) s_w[tid] *= s_half;
    if (tid == 0) last[(size_t)blockIdx.x * heads + h] *= s_half;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < VN; ++i) {
        const int t = (i * THREADS + tid) / VQ;
        const float w = s_w[t];
        v4[i].x *= w; v4[i].y *= w; v4[i].z *= w; v4[i].w *= w;
        tq_put4<DV>(sv, F::V_PART, t, tid % VQ * 4, v4[i]);
    }
    __syncthreads();
    float* out = ends + ((size_t)blockIdx.x * heads + h) * (DV + 1) * DK;
    constexpr int MT = DV / 64;        // groups of 16 columns a warp takes
    for (int d4 = 0; d4 < DK / 32; ++d4) {
        float big[MT][4][4], small[MT][4][4];
#pragma unroll
        for (int k = 0; k < L / 16; ++k) {
            uint32_t b[3][2][4];
#pragma unroll
            for (int p = 0; p < 3; ++p)
#pragma unroll
                for (int j = 0; j < 2; ++j) tq_ldm4t(b[p][j], sk + p * F::K_PART + tq_piece<DK>(16 * k + ln.t_row, 4 * d4 + 2 * j + ln.t_c));
#pragma unroll
            for (int mt = 0; mt < MT; ++mt) {
                uint32_t a[3][4];
#pragma unroll
                for (int p = 0; p < 3; ++p) tq_ldm4t(a[p], sv + p * F::V_PART + tq_piece<DV>(16 * k + ln.v_row, 2 * (warp * MT + mt) + ln.v_c));
                if (k == 0) tq_six<4, true, true>(big[mt], small[mt], a, b); else tq_six<4, false, false>(big[mt], small[mt], a, b);
            }
        }
#pragma unroll
        for (int mt = 0; mt < MT; ++mt)
#pragma unroll
            for (int u = 0; u < 4; ++u)
#pragma unroll
                for (int r = 0; r < 2; ++r)
                    *reinterpret_cast<float2*>(out + (size_t)(16 * (warp * MT + mt) + ln.r + 8 * r) * DK + 32 * d4 + 8 * u + ln.c) =
                        make_float2(big[mt][u][2 * r] + small[mt][u][2 * r], big[mt][u][2 * r + 1] + small[mt][u][2 * r + 1]);
    }
    if (tid < DK) {
        float n = 0.f;
#pragma unroll 16
        for (int s = 0; s < c.n; ++s) n = fmaf(s_w[s], tok[(size_t)s * C + k_off + h * DK + tid], n);
        out[(size_t)DV * DK + tid] = n;
    }
}

// ---- the states the group's chunks start from, in the place of their own sums; the kept state moves to the end of the last -----
__global__ void __launch_bounds__(256)
chunk_starts_kernel(float* __restrict__ state, long long slot_stride, const int* __restrict__ slots, float* __restrict__ ends,
                    const float* __restrict__ last, int heads, int per_head, int chunk0, int group, const int* __restrict__ cu_seqlens) {
    tq_grid_wait();                    // everything below may read what the previous kernel wrote
    tq_grid_launch_dependents();       // the next kernel's CTAs may move in as SMs free up
    __shared__ int s_first;
    const int s = blockIdx.y, h = blockIdx.z, e = blockIdx.x * blockDim.x + threadIdx.x;
    if (threadIdx.x < 32) {            // chunks of the sequences before this one
        int before = 0;
        for (int i = threadIdx.x; i < s; i += 32) before += (cu_seqlens[i + 1] - cu_seqlens[i] + L - 1) / L;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) before += __shfl_xor_sync(0xffffffffu, before, o);
        if (threadIdx.x == 0) s_first = before;
    }
    __syncthreads();
    // the sequence's chunks that are in the group, counted from chunk0
    const int from = max(s_first - chunk0, 0), to = min(s_first + (cu_seqlens[s + 1] - cu_seqlens[s] + L - 1) / L - chunk0, group), n = to - from;
    if (e >= per_head || n <= 0) return;
    float* cell = state + (size_t)slots[s] * slot_stride + (size_t)h * per_head + e;
    float* at = ends + ((size_t)from * heads + h) * per_head + e;
    const float* d = last + (size_t)from * heads + h;
    const size_t step = (size_t)heads * per_head;
    float S = *cell;
    constexpr int AHEAD = 8;           // the sums do not depend on the chain: eight of them on their way together
    for (int c = 0; c < n; c += AHEAD) {
        float own[AHEAD], a[AHEAD];
#pragma unroll
        for (int i = 0; i < AHEAD; ++i) {
            own[i] = c + i < n ? at[(size_t)(c + i) * step] : 0.f;
            a[i] = c + i < n ? d[(size_t)(c + i) * heads] : 0.f;
        }
#pragma unroll
        for (int i = 0; i < AHEAD; ++i)
            if (c + i < n) {
                at[(size_t)(c + i) * step] = S;
                S = a[i] * S + own[i];
            }
    }
    *cell = S;
}

// ---- a chunk's outputs ----------------------------------------------------------------------------------------------------------
// A warp has 16 tokens; the weights of the chunk's own tokens stay in its registers, the columns come 32 at a time while the 32 ahead
// are multiplied.
template <int DK, int DV>
__global__ void __launch_bounds__(THREADS, 2)
memory_outputs_kernel(const float* __restrict__ rows, int C, int q_off, int k_off, int v_off, const float2* __restrict__ gates, int heads,
                      int chunk0, const int* __restrict__ cu_seqlens, int n_seqs, const float* __restrict__ starts, float* __restrict__ y,
                      float* __restrict__ dots) {
    tq_grid_wait();                    // everything below may read what the previous kernel wrote
    tq_grid_launch_dependents();       // the next kernel's CTAs may move in as SMs free up
    using F = MemoryCfg<DK, DV>;
    extern __shared__ __align__(128) uint8_t smem[];
    const uint32_t sq = tq_smem_u32(smem), sk = sq + 3 * F::K_PART, sv = sk + 3 * F::SQ_PART;   // Q; K, then 32 columns of the state and of V
    float* m = reinterpret_cast<float*>(smem + 3 * F::K_PART + F::WORK);
    __shared__ Chunk s_chunk;
    // (Two CTAs an SM fit with 2 KB to spare: every 256 bytes count.  The b lie in the unused column of m, n . q where the a were.)
    __shared__ float s_a[L], s_A[L];
    __shared__ int s_bad[2];           // of the 32 columns at hand: the first token whose value is not finite
    const int h = blockIdx.y;
    const Chunk c = find_chunk(chunk0 + blockIdx.x, cu_seqlens, n_seqs, &s_chunk);
    if (c.n == 0) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const Lane ln(lane);
    const float* tok = rows + (size_t)c.t0 * C;
    const float* St = starts + ((size_t)blockIdx.x * heads + h) * (DV + 1) * DK;     // [column][dk]
    if (tid < L) {
        const float2 g = tid < c.n ? gates[(size_t)(c.t0 + tid) * heads + h] : make_float2(0.f, -INFINITY);
        s_a[tid] = expf(g.x);
        m[tid * LD + L] = expf(g.y);
    }
    if (tid == 0) s_bad[0] = L;
    constexpr int KQ = DK / 4, KN = L * KQ / THREADS;
    float from[KN];
    {
        float4 q4[KN], k4[KN];         // all of them asked for before the first is used
#pragma unroll
        for (int i = 0; i < KN; ++i) {
            const int t = (i * THREADS + tid) / KQ, e = tid % KQ * 4;
            const float* at = tok + (size_t)t * C + h * DK + e;
            q4[i] = t < c.n ? *reinterpret_cast<const float4*>(at + q_off) : zero4();
            k4[i] = t < c.n ? *reinterpret_cast<const float4*>(at + k_off) : zero4();
        }
        const float4 n4 = *reinterpret_cast<const float4*>(St + (size_t)DV * DK + tid % KQ * 4);       // the column whose value is one
#pragma unroll
        for (int i = 0; i < KN; ++i) {
            const int t = (i * THREADS + tid) / KQ, e = tid % KQ * 4;
            tq_put4<DK>(sq, F::K_PART, t, e, q4[i]);
            tq_put4<DK>(sk, F::K_PART, t, e, k4[i]);
            from[i] = fmaf(q4[i].x, n4.x, fmaf(q4[i].y, n4.y, fmaf(q4[i].z, n4.z, q4[i].w * n4.w)));
#pragma unroll
            for (int o = KQ / 2; o > 0; o >>= 1) from[i] += __shfl_xor_sync(0xffffffffu, from[i], o);
        }
    }
    __syncthreads();
    decays(m, s_a, s_A, nullptr);
    // the first 32 columns of the state and of the values are on their way meanwhile
    constexpr int SN = 32 * DK / 4 / THREADS, VN = L * 8 / THREADS;
    float4 ns[SN], nv[VN];
    auto ask = [&](int q) {
        const float4* s_at = reinterpret_cast<const float4*>(St + (size_t)32 * q * DK) + tid;
#pragma unroll
        for (int i = 0; i < SN; ++i) ns[i] = s_at[i * THREADS];
#pragma unroll
        for (int i = 0; i < VN; ++i) {
            const int t = (i * THREADS + tid) >> 3, e = (tid & 7) * 4;
            nv[i] = t < c.n ? *reinterpret_cast<const float4*>(tok + (size_t)t * C + v_off + h * DV + 32 * q + e) : zero4();
        }
    };
    ask(0);
    __syncthreads();
    if (tid % KQ == 0)
#pragma unroll
        for (int i = 0; i < KN; ++i) s_a[(i * THREADS + tid) / KQ] = from[i];
    uint32_t P[L / 16][3][4];          // (Q K^T) o D times b as left operands
    float own[2] = {0.f, 0.f};         // their sums: n of the chunk's own tokens
    for (int grp = 0; grp < 2; ++grp) {
        float big[4][4], small[4][4], first[4][4];
        if (grp <= warp >> 1) {
#pragma unroll
            for (int k = 0; k < DK / 16; ++k) {
                if (k == 4)
#pragma unroll
                    for (int u = 0; u < 4; ++u)
#pragma unroll
                        for (int e = 0; e < 4; ++e) first[u][e] = big[u][e];
                uint32_t a[3][4], b[3][2][4];
#pragma unroll
                for (int p = 0; p < 3; ++p) {
                    tq_ldm4(a[p], sq + p * F::K_PART + tq_piece<DK>(16 * warp + ln.a_row, 2 * k + ln.a_c));
#pragma unroll
                    for (int j = 0; j < 2; ++j) tq_ldm4(b[p][j], sk + p * F::K_PART + tq_piece<DK>(32 * grp + 16 * j + ln.b_row, 2 * k + ln.b_c));
                }
                if (k == 0) tq_six<4, true, true>(big, small, a, b);
                else if (k == 4) tq_six<4, true, false>(big, small, a, b);
                else tq_six<4, false, false>(big, small, a, b);
            }
        }
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const int t = 16 * warp + ln.r + 8 * r, s = 32 * grp + 8 * u + ln.c;
                // a token never meets a later one, whatever that is
                auto val = [&](int e) {
                    const int at = s + (e & 1);
                    return at > t ? 0.f : m[t * LD + at] * m[at * LD + L] * ((DK > 64 ? first[u][e] + big[u][e] : big[u][e]) + small[u][e]);
                };
                const float x = val(2 * r), z = val(2 * r + 1);
                own[r] += x + z;
                const int at = 2 * (u & 1) + r;
                if (grp == 0) tq_split2(x, z, P[u >> 1][0][at], P[u >> 1][1][at], P[u >> 1][2][at]);
                else tq_split2(x, z, P[2 + (u >> 1)][0][at], P[2 + (u >> 1)][1][at], P[2 + (u >> 1)][2][at]);
            }
    }
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        own[r] += __shfl_xor_sync(0xffffffffu, own[r], 1);
        own[r] += __shfl_xor_sync(0xffffffffu, own[r], 2);
    }
    const float A[2] = {s_A[16 * warp + ln.r], s_A[16 * warp + ln.r + 8]};
    for (int q = 0; q < DV / 32; ++q) {
        __syncthreads();               // what was there has been used
        if (q == 0 && ln.c == 0)       // n . q
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const int t = 16 * warp + ln.r + 8 * r;
                if (t < c.n) dots[(size_t)(c.t0 + t) * heads + h] = s_A[t] * s_a[t] + own[r];
            }
#pragma unroll
        for (int i = 0; i < SN; ++i) { const int at = (i * THREADS + tid) * 4; tq_put4<DK>(sk, F::SQ_PART, at / DK, at % DK, ns[i]); }
#pragma unroll
        for (int i = 0; i < VN; ++i) {
            const int t = (i * THREADS + tid) >> 3, e = (tid & 7) * 4;
            if (odd(nv[i]) != 0.f) {
                atomicMin(&s_bad[q & 1], t);
                auto held = [](float v) { return isfinite(v) ? v : 0.f; };
                nv[i] = make_float4(held(nv[i].x), held(nv[i].y), held(nv[i].z), held(nv[i].w));
            }
            const TqSplit4 v = tq_split4(nv[i]);
            const uint32_t at = sv + piece32(t, e >> 3) + (e & 4) * 2;
            asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(at), "r"(v.h.x), "r"(v.h.y) : "memory");
            asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(at + F::VQ_PART), "r"(v.m.x), "r"(v.m.y) : "memory");
            asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(at + 2 * F::VQ_PART), "r"(v.l.x), "r"(v.l.y) : "memory");
        }
        if (q + 1 < DV / 32) ask(q + 1);
        __syncthreads();
        if (tid == 0) s_bad[(q + 1) & 1] = L;
        float big[4][4], small[4][4], o[4][4];
#pragma unroll
        for (int k = 0; k < DK / 16; ++k) {
            if (k == 4)
#pragma unroll
                for (int u = 0; u < 4; ++u)
#pragma unroll
                    for (int e = 0; e < 4; ++e) o[u][e] = big[u][e];
            uint32_t a[3][4], b[3][2][4];
#pragma unroll
            for (int p = 0; p < 3; ++p) {
                tq_ldm4(a[p], sq + p * F::K_PART + tq_piece<DK>(16 * warp + ln.a_row, 2 * k + ln.a_c));
#pragma unroll
                for (int j = 0; j < 2; ++j) tq_ldm4(b[p][j], sk + p * F::SQ_PART + tq_piece<DK>(16 * j + ln.b_row, 2 * k + ln.b_c));
            }
            if (k == 0) tq_six<4, true, true>(big, small, a, b);
            else if (k == 4) tq_six<4, true, false>(big, small, a, b);
            else tq_six<4, false, false>(big, small, a, b);
        }
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
            for (int e = 0; e < 4; ++e) o[u][e] = A[e >> 1] * ((DK > 64 ? o[u][e] + big[u][e] : big[u][e]) + small[u][e]);
#pragma unroll
        for (int k = 0; k < L / 16; ++k) {
            if (k > warp) break;       // later tokens
            uint32_t b[3][2][4];
#pragma unroll
            for (int p = 0; p < 3; ++p)
#pragma unroll
                for (int j = 0; j < 2; ++j) tq_ldm4t(b[p][j], sv + p * F::VQ_PART + piece32(16 * k + ln.t_row, 2 * j + ln.t_c));
            if (k == 0) tq_six<4, true, true>(big, small, P[k], b); else tq_six<4, false, false>(big, small, P[k], b);
        }
        const int bad = *(volatile int*)&s_bad[q & 1];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const int t = 16 * warp + ln.r + 8 * r;
            float* at = y + ((size_t)(c.t0 + t) * heads + h) * DV + 32 * q + ln.c;
            if (t < c.n)
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    auto sum = [&](int e) { return o[u][e] + (big[u][e] + small[u][e]); };
                    *reinterpret_cast<float2*>(at + 8 * u) = make_float2(sum(2 * r), sum(2 * r + 1));
                }
        }
        if (bad < L)                   // the columns that have such a value, from its token on: the values are looked at once more
#pragma unroll 1
            for (int i = 0; i < 8; ++i) {
                const int column = h * DV + 32 * q + 8 * (i >> 1) + ln.c + (i & 1);
                bool lost = false;
                for (int t = bad; t < c.n; ++t) {
                    lost |= !isfinite(tok[(size_t)t * C + v_off + column]);
                    if (lost && t >> 4 == warp && (t & 7) == ln.r) y[(size_t)(c.t0 + t) * heads * DV + column] = NAN;
                }
            }
    }
}

template <int DK, int DV>
int launch_memory(const float* rows, int C, int q_off, int k_off, int v_off, const float2* gates, float* state, long long slot_stride, float* y,
           float* dots, float* ends, float* last, int chunks, int group, int n_seqs, int heads, const int* cu, const int* slots, cudaStream_t stream) {
    using F = MemoryCfg<DK, DV>;
    static std::atomic<unsigned long long> asked[2];
    cudaError_t e = tq_reserve_smem(memory_ends_kernel<DK, DV>, F::ENDS_BYTES, asked[0]);
    if (e == cudaSuccess) e = tq_reserve_smem(memory_outputs_kernel<DK, DV>, F::OUT_BYTES, asked[1]);
    if (e != cudaSuccess) TQ_FAIL(-1, "memory_chunks: %d bytes of shared memory refused: %s", F::OUT_BYTES, cudaGetErrorString(e));
    const int per_head = (DV + 1) * DK;
    for (int chunk0 = 0; chunk0 < chunks; chunk0 += group) {
        const int n = chunks - chunk0 < group ? chunks - chunk0 : group;
        tq_launch(dim3(n, heads), THREADS, F::ENDS_BYTES, stream)(memory_ends_kernel<DK, DV>, rows, C, k_off, v_off, gates, heads, chunk0, cu, n_seqs, ends, last);
        tq_launch(dim3((per_head + 255) / 256, n_seqs, heads), 256, 0, stream)(chunk_starts_kernel, state, slot_stride, slots, ends,
            (const float*)last, heads, per_head, chunk0, n, cu);
        tq_launch(dim3(n, heads), THREADS, F::OUT_BYTES, stream)(memory_outputs_kernel<DK, DV>, rows, C, q_off, k_off, v_off, gates, heads, chunk0, cu,
            n_seqs, (const float*)ends, y, dots);
    }
    TQ_CHECK_LAUNCH("memory_chunks");
    return 0;
}

}  // namespace tq_recurrence

// rows fp32 [T, C] with q, k (heads x dk) and v (heads x dv) from columns that are multiples of four, gates [T, heads] pairs of
// logarithms; state: the sequences' [heads][dv + 1][dk] at slots[s] * slot_stride, renewed; y [T, heads * dv], dots [T, heads] =
// n . q.  chunks: at least the sum of ceil(run / 64); ends [group, heads, dv + 1, dk] and last [group, heads]: scratch of a group.
TQ_EXPORT int tq_memory_chunks(const float* rows, int C, int q_off, int k_off, int v_off, const void* gates, float* state,
                               long long slot_stride, float* y, float* dots, float* ends, float* last, int chunks, int group, int n_seqs,
                               int heads, int dk, int dv, const int* cu_seqlens, const int* slots, cudaStream_t stream) {
    if (n_seqs == 0 || chunks == 0) return 0;
    TQ_REQUIRE(heads >= 1 && heads <= 65535 && n_seqs <= 65535 && group >= 1, "memory_chunks: %d heads, %d sequences, groups of %d chunks", heads, n_seqs, group);
    TQ_REQUIRE(C % 4 == 0 && q_off % 4 == 0 && k_off % 4 == 0 && v_off % 4 == 0 && ((uintptr_t)rows & 15) == 0 && ((uintptr_t)y & 15) == 0
               && ((uintptr_t)ends & 15) == 0, "memory_chunks: rows of %d floats are not aligned to 16 bytes", C);
#define MEM_CASE(DK_, DV_) if (dk == DK_ && dv == DV_) return tq_recurrence::launch_memory<DK_, DV_>(rows, C, q_off, k_off, v_off, (const float2*)gates, \
        state, slot_stride, y, dots, ends, last, chunks, group, n_seqs, heads, cu_seqlens, slots, stream);
    MEM_CASE(64, 64) MEM_CASE(64, 128) MEM_CASE(128, 64) MEM_CASE(128, 128)
#undef MEM_CASE
    TQ_FAIL(-2, "memory_chunks: keys of %d and values of %d elements", dk, dv);
}
