// Recurrences over runs of many tokens in chunks of 64, as matrix products in fp32.  A state S [dk, dv] per head with a decay
// and a write per token,
//   S_t = a_t S_(t-1) + b_t k_t v_t^T,   y_t = S_t^T q_t,
// is linear in the state it starts from: with D[t][s] = a_(s+1) ... a_t (products in token order; D[t][t] = 1) and
// A_t = a_first ... a_t, inside a chunk that starts from S_0
//   y_t = A_t S_0^T q_t + sum over s <= t of (q_t . k_s) D[t][s] b_s v_s
//   S_last = A_last S_0 + sum over s of D[last][s] b_s k_s v_s^T.
// Three launches: every chunk's own sum (the second formula from zero) side by side; the states the chunks start from, one chunk
// after the other but every element by itself; every chunk's outputs side by side.  A long step does this for a group of chunks after
// the other, the kept state going from group to group, so that the chunks' states take a bounded buffer.  Token by token (csrc/ssm.cu) a walk does 2
// multiply-adds an element of the state and token, a chain of its tokens with a shuffle tree each, and long runs are walked twice to
// fill the GPU; in chunks it is 2 + 64 (1 / dk + 1 / dv) of them, all in register-tiled products.  Everything is fp32 and
// stays on the CUDA cores: tensor cores round operands (two tf32 parts of each hold 22 of 24 bits; three bfloat16 parts hold all 24 in
// six products, a form that was not built).  Measured, 682 + 1,366 tokens, 16 heads of 128 x 129: 289 us for both walks token by token; here 37 us for the
// chunks' sums, 16 for the starts and 79 for the outputs (1.07 G multiply-adds, 30 us at the fp32 units' rate; what bounds them is shared
// memory, twelve 128-byte reads a warp for its 32 multiply-adds a thread; 102 us with transposed stores and weights that met in one
// bank).
// Part of csrc/ssm.cu's library.
//   memory_chunks   the matrix memory (a = e^gate0, b = e^gate1; n is one more column whose value is one)
#pragma once
#include "chunks.cuh"

namespace tq_recurrence {

constexpr int THREADS = 256;   // 16 x 16: a thread holds 4 x 4 blocks of a product, 64 apart in rows and columns

__device__ __forceinline__ float4 zero4() { return make_float4(0.f, 0.f, 0.f, 0.f); }

// rows [n tokens][N] at src (stride floats apart) -> smem [64][N], zeros behind the last
template <int N>
__device__ __forceinline__ void load_rows(float* dst, const float* __restrict__ src, int stride, int n) {
    constexpr int Q = N / 4;
#pragma unroll
    for (int i = threadIdx.x; i < L * Q; i += THREADS) {
        const int t = i / Q, c = i % Q * 4;
        *reinterpret_cast<float4*>(dst + t * N + c) = t < n ? *reinterpret_cast<const float4*>(src + (size_t)t * stride + c) : zero4();
    }
}
// K columns of R rows -> smem [K][R] (transposed); rows from n on are zeros.  A row's groups of four neighbours (along R) are shuffled
// by the bits of k above the lowest two, so that the lanes of a warp, which read a row's columns together, store into eight
// banks' groups instead of one; a product reads a whole group at one k, wherever it lies.
__device__ __forceinline__ int group_at(int k, int g) { return g ^ ((k >> 2) & 15); }
template <int K, int R>
__device__ __forceinline__ void load_transposed(float* dst, const float* __restrict__ src, int stride, int n) {
    constexpr int Q = K / 4;
#pragma unroll 8
    for (int i = threadIdx.x; i < R * Q; i += THREADS) {
        const int r = i / Q, c = i % Q * 4;
        const float4 v = r < n ? *reinterpret_cast<const float4*>(src + (size_t)r * stride + c) : zero4();
        float* at = dst + c * R + 4 * group_at(c, r >> 2) + (r & 3);
        at[0] = v.x;
        at[R] = v.y;
        at[2 * R] = v.z;
        at[3 * R] = v.w;
    }
}

// acc[4 i + r][2 j + p] += a[k][64 i + 4 ty + r] * b[k][64 j + 4 tx + 2 p, + 1] over k in [k0, k1): a [k][LDA], b [k][LDB] in shared memory
// (TA, TB: as load_transposed leaves them)
template <int RI, int RJ, int LDA, int LDB, bool TA = false, bool TB = false>
__device__ __forceinline__ void product(tq_f32x2 (&acc)[4 * RI][2 * RJ], const float* a, const float* b, int k0, int k1, int ty, int tx) {
#pragma unroll 4
    for (int k = k0; k < k1; ++k) {
        float4 av[RI];
        ulonglong2 bv[RJ];
#pragma unroll
        for (int i = 0; i < RI; ++i) av[i] = *reinterpret_cast<const float4*>(a + k * LDA + 64 * i + 4 * (TA ? group_at(k, ty) : ty));
#pragma unroll
        for (int j = 0; j < RJ; ++j) bv[j] = *reinterpret_cast<const ulonglong2*>(b + k * LDB + 64 * j + 4 * (TB ? group_at(k, tx) : tx));
#pragma unroll
        for (int i = 0; i < RI; ++i) {
            const float ar[4] = {av[i].x, av[i].y, av[i].z, av[i].w};
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const tq_f32x2 x = tq_pack2(ar[r], ar[r]);
#pragma unroll
                for (int j = 0; j < RJ; ++j) {
                    acc[4 * i + r][2 * j] = tq_fma2(x, bv[j].x, acc[4 * i + r][2 * j]);
                    acc[4 * i + r][2 * j + 1] = tq_fma2(x, bv[j].y, acc[4 * i + r][2 * j + 1]);
                }
            }
        }
    }
}
// acc[r][..] += sum over s <= t of Pt[s][t] Vs[s][..] for the thread's rows t = 4 ty + r: the tokens ahead of the warp's eight
// rows as a product, those eight one by one, so that a token never meets a later one's values, whatever they are
template <int RJ, int LDA, int LDB>
__device__ __forceinline__ void add_earlier(tq_f32x2 (&acc)[4][2 * RJ], const float* Pt, const float* Vs, int ty, int tx) {
    const int first = 8 * (ty >> 1);
    product<1, RJ, LDA, LDB>(acc, Pt, Vs, 0, first, ty, tx);
#pragma unroll 2
    for (int s = first; s < first + 8; ++s) {
        const float4 p = *reinterpret_cast<const float4*>(Pt + s * LDA + 4 * ty);
        const float pr[4] = {p.x, p.y, p.z, p.w};
#pragma unroll
        for (int j = 0; j < RJ; ++j) {
            const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(Vs + s * LDB + 64 * j + 4 * tx);
#pragma unroll
            for (int r = 0; r < 4; ++r)
                if (s <= 4 * ty + r) {
                    const tq_f32x2 x = tq_pack2(pr[r], pr[r]);
                    acc[r][2 * j] = tq_fma2(x, v.x, acc[r][2 * j]);
                    acc[r][2 * j + 1] = tq_fma2(x, v.y, acc[r][2 * j + 1]);
                }
        }
    }
}
template <int M, int N>
__device__ __forceinline__ void clear(tq_f32x2 (&acc)[M][N]) {
#pragma unroll
    for (int i = 0; i < M; ++i)
#pragma unroll
        for (int j = 0; j < N; ++j) acc[i][j] = 0ull;
}
__device__ __forceinline__ float4 four(tq_f32x2 a, tq_f32x2 b) {
    const float2 x = tq_unpack2(a), y = tq_unpack2(b);
    return make_float4(x.x, x.y, y.x, y.y);
}

// ---- a chunk's own sum, of the group from chunk0 on: ends [chunk - chunk0][head][dv + 1][dk] (the last row n), decays [..][head] ----
template <int DK, int DV>
__global__ void __launch_bounds__(THREADS, 2)
memory_ends_kernel(const float* __restrict__ rows, int C, int k_off, int v_off, const float2* __restrict__ gates, int heads, int chunk0,
                   const int* __restrict__ cu_seqlens, int n_seqs, float* __restrict__ ends, float* __restrict__ decays) {
    tq_grid_wait();                    // everything below may read what the previous kernel wrote
    tq_grid_launch_dependents();       // the next kernel's CTAs may move in as SMs free up
    extern __shared__ __align__(16) float smem[];
    float* Ks = smem;                  // [64][DK], times the weight of its token
    float* Vs = smem + L * DK;         // [64][DV]
    __shared__ Chunk s_chunk;
    __shared__ float s_w[L], s_half;
    const int h = blockIdx.y;
    const Chunk c = find_chunk(chunk0 + blockIdx.x, cu_seqlens, n_seqs, &s_chunk);
    if (c.n == 0) return;
    const int tid = threadIdx.x, lane = tid & 31;
    load_rows<DV>(Vs, rows + (size_t)c.t0 * C + v_off + h * DV, C, c.n);
    if (tid < L) {                     // D[last][s] b_s: what is left of token s at the chunk's end
        const float2 g = tid < c.n ? gates[(size_t)(c.t0 + tid) * heads + h] : make_float2(0.f, -INFINITY);
        float a = expf(g.x), down = a;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) { const float v = __shfl_down_sync(0xffffffffu, down, o); if (lane + o < 32) down *= v; }
        float after = __shfl_down_sync(0xffffffffu, down, 1);
        if (lane == 31) after = 1.f;
        s_w[tid] = after * expf(g.y);
        if (tid == L / 2) s_half = down;
        if (tid == 0) decays[(size_t)blockIdx.x * heads + h] = down;       // the first half's; completed below
    }
    __syncthreads();
    if (tid < L / 2) s_w[tid] *= s_half;
    if (tid == 0) decays[(size_t)blockIdx.x * heads + h] *= s_half;
    __syncthreads();
    {
        constexpr int Q = DK / 4;
        const float* src = rows + (size_t)c.t0 * C + k_off + h * DK;
#pragma unroll
        for (int i = tid; i < L * Q; i += THREADS) {
            const int t = i / Q, e = i % Q * 4;
            float4 v = t < c.n ? *reinterpret_cast<const float4*>(src + (size_t)t * C + e) : zero4();
            const float w = s_w[t];
            v.x *= w; v.y *= w; v.z *= w; v.w *= w;
            *reinterpret_cast<float4*>(Ks + t * DK + e) = v;
        }
    }
    __syncthreads();
    constexpr int RI = DV / 64, RJ = DK / 64;
    const int ty = tid / 16, tx = tid % 16;
    tq_f32x2 acc[4 * RI][2 * RJ];
    clear(acc);
    product<RI, RJ, DV, DK>(acc, Vs, Ks, 0, L, ty, tx);
    float* out = ends + ((size_t)blockIdx.x * heads + h) * (DV + 1) * DK;
#pragma unroll
    for (int i = 0; i < 4 * RI; ++i)
#pragma unroll
        for (int j = 0; j < RJ; ++j)
            *reinterpret_cast<float4*>(out + (size_t)(i / 4 * 64 + 4 * ty + i % 4) * DK + 64 * j + 4 * tx) = four(acc[i][2 * j], acc[i][2 * j + 1]);
    if (tid < DK) {
        float n = 0.f;
#pragma unroll 8
        for (int s = 0; s < L; ++s) n += Ks[s * DK + tid];
        out[(size_t)DV * DK + tid] = n;
    }
}

// ---- the states the group's chunks start from, in the place of their own sums; the kept state moves to the end of the last -----
__global__ void __launch_bounds__(256)
chunk_starts_kernel(float* __restrict__ state, long long slot_stride, const int* __restrict__ slots, float* __restrict__ ends,
                    const float* __restrict__ decays, int heads, int per_head, int chunk0, int group, const int* __restrict__ cu_seqlens) {
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
    const float* d = decays + (size_t)from * heads + h;
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
template <int DK, int DV>
__global__ void __launch_bounds__(THREADS, 2)
memory_outputs_kernel(const float* __restrict__ rows, int C, int q_off, int k_off, int v_off, const float2* __restrict__ gates, int heads,
                      int chunk0, const int* __restrict__ cu_seqlens, int n_seqs, const float* __restrict__ starts, float* __restrict__ y,
                      float* __restrict__ dots) {
    tq_grid_wait();                    // everything below may read what the previous kernel wrote
    tq_grid_launch_dependents();       // the next kernel's CTAs may move in as SMs free up
    extern __shared__ __align__(16) float smem[];
    constexpr int BUF = 64 * (DK > DV ? DK : DV);
    float* Qt = smem;                  // [DK][64]
    float* X = Qt + DK * L;            // keys [DK][64], then the second 64 rows of the state [64][DV] (DK 128) or the values
    float* Y = X + BUF;                // the state's first 64 rows [64][DV], then (DK 128) the values [64][DV]
    float* Pt = Y + 64 * DV;           // [s][t]: D[t][s], then the weight of value s in output t
    __shared__ Chunk s_chunk;
    __shared__ float s_a[L], s_b[L], s_A[L];
    const int h = blockIdx.y;
    const Chunk c = find_chunk(chunk0 + blockIdx.x, cu_seqlens, n_seqs, &s_chunk);
    if (c.n == 0) return;
    const int tid = threadIdx.x, ty = tid / 16, tx = tid % 16;
    const float* tok = rows + (size_t)c.t0 * C;
    const float* St = starts + ((size_t)blockIdx.x * heads + h) * (DV + 1) * DK;     // [column][dk]
    if (tid < L) {
        const float2 g = tid < c.n ? gates[(size_t)(c.t0 + tid) * heads + h] : make_float2(0.f, -INFINITY);
        s_a[tid] = expf(g.x);
        s_b[tid] = expf(g.y);
    }
    load_transposed<DK, L>(Qt, tok + q_off + h * DK, C, c.n);
    load_transposed<DK, L>(X, tok + k_off + h * DK, C, c.n);
    __syncthreads();
    if (tid < L) {                     // row t of D, a thread each (neighbouring threads store side by side)
        float d = 1.f;
        for (int s = L - 1; s >= 0; --s) {
            if (s < tid) d *= s_a[s + 1];
            Pt[s * L + tid] = s <= tid ? d : 0.f;
        }
    } else if (tid == L) {
        float d = 1.f;
        for (int t = 0; t < L; ++t) { d *= s_a[t]; s_A[t] = d; }
    }
    load_transposed<64, DV>(Y, St, DK, DV);
    __syncthreads();
    {
        tq_f32x2 p[4][2];              // k_s . q_t: rows s, columns t
        clear(p);
        product<1, 1, L, L, true, true>(p, X, Qt, 0, DK, ty, tx);
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const float4 v = four(p[r][0], p[r][1]);
            const float b = s_b[4 * ty + r];
            float4* at = reinterpret_cast<float4*>(Pt + (4 * ty + r) * L + 4 * tx);
            float4 d = *at;
            d.x *= v.x * b; d.y *= v.y * b; d.z *= v.z * b; d.w *= v.w * b;
            *at = d;
        }
    }
    __syncthreads();
    constexpr int RJ = DV / 64;
    tq_f32x2 acc[4][2 * RJ];
    clear(acc);
    if (DK > 64) load_transposed<64, DV>(X, St + 64, DK, DV);
    else load_rows<DV>(X, tok + v_off + h * DV, C, c.n);
    product<1, RJ, L, DV, true, true>(acc, Qt, Y, 0, 64, ty, tx);
    __syncthreads();
    const float* Vs = X;
    if (DK > 64) {
        load_rows<DV>(Y, tok + v_off + h * DV, C, c.n);
        product<1, RJ, L, DV, true, true>(acc, Qt + 64 * L, X, 0, 64, ty, tx);
        __syncthreads();
        Vs = Y;
    }
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const float A = s_A[4 * ty + r];
        const tq_f32x2 AA = tq_pack2(A, A);
#pragma unroll
        for (int j = 0; j < 2 * RJ; ++j) acc[r][j] = tq_mul2(acc[r][j], AA);
    }
    add_earlier<RJ, L, DV>(acc, Pt, Vs, ty, tx);
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const int t = 4 * ty + r;
        if (t < c.n)
#pragma unroll
            for (int j = 0; j < RJ; ++j)
                *reinterpret_cast<float4*>(y + ((size_t)(c.t0 + t) * heads + h) * DV + 64 * j + 4 * tx) = four(acc[r][2 * j], acc[r][2 * j + 1]);
    }
    // n . q: the column whose value is one
    if (tid < c.n) {
        const float* n0 = St + (size_t)DV * DK;
        float from = 0.f, own = 0.f;
#pragma unroll 4
        for (int k = 0; k < DK; ++k) from += Qt[k * L + 4 * group_at(k, tid >> 2) + (tid & 3)] * n0[k];
        for (int s = 0; s <= tid; ++s) own += Pt[s * L + tid];
        dots[(size_t)(c.t0 + tid) * heads + h] = s_A[tid] * from + own;
    }
}

template <int DK, int DV>
int launch_memory(const float* rows, int C, int q_off, int k_off, int v_off, const float2* gates, float* state, long long slot_stride,
                  float* y, float* dots, float* ends, float* decays, int chunks, int group, int n_seqs, int heads, const int* cu, const int* slots,
                  cudaStream_t stream) {
    constexpr int A_BYTES = L * (DK + DV) * 4, C_BYTES = (DK * L + 64 * (DK > DV ? DK : DV) + 64 * DV + L * L) * 4;
    auto ka = memory_ends_kernel<DK, DV>;
    auto kc = memory_outputs_kernel<DK, DV>;
    static std::atomic<unsigned long long> asked_a{0}, asked_c{0};
    cudaError_t e = tq_reserve_smem(ka, A_BYTES, asked_a);
    if (e == cudaSuccess) e = tq_reserve_smem(kc, C_BYTES, asked_c);
    if (e != cudaSuccess) TQ_FAIL(-1, "memory_chunks: %d bytes of shared memory refused: %s", C_BYTES, cudaGetErrorString(e));
    const int per_head = (DV + 1) * DK;
    for (int chunk0 = 0; chunk0 < chunks; chunk0 += group) {
        const int n = chunks - chunk0 < group ? chunks - chunk0 : group;
        tq_launch(dim3(n, heads), THREADS, A_BYTES, stream)(ka, rows, C, k_off, v_off, gates, heads, chunk0, cu, n_seqs, ends, decays);
        tq_launch(dim3((per_head + 255) / 256, n_seqs, heads), 256, 0, stream)(chunk_starts_kernel, state, slot_stride, slots, ends,
            (const float*)decays, heads, per_head, chunk0, n, cu);
        tq_launch(dim3(n, heads), THREADS, C_BYTES, stream)(kc, rows, C, q_off, k_off, v_off, gates, heads, chunk0, cu, n_seqs, (const float*)ends, y, dots);
    }
    TQ_CHECK_LAUNCH("memory_chunks");
    return 0;
}


}  // namespace tq_recurrence

// rows fp32 [T, C] with q, k (heads x dk) and v (heads x dv) from columns that are multiples of four, gates [T, heads] pairs of
// logarithms; state: the sequences' [heads][dv + 1][dk] at slots[s] * slot_stride, renewed; y [T, heads * dv], dots [T, heads] =
// n . q.  chunks: at least the sum of ceil(run / 64); ends [group, heads, dv + 1, dk] and decays [group, heads]: scratch of a group.
TQ_EXPORT int tq_memory_chunks(const float* rows, int C, int q_off, int k_off, int v_off, const void* gates, float* state,
                               long long slot_stride, float* y, float* dots, float* ends, float* decays, int chunks, int group, int n_seqs,
                               int heads, int dk, int dv, const int* cu_seqlens, const int* slots, cudaStream_t stream) {
    if (n_seqs == 0 || chunks == 0) return 0;
    TQ_REQUIRE(heads >= 1 && heads <= 65535 && n_seqs <= 65535 && group >= 1, "memory_chunks: %d heads, %d sequences, groups of %d chunks", heads, n_seqs, group);
    TQ_REQUIRE(C % 4 == 0 && q_off % 4 == 0 && k_off % 4 == 0 && v_off % 4 == 0 && ((uintptr_t)rows & 15) == 0 && ((uintptr_t)y & 15) == 0
               && ((uintptr_t)ends & 15) == 0, "memory_chunks: rows of %d floats are not aligned to 16 bytes", C);
#define MEM_CASE(DK_, DV_) if (dk == DK_ && dv == DV_) return tq_recurrence::launch_memory<DK_, DV_>(rows, C, q_off, k_off, v_off, (const float2*)gates, \
        state, slot_stride, y, dots, ends, decays, chunks, group, n_seqs, heads, cu_seqlens, slots, stream);
    MEM_CASE(64, 64) MEM_CASE(64, 128) MEM_CASE(128, 64) MEM_CASE(128, 128)
#undef MEM_CASE
    TQ_FAIL(-2, "memory_chunks: keys of %d and values of %d elements", dk, dv);
}
