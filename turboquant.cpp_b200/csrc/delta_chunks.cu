// The delta rule with one decay per head over runs of many tokens, in chunks of 64 as float32 matrix products on the tensor
// cores, operands as three bfloat16 values each (split3.cuh).
//
// Per head, S [dk, dv]: S_t = g_t S_(t-1) + k_t u_t^T, u_t = beta_t (v_t - g_t S_(t-1)^T k_t), o_t = S_t^T q_t (token by token: csrc/ssm.cu).
// Inside a chunk that starts from S, with A_t = g_1 ... g_t and D[t][s] = g_(s+1) ... g_t, the u of the chunk solve
//   (1 + B) U = diag(beta) (V - diag(A) K S),   B[t][s] = beta_t D[t][s] k_t . k_s for s < t,
// so with T = (1 + B)^-1
//   U = T diag(beta) (V - diag(A) K S);   S' = A_last S + K^T diag(D[last]) U;   o = diag(A) Q S + (D o Q K^T) U.
// A chain of one link per chunk instead of one per token.  (The chunkwise form of Yang, Wang, Zhang, Shen and Kim, "Parallelizing
// linear transformers with the delta rule over sequence length", 2024, with decays.)  Three launches:
//   delta_solve    T of every chunk, side by side: by blocks of 16, the diagonal ones by forward substitution, the others from them, in
//                  float32 on the CUDA cores.  Leaves T and K in parts, as the next launches' shared memory holds them
//   delta_chain    the chunks in order; a CTA has 16 columns of a head's state, in registers.  Three products a link, 64 x 128 x 16,
//                  64 x 64 x 16, 128 x 64 x 16.  Leaves U and the states the chunks start from
//   delta_outputs  the outputs of every chunk, side by side
// 2,048 tokens, 16 heads of 128: 187 us with delta_prepare (12), the solving 40, the chain 80 and the outputs 54; token by token 337.
// Errors against 64 bits are those of the walk: outputs 1.8e-7 to 2.1e-7, states 1.6e-7 to 1.9e-7 (walk 1.8e-7 to 2.1e-7, 1.6e-7 to 1.9e-7).
// A link is 2.4 us: products 1.0 (1,019 multiply-adds a cycle and SM), the rest their way through shared memory and 72 KB of K and T.
// Chains that were longer: W = T diag(beta A) K in the place of K S, a product less but 96 KB, 2.1 us and a third more work beside the chain;
// the same with keys brought in float32 and split by four more warps 2.9.
// A long step does this for a group of chunks after the other, the kept state going from group to group.
// What is not finite leaves the tokens ahead of it in its chunk as they are (it takes no part in the products).  A key, decay or
// beta: the token's own output, all later ones and the state are NaN for that head.  An element of a value: the same for its own column,
// and no other.
// Everything is kept and added up in float32; products are six bfloat16 ones whose largest are summed over at most 64 elements.
#include "split3.cuh"
#include "chunks.cuh"

TQ_DEFINE_LAST_ERROR

namespace {

using namespace tq_recurrence;

constexpr int THREADS = 128, CHAIN_WARPS = 4;
constexpr int T_PART = L * L * 2;
constexpr int XLD = 72;                                         // row stride of the warps' shares of K S: four rows' pairs in different banks
constexpr uint32_t WAIT_LIMIT = 1u << 20;                       // polls of an mbarrier before a wait gives up ...
constexpr uint64_t WAIT_NS = 2000000000ull;                     // ... or two seconds

template <int DK, int DV>
struct Cfg {
    static constexpr int K_PART = L * DK * 2, IMAGE = 3 * K_PART;                    // 64 rows of dk in parts, as they lie in shared memory
    static constexpr int SOLVE_BYTES = IMAGE + 3 * T_PART + 2 * L * LD * 4 + 3 * 16 * 17 * 4;
    static constexpr int K_STAGES = 3, T_STAGES = 2, U_PART = 16 * L * 2;
    static constexpr int CHAIN_BYTES = K_STAGES * IMAGE + T_STAGES * 3 * T_PART + 6 * U_PART + CHAIN_WARPS * 16 * XLD * 4 + 128 /* alignment */;
    static_assert(CHAIN_BYTES <= 227 * 1024, "shared memory");
    static constexpr int SQ_PART = 32 * DK * 2, UQ_PART = 32 * L * 2;                // 32 columns of a state and of U
    static constexpr int WORK = IMAGE > 3 * SQ_PART + 3 * UQ_PART ? IMAGE : 3 * SQ_PART + 3 * UQ_PART;
    static constexpr int OUT_BYTES = IMAGE + WORK + L * LD * 4;
};

// What the launches pass on: per (chunk, key head) K, per (chunk, head) T, both as images; U [dv][64]; the states the chunks start from
// [dv][dk]; a row of numbers.
struct Scratch { uint8_t *k, *t; float *u, *s, *d; };
constexpr int T_IMAGE = 3 * T_PART;
constexpr int N_A = 0, N_BETA = L, N_D = 2 * L, N_LAST = 3 * L, N_BAD = 3 * L + 1;      // A, beta, D[last], A_last, the first token that is
constexpr int N_COLS = 3 * L + 4, N_ROW = N_COLS + 128;                                // not finite (64: none) and, per column, the first value

// What a token brings, as delta_prepare lays it out: [k: G x dk | q: G x dk | g: H | k.q: G | beta: H]
struct Rows { const float* at; int stride, heads, kv_heads; };

template <int DK, int DV>
__global__ void __launch_bounds__(THREADS, 2)
delta_solve_kernel(Rows rows, Scratch out, int chunk0, const int* __restrict__ cu_seqlens, int n_seqs) {
    tq_grid_wait();                    // everything below may read what the previous kernel wrote
    tq_grid_launch_dependents();       // the next kernel's CTAs may move in as SMs free up
    using F = Cfg<DK, DV>;
    extern __shared__ __align__(128) uint8_t smem[];
    const uint32_t sk = tq_smem_u32(smem), st = sk + F::IMAGE;                     // K, T
    float* m = reinterpret_cast<float*>(smem + F::IMAGE + T_IMAGE);                // D, then B
    float* T = m + L * LD;
    float* Y = T + L * LD;
    __shared__ Chunk s_chunk;
    __shared__ float s_g[L], s_beta[L], s_A[L], s_D[L];
    __shared__ int s_bad;
    const int h = blockIdx.y, g = h / (rows.heads / rows.kv_heads);
    const Chunk c = find_chunk(chunk0 + blockIdx.x, cu_seqlens, n_seqs, &s_chunk);
    if (c.n == 0) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const Lane ln(lane);
    const size_t unit = (size_t)blockIdx.x * rows.heads + h;
    const float* tok = rows.at + (size_t)c.t0 * rows.stride;
    if (tid == 0) s_bad = L;
    __syncthreads();
    if (tid < L) {
        const float* mine = tok + (size_t)tid * rows.stride + 2 * rows.kv_heads * DK;
        const float a = tid < c.n ? mine[h] : 1.f, b = tid < c.n ? mine[rows.heads + rows.kv_heads + h] : 0.f;
        const bool fine = isfinite(a) && isfinite(b);
        s_g[tid] = fine ? a : 1.f;
        s_beta[tid] = fine ? b : 0.f;
        if (!fine) atomicMin(&s_bad, tid);
    }
    {
        constexpr int KQ = DK / 4, KN = L * KQ / THREADS;
        float4 k4[KN];                 // all of them asked for before the first is used
#pragma unroll
        for (int i = 0; i < KN; ++i) {
            const int t = (i * THREADS + tid) / KQ;
            k4[i] = t < c.n ? *reinterpret_cast<const float4*>(tok + (size_t)t * rows.stride + g * DK + tid % KQ * 4) : zero4();
        }
#pragma unroll
        for (int i = 0; i < KN; ++i) {
            const int t = (i * THREADS + tid) / KQ;
            if (odd(k4[i]) != 0.f) { atomicMin(&s_bad, t); k4[i] = zero4(); }
            tq_put4<DK>(sk, F::K_PART, t, tid % KQ * 4, k4[i]);
        }
    }
    for (int i = tid; i < L * LD; i += THREADS) T[i] = 0.f;
    __syncthreads();
    decays(m, s_g, s_A, s_D);
    __syncthreads();
    // B
    for (int grp = 0; grp <= warp >> 1; ++grp) {               // 32 columns at a time, none that lie above the diagonal
        float big[4][4], small[4][4], first[4][4];
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
                tq_ldm4(a[p], sk + p * F::K_PART + tq_piece<DK>(16 * warp + ln.a_row, 2 * k + ln.a_c));
#pragma unroll
                for (int j = 0; j < 2; ++j) tq_ldm4(b[p][j], sk + p * F::K_PART + tq_piece<DK>(32 * grp + 16 * j + ln.b_row, 2 * k + ln.b_c));
            }
            if (k == 0) tq_six<4, true, true>(big, small, a, b);
            else if (k == 4) tq_six<4, true, false>(big, small, a, b);
            else tq_six<4, false, false>(big, small, a, b);
        }
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int t = 16 * warp + ln.r + 8 * (e >> 1), s = 32 * grp + 8 * u + ln.c + (e & 1);
                float* at = m + t * LD + s;
                *at = s < t ? s_beta[t] * *at * ((DK > 64 ? first[u][e] + big[u][e] : big[u][e]) + small[u][e]) : 0.f;
            }
    }
    __syncthreads();
    // T: its diagonal blocks, a column a thread ...
    if (tid < L) {
        const int b0 = tid & ~15, col = tid & 15;
        float x[16];
#pragma unroll
        for (int t = 0; t < 16; ++t) {
            float v = t == col ? 1.f : 0.f;
#pragma unroll
            for (int s = 0; s < t; ++s) v = fmaf(-m[(b0 + t) * LD + b0 + s], x[s], v);
            x[t] = v;
            T[(b0 + t) * LD + b0 + col] = v;
        }
    }
    __syncthreads();
    // ... then those 1, 2, 3 below it: T_ij = -T_ii sum over k of B_ik T_kj
    for (int below = 1; below < 4; ++below) {
        const int r = tid >> 3, c2 = (tid & 7) * 2;
        for (int j = 0; j + below < 4; ++j) {
            const int i = j + below;
            float y0 = 0.f, y1 = 0.f;
#pragma unroll 16
            for (int k = 16 * j; k < 16 * i; ++k) {
                const float b = m[(16 * i + r) * LD + k];
                y0 = fmaf(b, T[k * LD + 16 * j + c2], y0);
                y1 = fmaf(b, T[k * LD + 16 * j + c2 + 1], y1);
            }
            Y[(j * 16 + r) * 17 + c2] = y0;
            Y[(j * 16 + r) * 17 + c2 + 1] = y1;
        }
        __syncthreads();
        for (int j = 0; j + below < 4; ++j) {
            const int i = j + below;
            float y0 = 0.f, y1 = 0.f;
#pragma unroll
            for (int k = 0; k < 16; ++k) {
                const float b = T[(16 * i + r) * LD + 16 * i + k];
                y0 = fmaf(b, Y[(j * 16 + k) * 17 + c2], y0);
                y1 = fmaf(b, Y[(j * 16 + k) * 17 + c2 + 1], y1);
            }
            T[(16 * i + r) * LD + 16 * j + c2] = -y0;
            T[(16 * i + r) * LD + 16 * j + c2 + 1] = -y1;
        }
        __syncthreads();
    }
#pragma unroll 4
    for (int i = tid; i < L * L / 4; i += THREADS) {
        const int t = i / (L / 4), s = i % (L / 4) * 4;
        tq_put4<L>(st, T_PART, t, s, make_float4(T[t * LD + s], T[t * LD + s + 1], T[t * LD + s + 2], T[t * LD + s + 3]));
    }
    float* d = out.d + unit * N_ROW;
    if (tid < L) { d[N_A + tid] = s_A[tid]; d[N_BETA + tid] = s_beta[tid]; d[N_D + tid] = s_D[tid]; }
    if (tid == 0) { d[N_LAST] = s_A[L - 1]; d[N_BAD] = (float)s_bad; }
    __syncthreads();
    auto image = [&](uint8_t* to, const uint8_t* from, int bytes) {
#pragma unroll 8
        for (int i = tid; i < bytes / 16; i += THREADS) reinterpret_cast<uint4*>(to)[i] = reinterpret_cast<const uint4*>(from)[i];
    };
    image(out.t + unit * T_IMAGE, smem + F::IMAGE, T_IMAGE);
    if (h % (rows.heads / rows.kv_heads) == 0) image(out.k + ((size_t)blockIdx.x * rows.kv_heads + g) * F::IMAGE, smem, F::IMAGE);
}

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) { asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count)); }
__device__ __forceinline__ void mbar_arrive(uint32_t bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory"); }
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
    uint64_t t0 = 0;
    for (uint32_t i = 0; i < WAIT_LIMIT; ++i) {
        if (mbar_try_wait(bar, parity)) return true;
        if ((i & 255u) == 255u) {
            if (*abort_flag) return false;
            uint64_t now;
            asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
            if (t0 == 0) t0 = now;
            else if (now - t0 > WAIT_NS) break;
        }
    }
    *abort_flag = 1;
    return false;
}
__device__ __forceinline__ void chain_sync() { asm volatile("bar.sync 1, %0;" ::"n"(32 * CHAIN_WARPS) : "memory"); }
// ... and whether any of the warps says so
__device__ __forceinline__ bool chain_any(bool mine) {
    uint32_t any;
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %1, 0;\n\tbar.red.or.pred q, 1, %2, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
                 : "=r"(any) : "r"(mine ? 1u : 0u), "n"(32 * CHAIN_WARPS) : "memory");
    return any != 0;
}

__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}

// Six products of 16 rows and 16 columns with three sums a group of eight columns (big, and two in small), so that none is met again too soon.
template <bool FIRST>
__device__ __forceinline__ void six2(float (&big)[2][4], float (&small)[2][2][4], const uint32_t (&a)[3][4], const uint32_t (&b)[3][4]) {
#pragma unroll
    for (int u = 0; u < 2; ++u) tq_mma<FIRST>(big[u], a[0], b[0][2 * u], b[0][2 * u + 1]);
#pragma unroll
    for (int u = 0; u < 2; ++u) tq_mma<FIRST>(small[0][u], a[2], b[0][2 * u], b[0][2 * u + 1]);
#pragma unroll
    for (int u = 0; u < 2; ++u) tq_mma<FIRST>(small[1][u], a[1], b[0][2 * u], b[0][2 * u + 1]);
#pragma unroll
    for (int u = 0; u < 2; ++u) tq_mma<false>(small[0][u], a[1], b[1][2 * u], b[1][2 * u + 1]);
#pragma unroll
    for (int u = 0; u < 2; ++u) tq_mma<false>(small[1][u], a[0], b[1][2 * u], b[1][2 * u + 1]);
#pragma unroll
    for (int u = 0; u < 2; ++u) tq_mma<false>(small[0][u], a[0], b[2][2 * u], b[2][2 * u + 1]);
}

// Grid (sequence, head, 16 columns of the state); four warps multiply, a fifth brings K and T.  A link is a chain of three products that
// pass through shared memory, and what the warps read of it: every right operand serves 16 rows only.  A warp holds a quarter of the
// state's rows, so its share of K S has the state as left operand as it lies in the registers, and the shares are added up.  (With all rows of
// the state in shared memory and the tokens shared out over the warps a link took 2.6 us, over eight warps 2.8.)
template <int DK, int DV>
__global__ void __launch_bounds__(32 * (CHAIN_WARPS + 1), 1)
delta_chain_kernel(Scratch io, const float* __restrict__ xv, int C, int v_off, float* __restrict__ state, long long slot_stride,
                   const int* __restrict__ slots, int heads, int kv_heads, int chunk0, int group, const int* __restrict__ cu_seqlens,
                   int* __restrict__ status) {
    tq_grid_wait();                    // everything below may read what the previous kernel wrote
    tq_grid_launch_dependents();       // the next kernel's CTAs may move in as SMs free up
    using F = Cfg<DK, DV>;
    extern __shared__ uint8_t smem_raw[];
    constexpr int KS = F::K_STAGES, TS = F::T_STAGES;
    const uint32_t base = (tq_smem_u32(smem_raw) + 127u) & ~127u, tbase = base + KS * F::IMAGE, zp = tbase + TS * T_IMAGE, up = zp + 3 * F::U_PART;
    float* X = reinterpret_cast<float*>(smem_raw + (up + 3 * F::U_PART - tq_smem_u32(smem_raw)));      // the warps' shares of K S, [warp][16 columns][64 tokens]
    __shared__ int s_first, s_abort, s_cols[2][16];           // s_cols: a link's first value that is not finite, per column
    __shared__ __align__(8) uint64_t s_bars[2 * (F::K_STAGES + F::T_STAGES)];
    const int s = blockIdx.x, h = blockIdx.y, v0 = blockIdx.z * 16, g = h / (heads / kv_heads);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    auto k_full = [&](int st) { return tq_smem_u32(&s_bars[st]); };
    auto k_done = [&](int st) { return tq_smem_u32(&s_bars[KS + st]); };
    auto t_full = [&](int st) { return tq_smem_u32(&s_bars[2 * KS + st]); };
    auto t_done = [&](int st) { return tq_smem_u32(&s_bars[2 * KS + TS + st]); };
    if (warp == 0) {                   // chunks of the sequences before this one
        int before = 0;
        for (int i = lane; i < s; i += 32) before += (cu_seqlens[i + 1] - cu_seqlens[i] + L - 1) / L;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) before += __shfl_xor_sync(0xffffffffu, before, o);
        s_cols[lane >> 4][lane & 15] = L;
        if (lane == 0) {
            s_first = before;
            s_abort = 0;
            for (int i = 0; i < KS; ++i) { mbar_init(k_full(i), 1); mbar_init(k_done(i), CHAIN_WARPS); }
            for (int i = 0; i < TS; ++i) { mbar_init(t_full(i), 1); mbar_init(t_done(i), CHAIN_WARPS); }
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
    }
    __syncthreads();
    // the sequence's chunks that are in the group, counted from chunk0
    const int t_begin = cu_seqlens[s], run = cu_seqlens[s + 1] - t_begin;
    const int from = max(s_first - chunk0, 0), n = min(s_first + (run + L - 1) / L - chunk0, group) - from;
    if (n <= 0) return;
    if (warp == CHAIN_WARPS) {
        if (lane == 0) {
            auto load = [&](uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
                bulk_load(dst, src, bytes, bar);
            };
            int nk = 0, nt = 0;
            for (int i = 0; i < n; ++i) {
                if (i >= KS && !mbar_wait(k_done(i % KS), (uint32_t)(i / KS - 1) & 1u, &s_abort)) break;
                load(base + i % KS * F::IMAGE, io.k + ((size_t)(from + i) * kv_heads + g) * F::IMAGE, F::IMAGE, k_full(i % KS));
                ++nk;
                if (i >= TS && !mbar_wait(t_done(i % TS), (uint32_t)(i / TS - 1) & 1u, &s_abort)) break;
                load(tbase + i % TS * T_IMAGE, io.t + ((size_t)(from + i) * heads + h) * T_IMAGE, T_IMAGE, t_full(i % TS));
                ++nt;
            }
            if (s_abort) {             // no copy lands after the CTA is gone
                for (int j = max(nk - KS, 0); j < nk; ++j)
                    for (uint32_t k = 0; k < WAIT_LIMIT && !mbar_try_wait(k_full(j % KS), (uint32_t)(j / KS) & 1u); ++k) {}
                for (int j = max(nt - TS, 0); j < nt; ++j)
                    for (uint32_t k = 0; k < WAIT_LIMIT && !mbar_try_wait(t_full(j % TS), (uint32_t)(j / TS) & 1u); ++k) {}
            }
        }
    } else {
        const Lane ln(lane);
        constexpr int NT = DK / (8 * CHAIN_WARPS);              // groups of eight rows of the state that a warp holds
        const int i0 = warp * (8 * NT), s0 = 16 * warp + ln.c;  // the warp's rows of the state; the thread's tokens: s0, s0 + 1, s0 + 8, s0 + 9
        float S[NT][4];                                         // [column v0 + ln.r (+ 8)][row i0 + 8 u + ln.c (+ 1)]
        float* cell = state + (size_t)slots[s] * slot_stride + ((size_t)h * DV + v0) * DK + i0;
#pragma unroll
        for (int u = 0; u < NT; ++u)
#pragma unroll
            for (int e = 0; e < 4; ++e) S[u][e] = cell[(size_t)(ln.r + 8 * (e >> 1)) * DK + 8 * u + ln.c + (e & 1)];
        // what a link needs besides, on its way while the link before is computed
        float V[2][4], last, bad;
        float2 A[2], beta[2], left[2];
        auto ask = [&](int i) {
            const float* d = io.d + ((size_t)(from + i) * heads + h) * N_ROW;
            const int t0 = (from + chunk0 - s_first + i) * L, held = min(L, run - t0);
            const float* v_at = xv + (size_t)(t_begin + t0 + s0) * C + v_off + h * DV + v0 + ln.r;
#pragma unroll
            for (int u = 0; u < 2; ++u) {
#pragma unroll
                for (int e = 0; e < 4; ++e) V[u][e] = s0 + 8 * u + (e & 1) < held ? v_at[(size_t)(8 * u + (e & 1)) * C + 8 * (e >> 1)] : 0.f;
                A[u] = *reinterpret_cast<const float2*>(d + N_A + s0 + 8 * u);
                beta[u] = *reinterpret_cast<const float2*>(d + N_BETA + s0 + 8 * u);
                left[u] = *reinterpret_cast<const float2*>(d + N_D + s0 + 8 * u);
            }
            last = d[N_LAST];
            bad = d[N_BAD];
        };
        ask(0);
        for (int i = 0; i < n; ++i) {
            const size_t unit = (size_t)(from + i) * heads + h;
            const uint32_t sk = base + i % KS * F::IMAGE, tk = tbase + i % TS * T_IMAGE;
            bool ok = __all_sync(0xffffffffu, mbar_wait(k_full(i % KS), (uint32_t)(i / KS) & 1u, &s_abort));
            if (ok) {   // the warp's rows' share of (K S)^T: 16 columns x 64 tokens
                float big[8][4], small[8][4];
#pragma unroll
                for (int k = 0; k < NT / 2; ++k) {
                    uint32_t a[3][4];
#pragma unroll
                    for (int q = 0; q < 4; ++q)
                        tq_split2(S[2 * k + (q >> 1)][2 * (q & 1)], S[2 * k + (q >> 1)][2 * (q & 1) + 1], a[0][q], a[1][q], a[2][q]);
#pragma unroll
                    for (int t = 0; t < 2; ++t) {
                        uint32_t b[3][2][4];
#pragma unroll
                        for (int p = 0; p < 3; ++p)
#pragma unroll
                            for (int j = 0; j < 2; ++j) tq_ldm4(b[p][j], sk + p * F::K_PART + tq_piece<DK>(32 * t + 16 * j + ln.b_row, i0 / 8 + 2 * k + ln.b_c));
                        if (k == 0) tq_six<4, true, true>(big + 4 * t, small + 4 * t, a, b); else tq_six<4, false, false>(big + 4 * t, small + 4 * t, a, b);
                    }
                }
                float* x = X + (warp * 16 + ln.r) * XLD + ln.c;
#pragma unroll
                for (int u = 0; u < 8; ++u)
#pragma unroll
                    for (int r = 0; r < 2; ++r)
                        *reinterpret_cast<float2*>(x + 8 * r * XLD + 8 * u) = make_float2(big[u][2 * r] + small[u][2 * r], big[u][2 * r + 1] + small[u][2 * r + 1]);
            }
            float* s_at = io.s + (unit * DV + v0 + ln.r) * DK + i0 + ln.c;
#pragma unroll
            for (int u = 0; u < NT; ++u)
#pragma unroll
                for (int r = 0; r < 2; ++r) *reinterpret_cast<float2*>(s_at + (size_t)8 * r * DK + 8 * u) = make_float2(S[u][2 * r], S[u][2 * r + 1]);
            if (ok) ok = __all_sync(0xffffffffu, mbar_wait(t_full(i % TS), (uint32_t)(i / TS) & 1u, &s_abort));
            if (chain_any(!ok)) break;
#pragma unroll
            for (int u = 0; u < 2; ++u)
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    float2 x[CHAIN_WARPS];
#pragma unroll
                    for (int w = 0; w < CHAIN_WARPS; ++w) x[w] = *reinterpret_cast<const float2*>(X + (w * 16 + ln.r + 8 * r) * XLD + s0 + 8 * u);
                    auto z = [&](int e, float b, float a, float ks) {
                        float v = V[u][2 * r + e];
                        if (!isfinite(v)) { atomicMin(&s_cols[i & 1][ln.r + 8 * r], s0 + 8 * u + e); v = 0.f; }
                        return b * (v - a * ks);
                    };
                    tq_put2<L>(zp, F::U_PART, ln.r + 8 * r, s0 + 8 * u, z(0, beta[u].x, A[u].x, (x[0].x + x[1].x) + (x[2].x + x[3].x)),
                               z(1, beta[u].y, A[u].y, (x[0].y + x[1].y) + (x[2].y + x[3].y)));
                }
            const float2 d_left[2] = {left[0], left[1]};
            const float left_last = bad < (float)L ? NAN : last;     // a token that is not finite: so is the state behind it
            if (i + 1 < n) ask(i + 1);
            chain_sync();
            const float d_last[2] = {s_cols[i & 1][ln.r] < L ? NAN : left_last, s_cols[i & 1][ln.r + 8] < L ? NAN : left_last};
            if (tid < 16) {
                io.d[unit * N_ROW + N_COLS + v0 + tid] = (float)s_cols[i & 1][tid];
                s_cols[(i + 1) & 1][tid] = L;
            }
            {   // U^T = Z^T T^T.  (T is lower triangular, but the last warp needs all of its row, and
                // the others would wait for it)
                float big[2][4], small[2][2][4];
                float* u_at = io.u + unit * DV * L + (size_t)(v0 + ln.r) * L + s0;
                uint32_t a[L / 16][3][4], b[L / 16][3][4];       // all of them asked for before the first product
#pragma unroll
                for (int k = 0; k < L / 16; ++k)
#pragma unroll
                    for (int p = 0; p < 3; ++p) {
                        tq_ldm4(a[k][p], zp + p * F::U_PART + tq_piece<L>(ln.a_row, 2 * k + ln.a_c));
                        tq_ldm4(b[k][p], tk + p * T_PART + tq_piece<L>(16 * warp + ln.b_row, 2 * k + ln.b_c));
                    }
#pragma unroll
                for (int k = 0; k < L / 16; ++k) {
                    if (k == 0) six2<true>(big, small, a[k], b[k]); else six2<false>(big, small, a[k], b[k]);
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(t_done(i % TS));
#pragma unroll
                for (int u = 0; u < 2; ++u)
#pragma unroll
                    for (int r = 0; r < 2; ++r) {
                        auto sum = [&](int e) { return big[u][e] + (small[0][u][e] + small[1][u][e]); };
                        const float2 x = make_float2(sum(2 * r), sum(2 * r + 1));
                        *reinterpret_cast<float2*>(u_at + 8 * r * L + 8 * u) = x;
                        tq_put2<L>(up, F::U_PART, ln.r + 8 * r, s0 + 8 * u, x.x * d_left[u].x, x.y * d_left[u].y);
                    }
            }
            chain_sync();
            {
                float big[NT][4], small[NT][4];
#pragma unroll
                for (int k = 0; k < L / 16; ++k) {
                    uint32_t a[3][4], b[3][NT / 2][4];
#pragma unroll
                    for (int p = 0; p < 3; ++p) {
                        tq_ldm4(a[p], up + p * F::U_PART + tq_piece<L>(ln.a_row, 2 * k + ln.a_c));
#pragma unroll
                        for (int j = 0; j < NT / 2; ++j) tq_ldm4t(b[p][j], sk + p * F::K_PART + tq_piece<DK>(16 * k + ln.t_row, i0 / 8 + 2 * j + ln.t_c));
                    }
                    if (k == 0) tq_six<NT, true, true>(big, small, a, b); else tq_six<NT, false, false>(big, small, a, b);
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(k_done(i % KS));
#pragma unroll
                for (int u = 0; u < NT; ++u)
#pragma unroll
                    for (int e = 0; e < 4; ++e) S[u][e] = d_last[e >> 1] * S[u][e] + (big[u][e] + small[u][e]);
            }
        }
#pragma unroll
        for (int u = 0; u < NT; ++u)
#pragma unroll
            for (int e = 0; e < 4; ++e) cell[(size_t)(ln.r + 8 * (e >> 1)) * DK + 8 * u + ln.c + (e & 1)] = S[u][e];
    }
    __syncthreads();
    if (tid == 0 && s_abort) atomicExch(status, 1);
}

template <int DK, int DV>
__global__ void __launch_bounds__(THREADS, 2)
delta_outputs_kernel(Rows rows, Scratch in, float* __restrict__ y, int chunk0, const int* __restrict__ cu_seqlens, int n_seqs) {
    tq_grid_wait();                    // everything below may read what the previous kernel wrote
    tq_grid_launch_dependents();       // the next kernel's CTAs may move in as SMs free up
    using F = Cfg<DK, DV>;
    extern __shared__ __align__(128) uint8_t smem[];
    const uint32_t sq = tq_smem_u32(smem), sk = sq + F::IMAGE;                     // Q; K, then 32 columns of the state and of U at a time
    float* m = reinterpret_cast<float*>(smem + F::IMAGE + F::WORK);
    __shared__ Chunk s_chunk;
    __shared__ float s_g[L], s_A[L];
    const int h = blockIdx.y, g = h / (rows.heads / rows.kv_heads);
    const Chunk c = find_chunk(chunk0 + blockIdx.x, cu_seqlens, n_seqs, &s_chunk);
    if (c.n == 0) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const Lane ln(lane);
    const size_t unit = (size_t)blockIdx.x * rows.heads + h;
    const float* tok = rows.at + (size_t)c.t0 * rows.stride;
    {
        const uint8_t* image = in.k + ((size_t)blockIdx.x * rows.kv_heads + g) * F::IMAGE;
#pragma unroll 8
        for (int i = tid; i < F::IMAGE / 16; i += THREADS)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(sk + i * 16), "l"(image + (size_t)i * 16) : "memory");
        if (tid < L) {
            const float a = tid < c.n ? tok[(size_t)tid * rows.stride + 2 * rows.kv_heads * DK + h] : 1.f;
            s_g[tid] = isfinite(a) ? a : 1.f;
        }
        constexpr int Q = DK / 4, QN = L * Q / THREADS;
        float4 q4[QN];                 // all of them asked for before the first is used
#pragma unroll
        for (int i = 0; i < QN; ++i) {
            const int t = (i * THREADS + tid) / Q;
            q4[i] = t < c.n ? *reinterpret_cast<const float4*>(tok + (size_t)t * rows.stride + (rows.kv_heads + g) * DK + tid % Q * 4) : zero4();
        }
#pragma unroll
        for (int i = 0; i < QN; ++i) tq_put4<DK>(sq, F::K_PART, (i * THREADS + tid) / Q, tid % Q * 4, q4[i]);
        asm volatile("cp.async.wait_all;" ::: "memory");
    }
    __syncthreads();
    decays(m, s_g, s_A, nullptr);
    // the first 32 columns of the state and of U are on their way meanwhile
    constexpr int SN = 32 * DK / 4 / THREADS, UN = 32 * L / 4 / THREADS;
    float4 ns[SN], nu[UN];
    auto ask = [&](int q) {
        const float4* s_at = reinterpret_cast<const float4*>(in.s + (unit * DV + 32 * q) * DK) + tid;
        const float4* u_at = reinterpret_cast<const float4*>(in.u + (unit * DV + 32 * q) * L) + tid;
#pragma unroll
        for (int i = 0; i < SN; ++i) ns[i] = s_at[i * THREADS];
#pragma unroll
        for (int i = 0; i < UN; ++i) nu[i] = u_at[i * THREADS];
    };
    ask(0);
    __syncthreads();
    // per column the first value that is not finite, in the place of the decays, which have been used (two CTAs an SM fit with no room for more)
    uint8_t* cols = reinterpret_cast<uint8_t*>(s_g);
    const int bad = (int)in.d[unit * N_ROW + N_BAD];
    if (tid < DV) cols[tid] = (uint8_t)min(bad, (int)in.d[unit * N_ROW + N_COLS + tid]);
    uint32_t P[L / 16][3][4];          // D o Q K^T as left operands
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
                const float* d = m + (16 * warp + ln.r + 8 * r) * LD + 32 * grp + 8 * u + ln.c;
                auto val = [&](int e) { return grp > warp >> 1 ? 0.f : d[e & 1] * ((DK > 64 ? first[u][e] + big[u][e] : big[u][e]) + small[u][e]); };
                const float x = val(2 * r), z = val(2 * r + 1);
                const int at = 2 * (u & 1) + r;
                if (grp == 0) tq_split2(x, z, P[u >> 1][0][at], P[u >> 1][1][at], P[u >> 1][2][at]);
                else tq_split2(x, z, P[2 + (u >> 1)][0][at], P[2 + (u >> 1)][1][at], P[2 + (u >> 1)][2][at]);
            }
    }
    const uint32_t su = sk + 3 * F::SQ_PART;
    const float A[2] = {s_A[16 * warp + ln.r], s_A[16 * warp + ln.r + 8]};
    for (int q = 0; q < DV / 32; ++q) {
        __syncthreads();               // what was there has been used
#pragma unroll
        for (int i = 0; i < SN; ++i) { const int at = (i * THREADS + tid) * 4; tq_put4<DK>(sk, F::SQ_PART, at / DK, at % DK, ns[i]); }
#pragma unroll
        for (int i = 0; i < UN; ++i) { const int at = (i * THREADS + tid) * 4; tq_put4<L>(su, F::UQ_PART, at / L, at % L, nu[i]); }
        if (q + 1 < DV / 32) ask(q + 1);
        __syncthreads();
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
                for (int j = 0; j < 2; ++j) tq_ldm4(b[p][j], su + p * F::UQ_PART + tq_piece<L>(16 * j + ln.b_row, 2 * k + ln.b_c));
            if (k == 0) tq_six<4, true, true>(big, small, P[k], b); else tq_six<4, false, false>(big, small, P[k], b);
        }
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const int t = 16 * warp + ln.r + 8 * r;
            float* at = y + ((size_t)(c.t0 + t) * rows.heads + h) * DV + 32 * q + ln.c;
            if (t < c.n)
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    auto sum = [&](int e) { return t < cols[32 * q + 8 * u + ln.c + (e & 1)] ? o[u][e] + (big[u][e] + small[u][e]) : NAN; };
                    *reinterpret_cast<float2*>(at + 8 * u) = make_float2(sum(2 * r), sum(2 * r + 1));
                }
        }
    }
}

template <int DK, int DV>
int launch(const Rows& rows, const float* xv, int C, int v_off, const Scratch& scratch, float* state, long long slot_stride, float* y, int chunks,
           int group, int n_seqs, const int* cu, const int* slots, int* status, cudaStream_t stream) {
    using F = Cfg<DK, DV>;
    static std::atomic<unsigned long long> asked[3];
    cudaError_t e = tq_reserve_smem(delta_solve_kernel<DK, DV>, F::SOLVE_BYTES, asked[0]);
    if (e == cudaSuccess) e = tq_reserve_smem(delta_chain_kernel<DK, DV>, F::CHAIN_BYTES, asked[1]);
    if (e == cudaSuccess) e = tq_reserve_smem(delta_outputs_kernel<DK, DV>, F::OUT_BYTES, asked[2]);
    if (e != cudaSuccess) TQ_FAIL(-1, "delta_chunks: %d bytes of shared memory refused: %s", F::CHAIN_BYTES, cudaGetErrorString(e));
    for (int chunk0 = 0; chunk0 < chunks; chunk0 += group) {
        const int n = chunks - chunk0 < group ? chunks - chunk0 : group;
        tq_launch(dim3(n, rows.heads), THREADS, F::SOLVE_BYTES, stream)(delta_solve_kernel<DK, DV>, rows, scratch, chunk0, cu, n_seqs);
        tq_launch(dim3(n_seqs, rows.heads, DV / 16), 32 * (CHAIN_WARPS + 1), F::CHAIN_BYTES, stream)(delta_chain_kernel<DK, DV>, scratch, xv, C, v_off, state,
            slot_stride, slots, rows.heads, rows.kv_heads, chunk0, n, cu, status);
        tq_launch(dim3(n, rows.heads), THREADS, F::OUT_BYTES, stream)(delta_outputs_kernel<DK, DV>, rows, scratch, y, chunk0, cu, n_seqs);
    }
    TQ_CHECK_LAUNCH("delta_chunks");
    return 0;
}

}  // namespace

// Bytes of scratch that a group of chunks takes.
TQ_EXPORT long long tq_delta_chunks_bytes(int group, int heads, int kv_heads, int dk, int dv) {
    return (long long)group * (6ll * L * dk * kv_heads + heads * (T_IMAGE + 4ll * ((long long)dv * L + (long long)dv * dk + N_ROW)));
}

// rows [T, R] as tq_delta_prepare lays them out (one decay per head), values from xv's rows of C floats, column v_off; state: the sequences'
// [heads][dv][dk] at slots[s] * slot_stride, renewed; y [T, heads * dv].  chunks: at least the sum of ceil(run / 64), group: of them at
// a time; scratch of tq_delta_chunks_bytes(group, ...).  status: one int, set to 1 if a bounded wait ran out.
TQ_EXPORT int tq_delta_chunks(const float* rows, int R, const float* xv, int C, int v_off, float* state, long long slot_stride, float* y, void* scratch,
                              int chunks, int group, int n_seqs, int heads, int kv_heads, int dk, int dv, const int* cu_seqlens, const int* slots,
                              int* status, cudaStream_t stream) {
    if (n_seqs == 0 || chunks == 0) return 0;
    TQ_REQUIRE(heads >= 1 && kv_heads >= 1 && heads % kv_heads == 0 && heads <= 65535 && group >= 1, "delta_chunks: %d heads on %d query/key heads, groups of %d chunks", heads, kv_heads, group);
    TQ_REQUIRE(R % 4 == 0 && C % 4 == 0 && v_off % 4 == 0 && ((uintptr_t)rows & 15) == 0 && ((uintptr_t)xv & 15) == 0 && ((uintptr_t)y & 15) == 0
               && ((uintptr_t)scratch & 15) == 0, "delta_chunks: rows of %d and %d floats are not aligned to 16 bytes", R, C);
    TQ_REQUIRE(v_off >= 0 && v_off + heads * dv <= C && 2 * kv_heads * dk + 2 * heads + kv_heads <= R, "delta_chunks: the heads lie outside their rows");
    TQ_REQUIRE(status != nullptr, "delta_chunks: a status word is required");
    Scratch s;
    s.k = (uint8_t*)scratch;
    s.t = s.k + (size_t)group * kv_heads * 6 * L * dk;
    s.u = (float*)(s.t + (size_t)group * heads * T_IMAGE);
    s.s = s.u + (size_t)group * heads * dv * L;
    s.d = s.s + (size_t)group * heads * dv * dk;
    const Rows r{rows, R, heads, kv_heads};
#define DELTA_CASE(DK_, DV_) if (dk == DK_ && dv == DV_) return launch<DK_, DV_>(r, xv, C, v_off, s, state, slot_stride, y, chunks, group, n_seqs, cu_seqlens, slots, status, stream);
    DELTA_CASE(64, 64) DELTA_CASE(64, 128) DELTA_CASE(128, 64) DELTA_CASE(128, 128)
#undef DELTA_CASE
    TQ_FAIL(-2, "delta_chunks: keys of %d and values of %d elements", dk, dv);
}
