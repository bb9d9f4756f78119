// Causal attention for prompts on the 5th-generation tensor cores: S = Q K^T and O = P V as
// tcgen05.mma with the accumulators in tensor memory, Q/K/V tiles brought in by TMA straight from
// the query buffer and the paged cache, online softmax in fp32 registers.
//
// Same mathematics as the exact kernels (csrc/attention.cu, csrc/bias_attention.cu) and as the reference's
// per-token loop (src/engine/tq_transformer.c:1909-1936 scores with scale 1/sqrt(hd), :1960 softmax, :2183-2191
// weighted sum of V, head h reading KV head h/(nh/nkv) :1679, window start :1646-1654): scores,
// running maximum, sum and the output accumulator are fp32; only P is rounded to bf16 to feed the
// second product.  One kernel serves every softmax attention over rows: keys and values of 64 or 128 elements each
// in planes of their own or side by side in a row, a window (with a sequence's first positions kept) or cells of
// positions, a cap on the scores, a bias per distance, a sink in the denominator.  Keys may also be 192 long, and lie
// in plain matrices instead of pages, the last 64 elements shared by all heads (latent attention's prompts).
//
// A unit of work = two query tiles of 128 rows (slots A and B) that walk the same keys in tiles of 128 (= two cache
// pages; the last tile may hold one): two heads of one key/value head, or two tiles of one head's run.  Persistent
// CTAs, one per SM, take units until none is left:
//   warps 0..3    softmax of slot A, a thread per row; warps 4..7 of slot B: read S, mask, online softmax, write P
//                 (bf16) over S in tensor memory, where the second product takes it as its left operand.  O stays in
//                 tensor memory: it is rescaled there when a tile's maximum is larger than the one the row's exponentials are
//                 taken against (attention over rows), or larger by more than 2^8 (until then P is simply larger, at most
//                 256, and the row's sum carries the same factor)
//   warp 8        TMA: Q of both slots, then K and V pages through rings that both slots read
//   warp 9        owns tensor memory, issues  O += P V  of a slot's tile and right behind it  S = Q K^T  of its next
// The two slots take turns: while one's scores are exponentiated the other's products run, which is what bounds a
// tile pair: 2 x 16,384 exponentials at 16 a cycle and SM (2,048 cycles) beside 32 products of 128 x 128 x 16 (2,048).
// Neither is reached: the tensor pipe is active 31 % of the plain form's time, the exponentials' unit as long; what remains is the turn
// from one to the other (a slot's softmax, then its products, some 1,500 cycles).  One slot (eight warps on one tile, P
// through shared memory, products issued by one lane) took 6,000 cycles a tile.
// Prompts of 682 + 1,365 + 2,049 tokens, 16 heads of 128, the replaced kernels (one slot; mma.sync for rows) and this one, us: 16 kv
// heads, plain 79 / 52; rows with 4 kv heads, plain 151 / 64, cells of 512 111 / 36, cap 50 441 / 77, cap 4 with large scores 441 / 119;
// 2,048 tokens, window 1,024 with a bias 89 / 47.
// Every wait on an mbarrier is bounded; a wait that runs out sets *status and the CTA
// leaves cleanly.
#include <cuda.h>
#include "common.cuh"

TQ_DEFINE_LAST_ERROR

namespace {

constexpr int BM = 128;      // query rows per CTA
// eight softmax warps; TMA warp, MMA warp and two that only fill their warpgroup.  Registers: 384 threads start with 168 each,
// the last warpgroup gives back all but 72 and the softmax warps take 216 (256 * 216 + 128 * 72 = 384 * 168)
constexpr int THREADS = 384;
constexpr uint32_t WAIT_LIMIT = 1u << 20;
constexpr uint64_t WAIT_NS = 2000000000ull;

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}
__device__ __forceinline__ uint64_t global_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
    uint64_t t0 = 0;
    for (uint32_t i = 0; i < WAIT_LIMIT; ++i) {
        if (mbar_try_wait(bar, parity)) return true;
        if ((i & 255u) == 255u) {
            if (*abort_flag) return false;
            const uint64_t now = global_ns();
            if (t0 == 0) t0 = now;
            else if (now - t0 > WAIT_NS) break;
        }
    }
    *abort_flag = 1;
    return false;
}
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
        ::"r"(dst), "l"((uint64_t)map), "r"(bar), "r"(x), "r"(y) : "memory");
}
// K-major operand, rows of 128 bytes, 128-byte swizzle (see csrc/gemm_tc.cu)
__device__ __forceinline__ uint64_t desc_k_major(uint32_t addr) {
    return (uint64_t)((addr & 0x3FFFFu) >> 4) | (1ull << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
// MN-major operand (V as stored: one key per 128-byte row of 64 head elements): leading byte offset =
// distance between blocks of 64 head elements, stride byte offset = eight keys (1024 bytes)
__device__ __forceinline__ uint64_t desc_mn_major(uint32_t addr, uint32_t lbo_bytes) {
    return (uint64_t)((addr & 0x3FFFFu) >> 4) | ((uint64_t)((lbo_bytes >> 4) & 0x3FFF) << 16) |
           ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
// kind::f16 instruction descriptor: D fp32, A/B bf16, M 128, N n; b_mn: B is MN-major
__device__ __forceinline__ uint32_t idesc(int n, int b_mn) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)b_mn << 16) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
}
// One lane of the warp, the same each time.  The products and commits below are issued under its predicate by code the
// whole warp runs, so that their operands stay in uniform registers: issued from a one-lane branch each product cost
// some 140 cycles of moving its descriptors there, more than the product itself.
__device__ __forceinline__ uint32_t elect_one() {
    uint32_t e;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(e));
    return e;
}
__device__ __forceinline__ void umma(uint32_t tmem_d, uint64_t a, uint64_t b, uint32_t id, uint32_t accumulate, uint32_t elected) {
    asm volatile(
        "{\n\t.reg .pred p, e;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "setp.ne.b32 e, %5, 0;\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(a), "l"(b), "r"(id), "r"(accumulate), "r"(elected) : "memory");
}
// the same with the left operand in tensor memory: a lane per row, two K elements in each 32-bit column
__device__ __forceinline__ void umma_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t b, uint32_t id, uint32_t accumulate, uint32_t elected) {
    asm volatile(
        "{\n\t.reg .pred p, e;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "setp.ne.b32 e, %5, 0;\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(b), "r"(id), "r"(accumulate), "r"(elected) : "memory");
}
__device__ __forceinline__ void umma_commit(uint32_t bar, uint32_t elected) {
    asm volatile(
        "{\n\t.reg .pred e;\n\t"
        "setp.ne.b32 e, %1, 0;\n\t"
        "@e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(bar), "r"(elected) : "memory");
}
// 2^x, one MUFU instruction; 2^-inf = 0
__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&v)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
          "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]),
          "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]),
          "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
        : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&v)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
          "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(taddr));
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&v)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
        ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]),
          "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
        : "memory");
}
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&v)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
        "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
        ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]),
          "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(v[16]), "r"(v[17]),
          "r"(v[18]), "r"(v[19]), "r"(v[20]), "r"(v[21]), "r"(v[22]), "r"(v[23]), "r"(v[24]), "r"(v[25]), "r"(v[26]),
          "r"(v[27]), "r"(v[28]), "r"(v[29]), "r"(v[30]), "r"(v[31])
        : "memory");
}
constexpr int PAGE = 64;     // tokens per cache page
constexpr int BN = 128;      // keys per tile = two cache pages (a unit's last tile may hold one)
constexpr float LOG2E = 1.4426950408889634f;

template <int DK, int DV>
struct Cfg {
    static constexpr int KB = DK / 64, VB = DV / 64;       // 64-element (128-byte) column blocks of a key and of a value
    static constexpr int Q_BYTES = BM * DK * 2;            // one slot's queries
    static constexpr int K_BYTES = BN * DK * 2, V_BYTES = BN * DV * 2;
    static constexpr int K_PAGE = PAGE * DK * 2, V_PAGE = PAGE * DV * 2;
    static constexpr int KST = 2, VST = DK > 128 ? 1 : 2;  // tiles of K and of V in flight
    static constexpr int TILE_BYTES = 2 * Q_BYTES + KST * K_BYTES + VST * V_BYTES;
    static constexpr int SMEM_BYTES = TILE_BYTES + 1024 /* alignment slack */ + 256 /* barriers */;
    static constexpr int TMEM_COLS = 512;                  // S (with P over it) and O of both slots: 2 x 128 + 2 x DV
    static_assert((DK == 64 || DK == 128 || DK == 192) && (DV == 64 || DV == 128), "key and value sizes");
    static_assert(SMEM_BYTES <= 227 * 1024, "shared memory");
};

// What a launch looks like.  A page's key row: page * kp + kv head * kg in map_k, its value row the same + v_plane in
// map_v; the head's columns begin at kv head * kc in map_k and at v_col + kv head * vc in map_v.  table null: keys lie
// densely, position 64 p of sequence s as page page_base[s] + p.
struct Shape {
    int nh, nkv, n_seqs, n_qt, pairing;
    int kp, kg, v_plane, kc, vc, v_col, k_blocks, r_col;   // k_blocks: 64-element blocks of a key that map_k holds; the rest come from
                                                           // map_r, whose columns begin at r_col
    int table_stride, n_pages, window, keep_first, cell, far;
    float scale, softcap;
};
enum { PAIR_HEADS, PAIR_ROWS };

// Two tiles of 128 consecutive query tokens of one sequence, each of one query head.
struct Unit { int seq, g, p0, first, kept, n_pages, n_tiles, h[2], t0[2], rows[2], p_first[2], n[2]; bool valid; };

// The query tile is the slowest index, last tiles (which see the most keys) first.
__device__ __forceinline__ Unit unit_of(int unit, const Shape& S, const int* cu_seqlens, const int* seq_start) {
    Unit u;
    const int hs = S.pairing == PAIR_HEADS ? S.nh / 2 : S.nh;
    const int per = S.n_seqs * hs, x = unit / per, rem = unit - x * per;
    u.seq = rem / hs;
    const int hx = rem - u.seq * hs;
    const int t_begin = cu_seqlens[u.seq], run = cu_seqlens[u.seq + 1] - t_begin;
    const int start = seq_start[u.seq], tiles = (run + BM - 1) / BM;
    int qa, qb;                                            // the slots' query tiles (-1: none)
    if (S.pairing == PAIR_HEADS) {
        qa = qb = S.n_qt - 1 - x;
        u.h[0] = 2 * hx; u.h[1] = 2 * hx + 1;
        u.valid = qa < tiles;
    } else {
        u.h[0] = u.h[1] = hx;
        qa = 2 * ((S.n_qt + 1) / 2 - 1 - x);
        qb = qa + 1 < tiles ? qa + 1 : -1;
        u.valid = qa < tiles;
    }
    u.g = u.h[0] / (S.nh / S.nkv);
    u.p0 = start + qa * BM;
    u.first = S.cell > 0 ? (u.p0 - u.p0 % S.cell) / PAGE : (S.window > 0 ? max(0, u.p0 + 1 - S.window) / PAGE : 0);
    u.kept = S.window > 0 && S.cell == 0 ? min((S.keep_first + PAGE - 1) / PAGE, u.first) : 0;
    u.n_pages = 0;
#pragma unroll
    for (int s = 0; s < 2; ++s) {
        const int q = s ? qb : qa;
        u.t0[s] = t_begin + q * BM;
        u.rows[s] = min(BM, run - q * BM);
        u.p_first[s] = start + q * BM;
        const int pages = u.kept + (u.p_first[s] + u.rows[s] - 1) / PAGE - u.first + 1;
        u.n[s] = q < 0 || !u.valid ? 0 : (pages + 1) / 2;
        if (u.n[s]) u.n_pages = max(u.n_pages, pages);
    }
    u.n_tiles = max(u.n[0], u.n[1]);
    return u;
}
// the n-th page a unit walks
__device__ __forceinline__ int page_at(const Unit& u, int n) { return n < u.kept ? n : u.first + n - u.kept; }

__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return tq_unpack2(tq_fma2(tq_pack2(a.x, a.y), tq_pack2(b.x, b.y), tq_pack2(c.x, c.y))); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return tq_unpack2(tq_mul2(tq_pack2(a.x, a.y), tq_pack2(b.x, b.y))); }
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return tq_unpack2(tq_add2(tq_pack2(a.x, a.y), tq_pack2(b.x, b.y))); }

__device__ __forceinline__ float max3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
// the largest of 32 values and `from`
__device__ __forceinline__ float max_of(const uint32_t (&v)[32], float from) {
    float top[2] = {from, __uint_as_float(v[0])};
#pragma unroll
    for (int c = 1; c < 31; c += 2) top[c / 2 % 2] = max3(top[c / 2 % 2], __uint_as_float(v[c]), __uint_as_float(v[c + 1]));
    return max3(top[0], top[1], __uint_as_float(v[31]));
}

// softcap * tanh(s * scale / softcap) of 32 scores: the odd series up to x^9, x = s * scale / softcap, where every x of the
// warp's rows lies below a quarter (the first term left out is 9e-9 of the result there), tanhf beyond, as in the decode kernels.
// Relative error against 64 bits, a million scores each, caps of 4 to 50: the series at most 1.1e-7 (root mean square 3.5e-8), tanhf
// 2.4e-7 (5e-8) over the same scores and 2.8e-7 (7.5e-8) beyond a quarter, where 1 - 2 / (e^2x + 1) of fast intrinsics was off by
// 7.5e-7 (1.2e-7).  s * (k + k_low): with a division a score the code outgrew the instruction caches (500 us for the case of 119 above).
// p: the series' coefficients in powers of s^2, times scale; below: the |x| up to which it serves (a cap so small against the
// scale that they overflow: none).
struct CapSeries { float p[5], k, k_low, cap, below; };
__device__ __forceinline__ CapSeries cap_series(float scale, float cap) {
    CapSeries r;
    r.cap = cap;
    r.k = scale / cap;
    r.k_low = fmaf(-r.k, cap, scale) / cap;        // what the quotient's rounding left out: s * (k + k_low) is rounded once
    const float k2 = r.k * r.k;
    r.p[0] = scale;
    r.p[1] = -1.0f / 3.0f * k2 * scale;
    r.p[2] = 2.0f / 15.0f * k2 * k2 * scale;
    r.p[3] = -17.0f / 315.0f * k2 * k2 * k2 * scale;
    r.p[4] = 62.0f / 2835.0f * k2 * k2 * k2 * k2 * scale;
    r.below = fabsf(r.p[4]) < INFINITY ? 0.25f : 0.0f;
    return r;
}
__device__ __forceinline__ void cap_scores(uint32_t (&v)[32], const CapSeries& s) {
    float top = 0.f;
#pragma unroll
    for (int c = 0; c < 32; c += 2) top = max3(top, fabsf(__uint_as_float(v[c])), fabsf(__uint_as_float(v[c + 1])));
    // (the maximum passes over NaN: such a score stays NaN in either form)
    if (!__any_sync(0xffffffffu, !(top * fabsf(s.k) < s.below))) {
#pragma unroll
        for (int c = 0; c < 32; c += 2) {
            const float2 x = make_float2(__uint_as_float(v[c]), __uint_as_float(v[c + 1])), x2 = mul2(x, x);
            float2 t = make_float2(s.p[4], s.p[4]);
#pragma unroll
            for (int j = 3; j >= 0; --j) t = fma2(x2, t, make_float2(s.p[j], s.p[j]));
            t = mul2(x, t);
            v[c] = __float_as_uint(t.x);
            v[c + 1] = __float_as_uint(t.y);
        }
    } else {
#pragma unroll
        for (int c = 0; c < 32; ++c) {
            const float f = __uint_as_float(v[c]), finite = fminf(fmaxf(f, -3e38f), 3e38f);      // an infinite score is the cap
            v[c] = __float_as_uint(s.cap * tanhf(fmaf(f, s.k, finite * s.k_low)));
        }
    }
}

// ROWS: the form of attention over rows.  Scores may pass through a cap and/or a bias per distance, and a row's largest weight is
// exactly one at the end of each tile; the other form (plain and latent attention) takes plain scores and keeps a maximum until it is
// outgrown by 2^8.
template <int DK, int DV, bool ROWS>
__global__ void __launch_bounds__(THREADS, 1)
attention_prefill_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                         const __grid_constant__ CUtensorMap map_r, const __grid_constant__ CUtensorMap map_v,
                         const __grid_constant__ Shape S, const int* __restrict__ cu_seqlens, const int* __restrict__ seq_start,
                         const int* __restrict__ page_table, const int* __restrict__ page_base,
                         const float* __restrict__ bias_t, const float* __restrict__ sink,
                         __nv_bfloat16* __restrict__ out, int* __restrict__ status) {
    tq_grid_wait();                    // everything below may read what the previous kernel wrote
    using C = Cfg<DK, DV>;
    extern __shared__ uint8_t smem_raw[];
    __shared__ int s_abort;
    __shared__ uint32_t s_tmem_base;
    __shared__ __align__(16) uint4 s_answer;               // the hardware's answer to a request for another block
    __shared__ int s_unit[2];                              // the units this CTA takes, two in turn
    __shared__ float s_bias[ROWS ? 8 : 1][2][ROWS ? 96 : 1];        // a warp's rows and a page's keys: the bias of their 95 distances

    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;      // the same for the whole warp, and known to be

    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    auto q_smem = [&](int s) { return base + s * C::Q_BYTES; };
    auto k_smem = [&](int s) { return base + 2 * C::Q_BYTES + s * C::K_BYTES; };
    auto v_smem = [&](int s) { return base + 2 * C::Q_BYTES + C::KST * C::K_BYTES + s * C::V_BYTES; };
    const uint32_t bars = base + C::TILE_BYTES;
    auto q_full = [&](int s) { return bars + 8u * s; };                   // a slot's Q is in / is no longer read
    auto q_free = [&](int s) { return bars + 8u * (2 + s); };
    auto k_full = [&](int s) { return bars + 8u * (4 + s); };
    auto k_empty = [&](int s) { return bars + 8u * (6 + s); };
    auto v_full = [&](int s) { return bars + 8u * (8 + s); };
    auto v_empty = [&](int s) { return bars + 8u * (10 + s); };
    auto s_ready = [&](int s) { return bars + 8u * (12 + s); };           // S of a slot's tile is done, and all products before it
    auto p_ready = [&](int s) { return bars + 8u * (14 + s); };           // P of a slot's tile is in place of its S
    auto o_done = [&](int s) { return bars + 8u * (16 + s); };            // a slot's last product of a unit is done
    auto o_free = [&](int s) { return bars + 8u * (18 + s); };            // ... and has been read
    auto n_full = [&](int s) { return bars + 8u * (20 + s); };            // a unit's number is there / has been read
    auto n_free = [&](int s) { return bars + 8u * (22 + s); };
    const uint32_t answered = bars + 8u * 24;

    if (threadIdx.x == 0) {
        s_abort = 0;
        for (int s = 0; s < 2; ++s) {
            mbar_init(q_full(s), 1); mbar_init(q_free(s), 1); mbar_init(k_full(s), 1); mbar_init(k_empty(s), 1);
            mbar_init(v_full(s), 1); mbar_init(v_empty(s), 1); mbar_init(s_ready(s), 1); mbar_init(o_done(s), 1);
            mbar_init(p_ready(s), 4); mbar_init(o_free(s), 4);            // 4: one arrival per softmax warp of the slot
            mbar_init(n_full(s), 1); mbar_init(n_free(s), 9);             // 9: the softmax warps and the MMA warp
        }
        mbar_init(answered, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 9) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(&s_tmem_base)), "r"((uint32_t)C::TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    // only now: a dependent kernel that took tensor memory first could starve a CTA of this grid that
    // had not allocated yet, and then wait forever for this grid to finish
    tq_grid_launch_dependents();
    auto tmem_s = [&](int s) { return s_tmem_base + (uint32_t)(s * BN); };              // S, and P over its first half
    auto tmem_o = [&](int s) { return s_tmem_base + (uint32_t)(2 * BN + s * DV); };

    // Every role walks the same units in the same order: the block's own first, then those of blocks that have not
    // started yet, which the TMA warp asks the hardware for (a block whose place is taken over never starts) and hands
    // on one unit ahead.  Heavy units come first in the grid, so the light ones fill the end.
    auto take_unit = [&](int k) -> int {                       // the CTA's k-th unit, -1: there is none; called by whole warps
        if (!__all_sync(0xffffffffu, mbar_wait(n_full(k & 1), (uint32_t)(k >> 1) & 1u, &s_abort))) return -1;
        const int unit = *(volatile int*)&s_unit[k & 1];
        __syncwarp();
        if (lane == 0) mbar_arrive(n_free(k & 1));
        return __shfl_sync(0xffffffffu, unit, 0);
    };
    // Tile number `ti`, counted across units, picks the K and V
    // stages and their barriers' phases; a slot's tiles and units, counted for the slot, the phases of its own.
    if (warp >= 8) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 72;");
        if (warp == 8) {
            // ------------------------------ TMA producer ------------------------------
            const uint32_t elected = elect_one();
            int ti = 0, vi = 0, asked = 0, units[2] = {0, 0};
            bool ok = true, pending = false;
            auto wait = [&](uint32_t bar, uint32_t parity) { return (bool)__all_sync(0xffffffffu, mbar_wait(bar, parity, &s_abort)); };
            auto ask = [&]() {
                if (elected) {
                    mbar_expect_tx(answered, 16);
                    asm volatile("clusterlaunchcontrol.try_cancel.async.shared::cta.mbarrier::complete_tx::bytes.b128 [%0], [%1];"
                        ::"r"(smem_u32(&s_answer)), "r"(answered) : "memory");
                }
                pending = true;
            };
            auto answer = [&]() -> int {                       // the block taken over, -1: all have started (no request follows)
                if (!wait(answered, (uint32_t)asked & 1u)) { ok = false; return -1; }
                pending = false;
                ++asked;
                uint32_t x, got;
                asm volatile(
                    "{\n\t.reg .b128 h;\n\t.reg .pred p;\n\t"
                        "ld.shared.b128 h, [%2];\n\t"
                        "clusterlaunchcontrol.query_cancel.is_canceled.pred.b128 p, h;\n\t"
                        "selp.u32 %1, 1, 0, p;\n\t"
                        "mov.u32 %0, 0;\n\t"
                        "@p clusterlaunchcontrol.query_cancel.get_first_ctaid::x.b32.b128 %0, h;\n\t}"
                    : "=r"(x), "=r"(got) : "r"(smem_u32(&s_answer)) : "memory");
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // this read before the next answer is written
                __syncwarp();
                return __shfl_sync(0xffffffffu, got ? (int)x : -1, 0);
            };
            // from a block on, the first whose unit exists (a short run has none at a late tile)
            auto settle = [&](int unit) -> int {
                while (ok && unit >= 0 && !unit_of(unit, S, cu_seqlens, seq_start).valid) { ask(); unit = answer(); }
                return ok ? unit : -1;
            };
            auto hand_on = [&](int k, int unit) {
                if (k >= 2 && !wait(n_free(k & 1), (uint32_t)((k >> 1) - 1) & 1u)) { ok = false; return; }
                if (elected) {
                    *(volatile int*)&s_unit[k & 1] = unit;
                    mbar_arrive(n_full(k & 1));
                }
                __syncwarp();
            };
            int unit = settle(blockIdx.x);
            hand_on(0, unit);
            for (int k = 0; ok && unit >= 0; ++k) {
                int following = -1;
                const Unit u = unit_of(unit, S, cu_seqlens, seq_start);
                auto load_q = [&](int s) {
                    if (!u.n[s]) return true;
                    // the products that read the slot's previous Q must be done
                    if (units[s] > 0 && !wait(q_free(s), (uint32_t)(units[s] - 1) & 1u)) return false;
                    if (elected) {
                        mbar_expect_tx(q_full(s), (uint32_t)C::Q_BYTES);
#pragma unroll
                        for (int c = 0; c < C::KB; ++c) tma_load_2d(q_smem(s) + c * (BM * 128), &map_q, u.h[s] * DK + c * 64, u.t0[s], q_full(s));
                    }
                    ++units[s];
                    return true;
                };
                ok = load_q(0);
                if (!ok) break;
                for (int i = 0; i < u.n_tiles; ++i, ++ti) {
                    // asked for at the unit's last tile, not before: a CTA that took its next unit when it began a long
                    // one held 24 tiles where others held 6
                    if (i + 1 == u.n_tiles) ask();
                    const int np = min(2, u.n_pages - 2 * i);
                    int page[2] = {0, 0};
                    for (int pg = 0; pg < np; ++pg) {
                        const int n = page_at(u, 2 * i + pg);
                        page[pg] = page_table != nullptr
                            ? TQ_CHECKED(page_table[(size_t)u.seq * S.table_stride + TQ_CHECKED(n, S.table_stride, TQ_IDX_TABLE_COLUMN)], S.n_pages, TQ_IDX_PAGE)
                            : page_base[u.seq] + n;
                    }
                    // a tile in shared memory: [column block of 64 elements][128 keys][128 bytes]; a page is 64 keys of it
                    const int ks = ti % C::KST;
                    if (!wait(k_empty(ks), ((uint32_t)(ti / C::KST) & 1u) ^ 1u)) { ok = false; break; }
                    if (elected) {
                        mbar_expect_tx(k_full(ks), (uint32_t)(np * C::K_PAGE));
                        for (int pg = 0; pg < np; ++pg)
#pragma unroll
                            for (int c = 0; c < C::KB; ++c) {
                            const uint32_t dst = k_smem(ks) + c * (BN * 128) + pg * (PAGE * 128);
                            if (c < S.k_blocks) tma_load_2d(dst, &map_k, u.g * S.kc + c * 64, page[pg] * S.kp + u.g * S.kg, k_full(ks));
                            else tma_load_2d(dst, &map_r, S.r_col + (c - S.k_blocks) * 64, page[pg] * S.kp, k_full(ks));
                        }
                    }
                    if (i == 0 && !load_q(1)) { ok = false; ++ti; break; }
                    const int vs = ti % C::VST;
                    if (!wait(v_empty(vs), ((uint32_t)(ti / C::VST) & 1u) ^ 1u)) { ok = false; ++ti; break; }
                    if (elected) {
                        mbar_expect_tx(v_full(vs), (uint32_t)(np * C::V_PAGE));
                        for (int pg = 0; pg < np; ++pg)
#pragma unroll
                            for (int c = 0; c < C::VB; ++c)
                            tma_load_2d(v_smem(vs) + c * (BN * 128) + pg * (PAGE * 128), &map_v, S.v_col + u.g * S.vc + c * 64,
                            page[pg] * S.kp + u.g * S.kg + S.v_plane, v_full(vs));
                    }
                    vi = ti + 1;
                    if (i + 1 == u.n_tiles) {
                        following = settle(answer());
                        if (ok) hand_on(k + 1, following);
                        if (!ok) { ++ti; break; }
                    }
                }
                unit = following;
            }
            if (s_abort) {      // let the answer and the copies this thread started land before the CTA goes away (bounded)
                if (pending) for (uint32_t j = 0; j < WAIT_LIMIT && !mbar_try_wait(answered, (uint32_t)asked & 1u); ++j) {}
                for (int s = 0; s < 2; ++s)
                    if (units[s]) for (uint32_t j = 0; j < WAIT_LIMIT && !mbar_try_wait(q_full(s), (uint32_t)(units[s] - 1) & 1u); ++j) {}
                for (int i = ti > C::KST ? ti - C::KST : 0; i < ti; ++i)
                    for (uint32_t j = 0; j < WAIT_LIMIT && !mbar_try_wait(k_full(i % C::KST), (uint32_t)(i / C::KST) & 1u); ++j) {}
                for (int i = vi > C::VST ? vi - C::VST : 0; i < vi; ++i)
                    for (uint32_t j = 0; j < WAIT_LIMIT && !mbar_try_wait(v_full(i % C::VST), (uint32_t)(i / C::VST) & 1u); ++j) {}
            }
        } else if (warp == 9) {
            // ------------------------------ MMA issuer ------------------------------
            // Tile by tile, slot by slot: the slot's P V product of this tile as soon as its P is there, then its scores of
            // the next tile (which may be the next unit's first): products are carried out in the order they are issued,
            // so the scores overwrite a P that has been read.
            const uint32_t elected = elect_one(), id_o = idesc(DV, 1);
            const uint32_t tm = __shfl_sync(0xffffffffu, s_tmem_base, 0);
            int ti = 0, taken = 0, tiles[2] = {0, 0}, units[2] = {0, 0};
            auto wait = [&](uint32_t bar, uint32_t parity) { return (bool)__all_sync(0xffffffffu, mbar_wait(bar, parity, &s_abort)); };
            auto next_unit = [&](Unit& u) {
                const int unit = take_unit(taken++);
                if (unit >= 0) u = unit_of(unit, S, cu_seqlens, seq_start);
                return unit >= 0;
            };
            const uint64_t q_desc = desc_k_major(q_smem(0)), k_desc = desc_k_major(k_smem(0)), v_desc = desc_mn_major(v_smem(0), BN * 128);
            // the scores of slot s for tile i of unit u, which is tile number t of the CTA; first, last: whether the other slot reads
            // the keys before or after it
            auto issue_qk = [&](const Unit& u, int i, int t, int s, bool first, bool last) -> bool {
                const int st = t % C::KST, np = min(2, u.n_pages - 2 * i);
                if (i == 0 && !wait(q_full(s), (uint32_t)units[s] & 1u)) return false;
                if (first && !wait(k_full(st), (uint32_t)(t / C::KST) & 1u)) return false;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t id_s = idesc(PAGE * np, 0);
                const uint64_t qd = q_desc + (uint64_t)(s * (C::Q_BYTES / 16)), kd = k_desc + (uint64_t)(st * (C::K_BYTES / 16));
#pragma unroll
                for (int k = 0; k < DK / 16; ++k)           // descriptors count in 16 bytes
                    umma(tm + (uint32_t)(s * BN), qd + (k / 4) * (BM * 8) + (k % 4) * 2, kd + (k / 4) * (BN * 8) + (k % 4) * 2, id_s, k > 0 ? 1u : 0u, elected);
                umma_commit(s_ready(s), elected);
                if (last) umma_commit(k_empty(st), elected);
                if (i == u.n[s] - 1) umma_commit(q_free(s), elected);           // the unit's last read of the slot's Q
                return true;
            };
            Unit u, v;
            bool more = next_unit(u), ok = true;
            if (more) {
                for (int s = 0; s < 2 && ok; ++s)
                    if (u.n[s]) ok = issue_qk(u, 0, 0, s, s == 0 || u.n[0] == 0, s == 1 || u.n[1] == 0);
            }
            while (more && ok) {
                bool follows = false;
                for (int i = 0; i < u.n_tiles && ok; ++i, ++ti) {
                    const bool crosses = i + 1 == u.n_tiles;             // the next tile is the next unit's first
                    if (crosses) follows = next_unit(v);
                    const int np = min(2, u.n_pages - 2 * i), st = ti % C::VST;
                    const int n0 = crosses ? (follows ? v.n[0] : 0) : u.n[0], n1 = crosses ? (follows ? v.n[1] : 0) : u.n[1];
                    const int j = crosses ? 0 : i + 1;                   // the next tile within its unit
                    for (int s = 0; s < 2 && ok; ++s) {
                        if (i < u.n[s]) {
                            ok = wait(p_ready(s), (uint32_t)tiles[s] & 1u);
                            if (ok && (s == 0 || i >= u.n[0])) ok = wait(v_full(st), (uint32_t)(ti / C::VST) & 1u);
                            if (ok && i == 0 && units[s] > 0) ok = wait(o_free(s), (uint32_t)(units[s] - 1) & 1u);
                            if (!ok) break;
                            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                            const uint64_t vd = v_desc + (uint64_t)(st * (C::V_BYTES / 16));
                            const uint32_t o = tm + (uint32_t)(2 * BN + s * DV), p = tm + (uint32_t)(s * BN);
#pragma unroll
                            for (int k = 0; k < BN / 16; ++k)            // O += P V, 16 keys at a time (a unit's first tile starts the sum)
                                if (k < PAGE / 16 || np > 1)             // a missing second page is not read
                                umma_ts(o, p + (uint32_t)(k * 8), vd + k * 128, id_o, (i > 0 || k > 0) ? 1u : 0u, elected);
                            if (s == 1 || i >= u.n[1]) umma_commit(v_empty(st), elected);
                            ++tiles[s];
                            if (i == u.n[s] - 1) { umma_commit(o_done(s), elected); ++units[s]; }
                        }
                        if (j < (s ? n1 : n0)) ok = issue_qk(crosses ? v : u, j, ti + 1, s, s == 0 || j >= n0, s == 1 || j >= n1);
                    }
                }
                more = follows;
                u = v;
            }
        }
    } else {
        // ------------------------------ softmax: a thread per query row ------------------------------
        asm volatile("setmaxnreg.inc.sync.aligned.u32 216;");
        constexpr int CW = ROWS ? 1 : 2;            // 32-key pieces a thread takes at a time
        constexpr float SLACK = ROWS ? 0.f : 8.f;   // powers of two by which a row's maximum may outgrow the one its exponentials are taken against
        const int slot = warp >> 2, quarter = warp & 3, r = quarter * 32 + lane;
        const uint32_t lane_addr = (uint32_t)(quarter * 32) << 16;
        const uint32_t s_addr = tmem_s(slot) + lane_addr, acc = tmem_o(slot) + lane_addr;
        // plain scores become exponents of two in the multiply-add that takes the maximum off; shaped ones keep their unit until it
        // is off, so that the largest finite values among them stay finite
        const float factor = ROWS ? 1.0f : S.scale * LOG2E, to_log2 = ROWS ? LOG2E : 1.0f;
        const bool capped = ROWS && S.softcap > 0.f;
        const CapSeries series = cap_series(S.scale, capped ? S.softcap : 1.f);
        int tiles = 0, units = 0, taken = 0;
        bool ok = true;
        for (int unit = take_unit(taken++); ok && unit >= 0; unit = ok ? take_unit(taken++) : -1) {
            const Unit u = unit_of(unit, S, cu_seqlens, seq_start);
            const int n = u.n[slot];
            if (n == 0) continue;
            const int h = u.h[slot], p_first = u.p_first[slot], qpos = p_first + r, p_last = p_first + BM - 1;
            const int start = S.cell > 0 ? qpos - qpos % S.cell : (S.window > 0 ? max(0, qpos + 1 - S.window) : 0);
            const int keep = S.cell > 0 || S.window == 0 ? 0 : S.keep_first;   // positions below it are seen besides those from `start` on
            // a page from here on is seen whole by every row that lies behind it
            const int open_from = S.cell > 0 ? p_last - p_last % S.cell : (S.window > 0 ? p_last + 1 - S.window : 0);
            const float* bias = ROWS && bias_t != nullptr ? bias_t + (size_t)h * (S.far + 1) : nullptr;
            float nb[6];                               // the next tile's bias values on their way to shared memory
            auto fetch_bias = [&](int i) {
#pragma unroll
                for (int j = 0; j < 6; ++j) {
                    const int d = p_first + quarter * 32 - page_at(u, 2 * i + j / 3) * PAGE - (PAGE - 1) + (j % 3) * 32 + lane;
                    nb[j] = __ldg(bias + min(max(d, 0), S.far));
                }
            };
            if (ROWS && bias != nullptr) fetch_bias(0);
            // m: what the row's exponents are counted from, its maximum or up to 2^SLACK below it; l: the sum of its exponentials
            const float floor_m = sink != nullptr ? sink[h] * (ROWS ? 1.0f : LOG2E) : -INFINITY;
            float m = -INFINITY, l = 0.f;
            for (int i = 0; i < n; ++i, ++tiles) {
                const int np = min(2, u.n_pages - 2 * i);
                if (ROWS && bias != nullptr) {
                    __syncwarp();                      // the previous tile's values have been read
#pragma unroll
                    for (int j = 0; j < 6; ++j) s_bias[ROWS ? warp : 0][j / 3][(j % 3) * 32 + lane] = nb[j];
                    __syncwarp();
                    if (i + 1 < n) fetch_bias(i + 1);
                }
                ok = __all_sync(0xffffffffu, mbar_wait(s_ready(slot), (uint32_t)tiles & 1u, &s_abort));   // warp-uniform
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                // half a page (plain scores: a page) at a time, twice: for the tile's maximum, which shapes and masks the scores and
                // leaves shaped ones in place of the products, then for the weights, written in bf16 over scores already
                // read.  The maximum comes first so that a row's largest weight can be exactly one: with it known only so far, and
                // corrected by powers of two, the error of rows against 64 bits was up to 1.3 times as large (here it is that of
                // the mma.sync kernel or less).  It costs 2 to 5 us of the times above (plain 49.6, cap 50 73.7, bias 42.1).  The loops are kept small: instructions come in at some 250 cycles per 128 bytes the first time and
                // fall out of the caches that ten warps share (the tile unrolled in two passes: 1.6 times the kernel's time).
                float2 sum[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
                float top = -INFINITY;
#pragma unroll 1
                for (int x = -2 * np; x < 2 * np; x += CW) {
                    const int q = x < 0 ? x + 2 * np : x;
                    if (x == 0) {
                        if (ROWS) asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                        const float mx = fmaxf(top * factor, floor_m);
                        float corr = 1.0f;
                        if (m == -INFINITY) {
                            m = mx;                        // l and O are still zero: nothing to rescale
                        } else if ((mx - m) * to_log2 > SLACK) {
                            corr = ex2((m - mx) * to_log2);
                            l *= corr;
                            m = mx;
                        }
                        if (i > 0 && __any_sync(0xffffffffu, corr != 1.0f)) {  // the products so far are done (s_ready)
#pragma unroll 1
                            for (int c0 = 0; c0 < DV; c0 += 16) {
                                uint32_t ov[16];
                                tmem_ld16(acc + c0, ov);
                                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                                for (int j = 0; j < 16; ++j) ov[j] = __float_as_uint(__uint_as_float(ov[j]) * corr);
                                tmem_st16(acc + c0, ov);
                            }
                        }
                    }
                    uint32_t sv[CW][32];
#pragma unroll
                    for (int w = 0; w < CW; ++w) tmem_ld32(s_addr + (q + w) * 32, sv[w]);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                    const int kq = page_at(u, 2 * i + (q >> 1)) * PAGE + (q & 1) * 32;   // position of the first of these keys
                    if (ROWS && x < 0) {
                        if (capped) cap_scores(sv[0], series);
                        if (bias != nullptr) {
                            const float2 f = capped ? make_float2(1.f, 1.f) : make_float2(S.scale, S.scale);
                            const float* sb = &s_bias[ROWS ? warp : 0][q >> 1][lane + PAGE - 1 - (q & 1) * 32];
#pragma unroll
                            for (int c = 0; c < 32; c += 2) {
                                const float2 t = fma2(make_float2(__uint_as_float(sv[0][c]), __uint_as_float(sv[0][c + 1])), f, make_float2(sb[-c], sb[-c - 1]));
                                sv[0][c] = __float_as_uint(t.x);
                                sv[0][c + 1] = __float_as_uint(t.y);
                            }
                        } else if (!capped) {
#pragma unroll
                            for (int c = 0; c < 32; ++c) sv[0][c] = __float_as_uint(__uint_as_float(sv[0][c]) * S.scale);
                        }
                    }
                    if ((!ROWS || x < 0) && (kq + 32 * CW - 1 > p_first || kq < open_from)) {        // some row does not see some of these keys
#pragma unroll
                        for (int w = 0; w < CW; ++w) {
                            // bit c: the row sees key kq + 32 w + c, i.e. c <= last and (c >= lo or c < kp)
                            const int last = qpos - kq - 32 * w, lo = start - kq - 32 * w, kp = keep - kq - 32 * w;
                            const uint32_t behind = last < 0 ? 0u : 0xffffffffu >> (31 - min(last, 31));
                            const uint32_t inside = lo >= 32 ? 0u : 0xffffffffu << max(lo, 0);
                            const uint32_t kept = kp <= 0 ? 0u : 0xffffffffu >> (32 - min(kp, 32));
                            const uint32_t seen = behind & (inside | kept);
#pragma unroll
                            for (int c = 0; c < 32; ++c)
                                if (!(seen & (1u << c))) sv[w][c] = 0xff800000u;
                        }
                    }
                    if (x < 0) {
                        top = max_of(sv[0], top);
                        if (CW > 1) top = max_of(sv[CW - 1], top);
                        if (ROWS) tmem_st32(s_addr + q * 32, sv[0]);
                        continue;
                    }
                    const float mref = m == -INFINITY ? 0.f : m;             // nothing visible yet: exponents of -inf
                    const float2 ff = make_float2(ROWS ? to_log2 : factor, ROWS ? to_log2 : factor), neg = make_float2(-mref, -mref);
#pragma unroll
                    for (int w = 0; w < CW; ++w) {
                        uint32_t pk[16];
#pragma unroll
                        for (int e = 0; e < 16; ++e) {
                            float2 x = make_float2(__uint_as_float(sv[w][2 * e]), __uint_as_float(sv[w][2 * e + 1]));
                            x = ROWS ? mul2(add2(x, neg), ff) : fma2(x, ff, neg);
                            x = make_float2(ex2(x.x), ex2(x.y));
                            const __nv_bfloat162 two = __floats2bfloat162_rn(x.x, x.y);
                            pk[e] = *reinterpret_cast<const uint32_t*>(&two);
                            // the sum of what the second product multiplies: part of the weights' rounding cancels
                            if (ROWS) x = make_float2(__uint_as_float(pk[e] << 16), __uint_as_float(pk[e] & 0xffff0000u));
                            sum[e % 2] = add2(sum[e % 2], x);
                        }
                        tmem_st16(s_addr + (q + w) * 16, pk);
                    }
                }
                l += (sum[0].x + sum[0].y) + (sum[1].x + sum[1].y);
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(p_ready(slot));
            }
            if (!ok) break;
            // the unit's products done: O / the row's sum
            ok = __all_sync(0xffffffffu, mbar_wait(o_done(slot), (uint32_t)units & 1u, &s_abort));
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (sink != nullptr) l += ex2((floor_m - m) * to_log2);
            const float inv = 1.0f / l;
            __nv_bfloat16* dst = out + ((size_t)(u.t0[slot] + r) * S.nh + h) * DV;
#pragma unroll 1
            for (int c0 = 0; c0 < DV; c0 += 32) {
                uint32_t ov[32];
                tmem_ld32(acc + c0, ov);               // every lane takes part: the load is warp-wide
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                if (r < u.rows[slot]) {
#pragma unroll
                    for (int d = 0; d < 32; d += 8) {
                        uint32_t packed[4];
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            const __nv_bfloat162 two = __floats2bfloat162_rn(__uint_as_float(ov[d + 2 * e]) * inv, __uint_as_float(ov[d + 2 * e + 1]) * inv);
                            packed[e] = *reinterpret_cast<const uint32_t*>(&two);
                        }
                        *reinterpret_cast<uint4*>(dst + c0 + d) = make_uint4(packed[0], packed[1], packed[2], packed[3]);
                    }
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(o_free(slot));
            ++units;
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 9) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(s_tmem_base), "r"((uint32_t)C::TMEM_COLS) : "memory");
    }
    if (threadIdx.x == 0 && s_abort) atomicExch(status, 1);
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = (EncodeTiledFn)p;
    }
    return fn;
}

// bf16 matrix [rows][cols] row-major; box [box_rows][64 columns], 128-byte swizzle
int make_map(CUtensorMap* map, const void* ptr, uint64_t rows, uint64_t cols, uint32_t box_rows) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) TQ_FAIL(-3, "attention_prefill: cuTensorMapEncodeTiled is not available from the driver");
    cuuint64_t dims[2] = {cols, rows};
    cuuint64_t strides[1] = {cols * 2};
    cuuint32_t box[2] = {64, box_rows};
    cuuint32_t elem[2] = {1, 1};
    CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), dims, strides, box, elem,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) TQ_FAIL(-3, "attention_prefill: cuTensorMapEncodeTiled failed with code %d", (int)r);
    return 0;
}

struct Maps { CUtensorMap q, k, r, v; };
struct Args {
    const int *cu, *starts, *table, *page_base;
    const float *bias_t, *sink;
    void* out;
    int* status;
};

template <int DK, int DV, bool ROWS>
int launch(const Maps& m, const Shape& S, const Args& a, cudaStream_t stream) {
    using C = Cfg<DK, DV>;
    auto kern = attention_prefill_kernel<DK, DV, ROWS>;
    static std::atomic<unsigned long long> asked{0};
    const cudaError_t e = tq_reserve_smem(kern, C::SMEM_BYTES, asked);
    if (e != cudaSuccess) TQ_FAIL(-1, "attention_prefill: cannot reserve %d bytes of shared memory: %s", C::SMEM_BYTES, cudaGetErrorString(e));
    // a block per unit; those that run take over the ones that have not started
    const int hs = S.pairing == PAIR_HEADS ? S.nh / 2 : S.nh, qs = S.pairing == PAIR_HEADS ? S.n_qt : (S.n_qt + 1) / 2;
    const int grid = qs * S.n_seqs * hs;
    tq_launch(grid, THREADS, C::SMEM_BYTES, stream)(kern, m.q, m.k, m.r, m.v, S, a.cu, a.starts, a.table, a.page_base, a.bias_t, a.sink,
                                                   (__nv_bfloat16*)a.out, a.status);
    TQ_CHECK_LAUNCH("attention_prefill");
    return 0;
}

int check_common(const Shape& S, int T_, int max_q_len, const void* q, const void* k, const void* v, const void* out, const int* status) {
    TQ_REQUIRE(S.nkv >= 1 && S.nh % S.nkv == 0, "attention_prefill: %d heads are not a multiple of %d key/value heads", S.nh, S.nkv);
    TQ_REQUIRE((long long)S.n_qt * S.n_seqs * S.nh < (1ll << 30), "attention_prefill: too many units of work");
    TQ_REQUIRE(S.window >= 0 && S.keep_first >= 0 && S.cell >= 0 && S.far >= 0 && max_q_len >= 1 && T_ >= 1,
               "attention_prefill: bad window %d, kept positions %d, cell %d or longest run %d", S.window, S.keep_first, S.cell, max_q_len);
    TQ_REQUIRE(((uintptr_t)q % 16) == 0 && ((uintptr_t)k % 16) == 0 && ((uintptr_t)v % 16) == 0 && ((uintptr_t)out % 16) == 0,
               "attention_prefill: q, cache and out must be 16-byte aligned");
    TQ_REQUIRE(status != nullptr, "attention_prefill: a status word is required");
    return 0;
}

}  // namespace

// q [T, nh, dk] bf16; cache bf16 (keys and values of this step already written): planes 2: [n_pages, 2, nkv, 64, dk] with
// dk == dv, planes 1: [n_pages, nkv, 64, dk + dv], a position's key followed by its value; out [T, nh*dv].
// cu_seqlens [n_seqs+1]: rows of each sequence in q; seq_start [n_seqs]: position of each sequence's first row.
// Position i sees j <= i with window == 0 or i - j < window or j < keep_first; with cell > 0 instead j <= i of its own
// cell.  Scores times scale, capped (softcap > 0), plus bias_t [nh][far + 1] (or null) at distance min(i - j, far); sink
// [nh] or null joins the denominator.  status: one int in device memory, set to 1 if a bounded wait ran out.
TQ_EXPORT int tq_attention_prefill(const void* q, const void* cache, int planes, const int* cu_seqlens, const int* seq_start,
                                   const int* page_table, int table_stride, int page_size, int n_pages, int window, int keep_first,
                                   int cell, float scale, float softcap, const float* bias_t, int far, const float* sink, void* out,
                                   int T_, int n_seqs, int max_q_len, int nh, int nkv, int dk, int dv, int* status, cudaStream_t stream) {
    if (T_ == 0 || n_seqs == 0) return 0;
    TQ_REQUIRE((dk == 64 || dk == 128) && (dv == 64 || dv == 128), "attention_prefill: key size %d or value size %d is not 64 or 128", dk, dv);
    TQ_REQUIRE(planes == 1 || (planes == 2 && dk == dv), "attention_prefill: %d planes of keys of %d and values of %d", planes, dk, dv);
    TQ_REQUIRE(page_size == PAGE, "attention_prefill: page size %d must be %d", page_size, PAGE);
    Shape S{};
    S.nh = nh; S.nkv = nkv; S.n_seqs = n_seqs; S.n_qt = (max_q_len + BM - 1) / BM;
    S.kp = planes * nkv * PAGE; S.kg = PAGE; S.v_plane = (planes - 1) * nkv * PAGE; S.v_col = planes == 1 ? dk : 0; S.k_blocks = dk / 64;
    S.table_stride = table_stride; S.n_pages = n_pages; S.window = window; S.keep_first = keep_first; S.cell = cell; S.far = far;
    S.scale = scale; S.softcap = softcap;
    int rc = check_common(S, T_, max_q_len, q, cache, cache, out, status);
    if (rc) return rc;
    TQ_REQUIRE((long long)n_pages * S.kp < (1ll << 31), "attention_prefill: a cache of %d pages is too large for one tensor map", n_pages);
    S.pairing = nh / nkv % 2 == 0 ? PAIR_HEADS : PAIR_ROWS;
    Maps m;
    rc = make_map(&m.q, q, (uint64_t)T_, (uint64_t)nh * dk, BM);
    if (rc) return rc;
    rc = make_map(&m.k, cache, (uint64_t)n_pages * S.kp, (uint64_t)(planes == 1 ? dk + dv : dk), PAGE);
    if (rc) return rc;
    m.r = m.v = m.k;
    const Args a{cu_seqlens, seq_start, page_table, nullptr, bias_t, sink, out, status};
    const bool shaped = planes == 1 || softcap > 0.f || bias_t != nullptr || !(scale > 0.f);     // (the other form compares unscaled scores)
#define AP_CASE(DK_, DV_) if (dk == DK_ && dv == DV_) return shaped ? launch<DK_, DV_, true>(m, S, a, stream) : launch<DK_, DV_, false>(m, S, a, stream);
    AP_CASE(64, 64) AP_CASE(64, 128) AP_CASE(128, 64) AP_CASE(128, 128)
#undef AP_CASE
    return -2;
}

// The same over keys and values that lie densely: kv [rows, nh * (dim + dv)] bf16, a position's keys of all heads, then its
// values; rot [rows, rot_stride] whose columns from r_col on are the `rot` (0 or 64) last elements of every head's key.  Position
// p of sequence s is row 64 * page_base[s] + p; rows up to the end of a position's 64 exist.  q [T, nh, dim + rot].
TQ_EXPORT int tq_attention_prefill_dense(const void* q, const void* kv, const void* rot_rows, int rows, int rot_stride, int r_col,
                                         const int* cu_seqlens, const int* seq_start, const int* page_base, int window, float scale,
                                         const float* sink, void* out, int T_, int n_seqs, int max_q_len, int nh, int dim, int rot,
                                         int dv, int* status, cudaStream_t stream) {
    if (T_ == 0 || n_seqs == 0) return 0;
    TQ_REQUIRE((rot == 0 || rot == 64) && (dim == 64 || dim == 128) && (dv == 64 || dv == 128) && (dim + rot < 192 || dv == 128),
               "attention_prefill_dense: keys of %d + %d elements and values of %d", dim, rot, dv);
    TQ_REQUIRE(rot == 0 || (r_col % 8 == 0 && rot_stride % 8 == 0 && r_col + rot <= rot_stride && ((uintptr_t)rot_rows % 16) == 0),
               "attention_prefill_dense: the shared key columns %d of %d are not aligned", r_col, rot_stride);
    TQ_REQUIRE(scale > 0.f, "attention_prefill_dense: scale %g", scale);
    Shape S{};
    S.nh = nh; S.nkv = nh; S.n_seqs = n_seqs; S.n_qt = (max_q_len + BM - 1) / BM; S.pairing = PAIR_ROWS;
    S.kp = PAGE; S.kc = dim; S.vc = dv; S.v_col = nh * dim; S.k_blocks = dim / 64; S.r_col = r_col;
    S.window = window; S.scale = scale;
    int rc = check_common(S, T_, max_q_len, q, kv, kv, out, status);
    if (rc) return rc;
    const int dk = dim + rot;
    Maps m;
    rc = make_map(&m.q, q, (uint64_t)T_, (uint64_t)nh * dk, BM);
    if (rc) return rc;
    rc = make_map(&m.k, kv, (uint64_t)rows, (uint64_t)nh * (dim + dv), PAGE);
    if (rc) return rc;
    m.r = m.v = m.k;
    if (rot) rc = make_map(&m.r, rot_rows, (uint64_t)rows, (uint64_t)rot_stride, PAGE);
    if (rc) return rc;
    const Args a{cu_seqlens, seq_start, nullptr, page_base, nullptr, sink, out, status};
#define AP_CASE(DK_, DV_) if (dk == DK_ && dv == DV_) return launch<DK_, DV_, false>(m, S, a, stream);
    AP_CASE(64, 64) AP_CASE(64, 128) AP_CASE(128, 64) AP_CASE(128, 128) AP_CASE(192, 128)
#undef AP_CASE
    return -2;
}
