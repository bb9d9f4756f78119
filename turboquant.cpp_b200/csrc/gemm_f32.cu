// out [T, N] = x [T, K] w [N, K]^T in float32 on the 5th-generation tensor cores (tcgen05): every operand as three bfloat16 values
// (split3.cuh), six products of them, or three as long as the weights of a tile are bfloat16 values.
//
// The reference's dense products in float32 go to the platform's BLAS (src/engine/tq_ops.c:297-306).  The fp32 units give 74
// TFLOP/s, the tensor cores a sixth to a third of 1,600.  Two CTAs on two SMs share a tile of 256 weight rows and up to 256 tokens
// (cta_group::2): each brings and splits 128 weight rows and half of the tokens, half the bytes and half the splitting of a CTA by itself.
//   warp 17       brings blocks of both operands by TMA
//   warps 0..7    split them and store the parts as K-major tiles of 32 elements, 64-byte swizzle
//   warp 16       issues the products (the first CTA's for both)
//   warps 8..15   add the accumulator of the largest products, h h', to sums in their registers every two blocks and write the result
//   warps 18, 19  of the second CTA: tell the first that its parts are stored, every other block each.  What the splitting warps wrote is
//                 seen in the other CTA only behind a release at the cluster's scope, and that takes most of a block's time
// The tensor cores' own sums cut bits off at every addition, so a chain of products over all of K is off by more than a
// float32 sum is (K 2,048: 2.2e-6 of the result; the library's sum 8.1e-7); sums of 64 elements added up in rounded float32 are
// off by less (1.3e-7).  The smaller products, 2^-8 of the result and less, stay in one accumulator
// for all of K, and the other accumulator is read in the time they take: it costs nothing.
// 700 tokens, K 2,048: 80 us for 6,144 rows (65 with bfloat16 weights; the library's fp32 product 309), 47 for 2,048 (145).  What bounds it is
// the splitting, some 1,200 cycles a block of 32 elements for 720 (three products) or 1,440 (six) of the tensor cores at 240 tokens.
// What a block cost otherwise: 450 cycles more with splitting warps that release at the cluster's scope themselves, 240 with one warp
// that tells of all blocks, 120 to 230 with three stages of parts where more fit; two groups of splitting warps taking every other
// block: nothing gained.
// Every result that is not finite is computed again as a plain sum, so infinities and NaN come out as fmaf leaves them.
// Waits on mbarriers are bounded: one that runs out sets a flag, every role leaves, and *status is set.
#include <cuda.h>
#include "split3.cuh"

TQ_DEFINE_LAST_ERROR

namespace {

constexpr int BM = 128;                        // weight rows of a CTA (half a tile of the pair)
constexpr int BK = 32;                         // elements of K per block: 64 bytes of bfloat16, one swizzled row
constexpr int UMMA_K = 16;
constexpr int MAX_TOKENS = 256;                // of a tile; the accumulators of h h' and of the rest fill the tensor memory
constexpr int CONV_WARPS = 8, DRAIN_WARPS = 8;
constexpr int THREADS = 32 * (CONV_WARPS + DRAIN_WARPS + 4);       // whole warpgroups: registers are given and taken by them
constexpr int CONV_REGS = 56, DRAIN_REGS = 168, MMA_REGS = 24, LAUNCH_REGS = 96;   // LAUNCH_REGS: what 640 threads are launched with
static_assert(32 * (CONV_WARPS * CONV_REGS + DRAIN_WARPS * DRAIN_REGS + 4 * MMA_REGS) <= THREADS * LAUNCH_REGS, "more registers than the block is launched with");
constexpr int ROWS_EACH = 8;                   // rows of a block that a thread splits four elements of
constexpr int PART = BM * BK * 2;              // one part of one operand of a block
constexpr int RAWS = 2;
// Shared memory by the tokens of a tile: a block's parts (weights h, m, l, tokens h, m, l), blocks as they come, and as many stages
// of parts as fit beside those
constexpr int SMEM_BYTES = 226 * 1024, MAX_STAGES = 6;
__host__ __device__ constexpr int stage_bytes(int n) { return 3 * PART + 3 * (n / 2) * BK * 2; }
__host__ __device__ constexpr int raw_bytes(int n) { return BM * BK * 4 + (n / 2) * BK * 4; }
__host__ __device__ constexpr int stages_of(int n) {
    const int fit = (SMEM_BYTES - 1024 /* alignment */ - RAWS * raw_bytes(n)) / stage_bytes(n);
    return fit < MAX_STAGES ? fit : MAX_STAGES;
}
static_assert(stages_of(MAX_TOKENS) >= 3, "shared memory");
constexpr int GROUP = 2;                       // blocks whose h h' the tensor cores add up: 64 elements
constexpr uint32_t WAIT_LIMIT = 1u << 20;      // polls of an mbarrier before a wait gives up ...
constexpr uint64_t WAIT_NS = 2000000000ull;    // ... or two seconds

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
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
__device__ __forceinline__ bool mbar_try_wait_cluster(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}
// CLUSTER: what the other CTA wrote before it arrived is seen
template <bool CLUSTER = false>
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
    uint64_t t0 = 0;
    for (uint32_t i = 0; i < WAIT_LIMIT; ++i) {
        if (CLUSTER ? mbar_try_wait_cluster(bar, parity) : mbar_try_wait(bar, parity)) return true;
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
__device__ __forceinline__ uint32_t map_to_cta(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_bar) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_bar) : "memory");
}
// ... without any data: for a barrier that only says that tensor memory has been read
__device__ __forceinline__ void mbar_arrive_order(uint32_t cluster_bar) {
    asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_bar) : "memory");
}
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory"); }
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int col, int row, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
        ::"r"(dst), "l"((uint64_t)map), "r"(bar), "r"(col), "r"(row) : "memory");
}

// K-major tile of 64-byte rows, 64-byte swizzle (layout type 4), eight rows 512 bytes apart
__device__ __forceinline__ uint64_t umma_desc(uint32_t addr) {
    return (uint64_t)((addr & 0x3FFFFu) >> 4) | (1ull << 16) | ((uint64_t)(512 >> 4) << 32) | (1ull << 46) | (4ull << 61);
}
// kind::f16, D fp32, A and B bf16, both K-major, M = 256 over the pair
__device__ __forceinline__ uint32_t umma_idesc(int n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(2 * BM >> 4) << 24);
}
// The products are issued by a convergent warp from values that are the same in all lanes, the instruction itself by the elected one:
// from a single thread's branch each of them costs some hundred cycles.
__device__ __forceinline__ uint32_t elect_one() {
    uint32_t e;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(e));
    return e;
}
__device__ __forceinline__ void umma_pair(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate, uint32_t elected) {
    asm volatile(
        "{\n\t.reg .pred p, e;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "setp.ne.b32 e, %5, 0;\n\t"
        "@e tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate), "r"(elected) : "memory");
}
// arrives on the barrier at this address in both CTAs once the products issued so far are done
__device__ __forceinline__ void umma_commit_pair(uint32_t bar, uint32_t elected) {
    asm volatile(
        "{\n\t.reg .pred e;\n\t"
        "setp.ne.b32 e, %2, 0;\n\t"
        "@e tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n\t}"
        ::"r"(bar), "h"((uint16_t)3), "r"(elected) : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&v)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
          "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// x rows ldx floats apart; n: tokens of a tile, a multiple of 16.  The maps' boxes: 32 floats of 128 weight rows, of n / 2 tokens.
__global__ void __launch_bounds__(THREADS, 1)
gemm_f32_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, const float* __restrict__ x, long long ldx, const float* __restrict__ w, float* __restrict__ out, int T, int N, int K, int n,
                int n_t, int* __restrict__ status) {
    tq_grid_wait();                    // everything below may read what the previous kernel wrote
    extern __shared__ uint8_t smem_raw[];
    __shared__ int s_abort;
    __shared__ uint32_t s_tmem_base;
    __shared__ uint32_t s_low;         // the weights so far were not all bfloat16 values (the first CTA's)
    __shared__ __align__(8) uint64_t s_bars[3 * MAX_STAGES + 3 + 2 * RAWS];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t rank = blockIdx.x & 1;
    const int tile = blockIdx.x >> 1;
    const int t0 = tile % n_t * n, n0 = tile / n_t * (2 * BM) + (int)rank * BM;     // token tiles side by side share the weights
    const int count = min(n, T - t0);
    const int blocks = (K + BK - 1) / BK;
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const int stages = stages_of(n), stage = stage_bytes(n), raw = raw_bytes(n), x_part = n / 2 * BK * 2;
    const uint32_t raw0 = base + stages * stage;
    auto full_bar = [&](int s) { return smem_u32(&s_bars[s]); };                    // parts stored (the first CTA's)
    auto done_bar = [&](int s) { return smem_u32(&s_bars[MAX_STAGES + s]); };       // ... and used
    const uint32_t sum_full = smem_u32(&s_bars[2 * MAX_STAGES]), sum_empty = sum_full + 8, all_done = sum_full + 16;
    auto raw_full = [&](int r) { return all_done + 8 + 8u * r; };                   // this CTA's: brought
    auto raw_done = [&](int r) { return all_done + 8 + 8u * (RAWS + r); };          // ... and split
    auto stored_bar = [&](int s) { return all_done + 8 + 8u * (2 * RAWS + s); };    // the second CTA's own: parts stored
    const int half = n / 2, x0 = t0 + (int)rank * half;                             // this CTA's tokens of the tile

    if (tid == 0) {
        s_abort = 0;
        s_low = 0;
        // the first CTA's warps and, for all of the second's, one that passes it on
        for (int s = 0; s < stages; ++s) { mbar_init(full_bar(s), CONV_WARPS + 1); mbar_init(done_bar(s), 1); mbar_init(stored_bar(s), CONV_WARPS); }
        mbar_init(sum_full, 1);
        mbar_init(sum_empty, 2 * DRAIN_WARPS);
        mbar_init(all_done, 1);
        for (int r = 0; r < RAWS; ++r) { mbar_init(raw_full(r), 1); mbar_init(raw_done(r), CONV_WARPS); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == CONV_WARPS + DRAIN_WARPS) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem_base)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    cluster_sync_all();                // barriers are ready in both CTAs before either signals the other
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    tq_grid_launch_dependents();       // only now: a dependent kernel that took tensor memory first could starve a CTA of this grid
    const uint32_t tmem = s_tmem_base;

    if (warp < CONV_WARPS) {
        // ---- both operands: split, stored ----
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(CONV_REGS));
        const int c = tid & 7, r0 = tid >> 3;
        bool told = false;
        // a row's 64 bytes hold four pieces of 16, their places shuffled by bits 1 and 2 of the row; the lanes' rows are 32 apart
        const uint32_t at = (uint32_t)r0 * 64 + (uint32_t)(((c >> 1) ^ ((r0 >> 1) & 3)) * 16 + (c & 1) * 8);
        int s = 0;
        uint32_t phase = 1;                                              // of the stage's last use
        for (int kb = 0; kb < blocks; ++kb) {
            const int rs = kb % RAWS;
            if (!mbar_wait(raw_full(rs), (uint32_t)(kb / RAWS) & 1u, &s_abort)) break;
            if (kb >= stages && !mbar_wait(done_bar(s), phase, &s_abort)) break;
            const uint32_t src = raw0 + rs * raw + (uint32_t)r0 * (BK * 4) + c * 16, dst = base + s * stage + at;
            uint32_t low = 0;
            float4 v[ROWS_EACH];
#pragma unroll
            for (int i = 0; i < ROWS_EACH; ++i)
                if (i < 4 || r0 + 32 * (i - 4) < half)
                    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v[i].x), "=f"(v[i].y), "=f"(v[i].z), "=f"(v[i].w)
                                 : "r"(src + i * (32 * BK * 4)) : "memory");
#pragma unroll
            for (int i = 0; i < ROWS_EACH; ++i)
                if (i < 4 || r0 + 32 * (i - 4) < half) {
                    const TqSplit4 p = tq_split4(v[i]);
                    const uint32_t d = dst + (i < 4 ? 0 : 3 * PART) + (i & 3) * (32 * 64), part = i < 4 ? PART : x_part;
                    asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(d), "r"(p.h.x), "r"(p.h.y) : "memory");
                    asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(d + part), "r"(p.m.x), "r"(p.m.y) : "memory");
                    asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(d + 2 * part), "r"(p.l.x), "r"(p.l.y) : "memory");
                    if (i < 4) low |= p.m.x | p.m.y | p.l.x | p.l.y;
                }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the tensor cores read through the other proxy
            const bool tell = !told && __any_sync(0xffffffffu, low != 0);
            __syncwarp();
            if (lane == 0) {
                if (tell)                                                 // once a warp
                    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(map_to_cta(smem_u32(&s_low), 0)), "r"(1u) : "memory");
                mbar_arrive(rank == 0 ? full_bar(s) : stored_bar(s));
                mbar_arrive(raw_done(rs));
            }
            told |= tell;
            if (++s == stages) { s = 0; phase ^= 1u; }
        }
    } else if (warp < CONV_WARPS + DRAIN_WARPS) {
        // ---- sums: lane = weight row, every other 16 tokens ----
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(DRAIN_REGS));
        const int quarter = warp & 3, odd = (warp - CONV_WARPS) >> 2;
        const uint32_t lane_addr = tmem + ((uint32_t)(quarter * 32) << 16);
        float acc[MAX_TOKENS / 32][16];
#pragma unroll
        for (int i = 0; i < MAX_TOKENS / 32; ++i)
#pragma unroll
            for (int j = 0; j < 16; ++j) acc[i][j] = 0.f;
        // adds columns of the accumulator at `col` to the sums; the next 16 are on their way meanwhile
        auto add = [&](uint32_t col) {
            uint32_t buf[2][16];
            if (odd * 16 < n) tmem_ld16(lane_addr + col + odd * 16, buf[0]);
#pragma unroll
            for (int i = 0; i < MAX_TOKENS / 32; ++i) {
                const int c0 = 32 * i + 16 * odd;
                if (c0 >= n) break;
                tmem_ld_wait();
                if (i + 1 < MAX_TOKENS / 32 && c0 + 32 < n) tmem_ld16(lane_addr + col + c0 + 32, buf[(i + 1) & 1]);
#pragma unroll
                for (int j = 0; j < 16; ++j) acc[i][j] += __uint_as_float(buf[i & 1][j]);
            }
        };
        const int groups = (blocks + GROUP - 1) / GROUP;
        bool ok = true;
        for (int g = 0; g < groups && ok; ++g) {
            ok = __all_sync(0xffffffffu, mbar_wait(sum_full, (uint32_t)g & 1u, &s_abort));
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            add(0);
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive_order(map_to_cta(sum_empty, 0));
        }
        if (ok) ok = __all_sync(0xffffffffu, mbar_wait(all_done, 0u, &s_abort));
        if (ok) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            add(MAX_TOKENS);
            const int row = n0 + quarter * 32 + lane;
            float* to = out + (size_t)t0 * N + row;
            float* p = to + (size_t)(16 * odd) * N;
            bool odd_ones = false;
            if (row < N) {
#pragma unroll
                for (int i = 0; i < MAX_TOKENS / 32; ++i) {
                    if (32 * i + 16 * odd >= count) break;
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        if (32 * i + 16 * odd + j < count) *p = acc[i][j];
                        odd_ones |= !isfinite(acc[i][j]);
                        p += N;
                    }
                    p += (size_t)16 * N;
                }
                // (kept out of the loop above: 128 copies of this one took longer to fetch than the whole product took)
                if (odd_ones)
                    for (int t = 0; t < count; ++t) {
                        if ((t >> 4 & 1) != odd || isfinite(to[(size_t)t * N])) continue;
                        float v = 0.f;
                        for (int k = 0; k < K; ++k) v = fmaf(x[(size_t)(t0 + t) * ldx + k], w[(size_t)row * K + k], v);
                        to[(size_t)t * N] = v;
                    }
            }
        }
    } else {
        // ---- products ----
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(MMA_REGS));
        if (warp == CONV_WARPS + DRAIN_WARPS && rank == 0) {
            const uint32_t elected = elect_one(), idesc = umma_idesc(n), sums = __shfl_sync(0xffffffffu, tmem, 0), rest = sums + MAX_TOKENS;
            const uint64_t desc0 = umma_desc(base);                          // descriptors count in 16 bytes
            auto wait = [&](uint32_t bar, uint32_t parity) { return (bool)__all_sync(0xffffffffu, mbar_wait<true>(bar, parity, &s_abort)); };
            int s = 0;
            uint32_t phase = 0;
            for (int kb = 0; kb < blocks; ++kb) {
                if (!wait(full_bar(s), phase)) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const bool low = __shfl_sync(0xffffffffu, *(volatile uint32_t*)&s_low, 0) != 0;
                const uint64_t wd = desc0 + (uint64_t)(s * (stage / 16)), xd = wd + 3 * PART / 16;
                auto times = [&](uint32_t d, int pw, int px, int k, uint32_t accumulate) {
                    umma_pair(d, wd + (pw * (PART / 16) + k * 2), xd + (px * (x_part / 16) + k * 2), idesc, accumulate, elected);
                };
#pragma unroll
                for (int k = 0; k < BK / UMMA_K; ++k) times(rest, 0, 2, k, kb > 0 || k > 0 ? 1u : 0u);
                if (low) {
#pragma unroll
                    for (int k = 0; k < BK / UMMA_K; ++k) {
                        times(rest, 2, 0, k, 1u);
                        times(rest, 1, 1, k, 1u);
                        times(rest, 1, 0, k, 1u);
                    }
                }
#pragma unroll
                for (int k = 0; k < BK / UMMA_K; ++k) times(rest, 0, 1, k, 1u);
                const int g = kb / GROUP;
                if (kb % GROUP == 0 && g > 0) {                              // the sums so far have been read
                    if (!wait(sum_empty, (uint32_t)(g - 1) & 1u)) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                }
#pragma unroll
                for (int k = 0; k < BK / UMMA_K; ++k) times(sums, 0, 0, k, kb % GROUP != 0 || k > 0 ? 1u : 0u);
                umma_commit_pair(done_bar(s), elected);
                if (kb % GROUP == GROUP - 1 || kb == blocks - 1) umma_commit_pair(sum_full, elected);
                if (kb == blocks - 1) umma_commit_pair(all_done, elected);
                if (++s == stages) { s = 0; phase ^= 1u; }
            }
        } else if (warp == CONV_WARPS + DRAIN_WARPS + 1 && lane == 0) {
            // ---- both operands' blocks, zeros behind their ends ----
            int issued = 0;
            for (; issued < blocks; ++issued) {
                const int r = issued % RAWS;
                if (issued >= RAWS && !mbar_wait(raw_done(r), (uint32_t)(issued / RAWS - 1) & 1u, &s_abort)) break;
                mbar_expect_tx(raw_full(r), (uint32_t)((BM + half) * BK * 4));
                tma_load_2d(raw0 + r * raw, &map_w, issued * BK, n0, raw_full(r));
                tma_load_2d(raw0 + r * raw + BM * BK * 4, &map_x, issued * BK, x0, raw_full(r));
            }
            if (s_abort)                                   // no copy lands after the CTA is gone
                for (int j = max(issued - RAWS, 0); j < issued; ++j)
                    for (uint32_t i = 0; i < WAIT_LIMIT && !mbar_try_wait(raw_full(j % RAWS), (uint32_t)(j / RAWS) & 1u); ++i) {}
        } else if (warp >= CONV_WARPS + DRAIN_WARPS + 2 && rank == 1 && lane == 0) {
            // ---- the second CTA's parts are stored (each writer fenced its own for the tensor cores); every other block each ----
            const uint32_t first = map_to_cta(full_bar(0), 0);
            int s = warp - (CONV_WARPS + DRAIN_WARPS + 2);
            uint32_t phase = 0;
            for (int kb = s; kb < blocks; kb += 2) {
                if (!mbar_wait(stored_bar(s), phase, &s_abort)) break;
                mbar_arrive_cluster(first + 8u * s);
                if ((s += 2) >= stages) { s -= stages; phase ^= 1u; }
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncwarp();
    cluster_sync_all();                // neither CTA leaves while the other can still signal it or read through it
    if (warp == CONV_WARPS + DRAIN_WARPS) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
    }
    if (tid == 0 && s_abort) atomicExch(status, 1);
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn encode_fn() {
    static const EncodeTiledFn fn = [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        return cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess
                   ? (EncodeTiledFn)p : (EncodeTiledFn) nullptr;
    }();
    return fn;
}
// float32 rows of k elements, ld apart; boxes of 32 elements of box_rows rows
int make_map(CUtensorMap* map, const float* ptr, int k, int rows, long long ld, int box_rows) {
    const EncodeTiledFn fn = encode_fn();
    if (!fn) TQ_FAIL(-3, "gemm_f32: cuTensorMapEncodeTiled is not available from the driver");
    const cuuint64_t dims[2] = {(cuuint64_t)k, (cuuint64_t)rows}, strides[1] = {(cuuint64_t)ld * 4};
    const cuuint32_t box[2] = {(cuuint32_t)BK, (cuuint32_t)box_rows}, elem[2] = {1, 1};
    const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(ptr), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
                          CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) TQ_FAIL(-3, "gemm_f32: cuTensorMapEncodeTiled failed with code %d", (int)r);
    return 0;
}

// Registers that a warpgroup asks for and the block was not launched with never come: the split rests on what the compiler took.
bool registers_suffice() {
    static const int regs = [] { cudaFuncAttributes a; return cudaFuncGetAttributes(&a, gemm_f32_kernel) == cudaSuccess ? a.numRegs : 0; }();
    return regs >= LAUNCH_REGS;
}

}  // namespace

// Whether this build of the kernel can be launched; where not, the products are the library's.
TQ_EXPORT int tq_gemm_f32_runs() { return registers_suffice() ? 1 : 0; }

// x [T, K] with rows ldx floats apart, w [N, K], out [T, N]; K and ldx multiples of four, x and w on 16-byte boundaries.  tokens: of a
// tile (a multiple of 16, at most 256), 0: chosen here.  status: one int, set to 1 if a bounded wait ran out.
TQ_EXPORT int tq_gemm_f32(const float* x, long long ldx, const float* w, float* out, int T, int N, int K, int tokens, int* status, cudaStream_t stream) {
    if (T == 0 || N == 0) return 0;
    TQ_REQUIRE(T > 0 && N > 0 && K > 0, "gemm_f32: bad sizes T=%d N=%d K=%d", T, N, K);
    TQ_REQUIRE(K % 4 == 0 && ldx % 4 == 0 && ldx >= K && ((uintptr_t)x & 15) == 0 && ((uintptr_t)w & 15) == 0, "gemm_f32: rows of %d floats, %lld apart, are not aligned to 16 bytes", K, ldx);
    TQ_REQUIRE(tokens >= 0 && tokens % 16 == 0 && tokens <= MAX_TOKENS, "gemm_f32: tiles of %d tokens", tokens);
    TQ_REQUIRE(status != nullptr, "gemm_f32: a status word is required");
    static std::atomic<unsigned long long> asked{0};
    const cudaError_t e = tq_reserve_smem(gemm_f32_kernel, SMEM_BYTES, asked);
    TQ_REQUIRE(registers_suffice(), "gemm_f32: built with fewer than %d registers a thread", LAUNCH_REGS);
    if (e != cudaSuccess) TQ_FAIL(-1, "gemm_f32: %d bytes of shared memory refused: %s", SMEM_BYTES, cudaGetErrorString(e));
    const int m_tiles = (N + 2 * BM - 1) / (2 * BM);
    int n_t = 0, n = tokens;
    if (n == 0) {
        // tiles of equal numbers of tokens: the number of them that is the least work in a row for the busiest pair of SMs (a block's
        // cycles: 1,090 at 32 tokens, 1,160 at 96, 1,700 at 240 before the result's writing was shortened)
        long long best = 0;
        for (int k = (T + MAX_TOKENS - 1) / MAX_TOKENS; k <= (T + 15) / 16; ++k) {
            if (n != 0 && (long long)m_tiles * (T / (T / k + 16)) / 74 * (256 + 16) >= best) break;       // at least as many tiles, of 16 tokens or more
            const int each = ((T + k - 1) / k + 15) / 16 * 16;
            const long long waves = ((long long)m_tiles * ((T + each - 1) / each) + 73) / 74, cost = waves * (256 + each);
            if (n == 0 || cost < best) { n = each; best = cost; }
        }
    }
    n_t = (T + n - 1) / n;
    TQ_REQUIRE((long long)m_tiles * n_t < (1 << 30), "gemm_f32: too many tiles");
    CUtensorMap mw, mx;
    int rc = make_map(&mw, w, K, N, K, BM);
    if (rc == 0) rc = make_map(&mx, x, K, T, ldx, n / 2);
    if (rc) return rc;
    tq_launch(2 * m_tiles * n_t, THREADS, SMEM_BYTES, stream, 2)(gemm_f32_kernel, mw, mx, x, ldx, w, out, T, N, K, n, n_t, status);
    TQ_CHECK_LAUNCH("gemm_f32");
    return 0;
}
