// float32 attention of whole runs of new tokens over the paged cache on the tensor cores, every operand as three bfloat16 values
// (split3.cuh), six products of them.
//
// The reference's prompt attention is float32 (src/engine/tq_transformer.c:1909-2191).  On the fp32 units 64 x 64 scores and their part of
// the outputs are 1 M multiply-adds, 8,192 cycles of an SM before a single operand is read from shared memory (the kernel for
// other head sizes, csrc/attention.cu, takes 4.6 times that); as six bfloat16 products they are 6,200 of mma.sync (1,019 multiply-adds a
// cycle and SM measured), whose operands a warp reads once for 16 rows.
// 16 heads of 128, one prompt: 82 us for 700 tokens (287 before), 19 for 100 (47), 420 for 2,048 (1,662); errors against 64 bits
// 1.5e-7 (3.6e-7), queries of spread 5 3.1e-7 (1.05e-6).  What bounds it: the tensor cores are active 39 % of the time, the rest is a warp's
// own chain of splitting, products and exponentials, two warps a scheduler (their sums take 255 registers).
//   A CTA takes 64 consecutive new tokens of one sequence and one query head, a warp of either half of it 16 of them.  Queries, scaled,
//   lie in shared memory in three parts.  The halves take every other 32 keys each, with sums of their own that are put together
//   at the end: one brings and splits while the other multiplies, and the chain of a long row is half as long.  A half's next
//   keys and values come by cp.async, into slots of the thread that will split them.  The last tiles of a run, which see the most
//   keys, start first.
// Sums: the tensor cores cut bits off at every addition, so h h' has accumulators of its own, for 64 elements of a score and for 32 keys
// of an output, which are then added in rounded float32; the smaller products have theirs.  Maxima, exponentials (expf)
// and the rows' sums are float32.  A row whose result is not finite is computed again, key by key.
#include "split3.cuh"

TQ_DEFINE_LAST_ERROR

namespace {

constexpr int BQ = 64, BKEYS = 32, WARPS = 4, HALVES = 2, THREADS = 32 * WARPS * HALVES;

template <int HD>
struct Cfg {
    static constexpr int Q_PART = BQ * HD * 2, K_PART = BKEYS * HD * 2;
    static constexpr int RAW = 2 * BKEYS * HD * 4, HALF = 6 * K_PART + RAW;              // a half's keys and values, in parts and as they come
    static constexpr int SMEM_BYTES = 3 * Q_PART + HALVES * HALF;
    static_assert(BQ * (HD + 4) * 4 <= HALF, "the second half's sums take the place of its keys");
};

__device__ __forceinline__ void half_sync(int half) { asm volatile("bar.sync %0, %1;" ::"r"(half + 1), "n"(32 * WARPS) : "memory"); }
// 16 bytes, or as many zeros
__device__ __forceinline__ void cp16(uint32_t dst, const float* src, bool there) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(there ? 16 : 0) : "memory");
}

template <int HD>
__global__ void __launch_bounds__(THREADS, 1)
attention_f32_kernel(const float* __restrict__ q, const float* __restrict__ cache, const int* __restrict__ cu_seqlens,
                     const int* __restrict__ seq_start, const int* __restrict__ page_table, int table_stride, int page_size, int window,
                     float scale, float* __restrict__ out, int n_seqs, int nh, int nkv, int n_pages) {
    tq_grid_wait();                    // everything below may read what the previous kernel wrote
    tq_grid_launch_dependents();       // the next kernel's CTAs may move in as SMs free up
    using C = Cfg<HD>;
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ int s_seq, s_row0;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5 & (WARPS - 1), half = threadIdx.x / (32 * WARPS);
    if (threadIdx.x == 0) {            // which sequence's which 64 rows this CTA takes, a sequence's last ones first
        int tile = blockIdx.x / nh, seq = -1, row0 = 0;
        for (int i = 0; i < n_seqs; ++i) {
            const int n = cu_seqlens[i + 1] - cu_seqlens[i], tiles = (n + BQ - 1) / BQ;
            if (tile < tiles) { seq = i; row0 = (tiles - 1 - tile) * BQ; break; }
            tile -= tiles;
        }
        s_seq = seq; s_row0 = row0;
    }
    __syncthreads();
    const int seq = s_seq;
    if (seq < 0) return;               // the grid is an upper bound of the number of tiles
    const int h = blockIdx.x % nh, g = h / (nh / nkv);
    const int t_first = cu_seqlens[seq] + s_row0, rows = min(BQ, cu_seqlens[seq + 1] - t_first);
    const int pos0 = seq_start[seq] + s_row0;                // position of the tile's first row
    const int* table = page_table + (size_t)seq * table_stride;
    const size_t v_plane = (size_t)nkv * page_size * HD;
    auto key_row = [&](int p) {
        const int page = TQ_CHECKED(table[TQ_CHECKED(p / page_size, table_stride, TQ_IDX_TABLE_COLUMN)], n_pages, TQ_IDX_PAGE);
        return cache + (((size_t)page * 2 * nkv + g) * page_size + p % page_size) * HD;
    };
    const uint32_t sq = tq_smem_u32(smem), sk = sq + 3 * C::Q_PART + half * C::HALF, sv = sk + 3 * C::K_PART;
    const uint32_t raw = sv + 3 * C::K_PART + (threadIdx.x & (32 * WARPS - 1)) * 16;
    constexpr int LANES = HD / 4, RPW = 32 / LANES;           // lanes of a row, rows a warp brings at a time
    const int sub = lane / LANES, d4 = lane % LANES * 4;
    for (int r = (half * WARPS + warp) * RPW + sub; r < BQ; r += HALVES * WARPS * RPW) {
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (r < rows) v = *reinterpret_cast<const float4*>(q + ((size_t)(t_first + r) * nh + h) * HD + d4);
        v.x *= scale; v.y *= scale; v.z *= scale; v.w *= scale;
        tq_put4<HD>(sq, C::Q_PART, r, d4, v);
    }
    // the thread's rows: two, of the accumulators' layout (lane / 4 and 8 below)
    const int row_a = warp * 16 + (lane >> 2), pos_a = pos0 + row_a, pos_b = pos_a + 8;
    const int pos_w0 = pos0 + warp * 16, pos_w1 = pos0 + min(rows - 1, warp * 16 + 15);       // the warp's first and last
    const int k_lo = window > 0 ? max(0, pos0 + 1 - window) : 0, k_hi = pos0 + rows - 1;
    const int start_a = window > 0 ? max(0, pos_a + 1 - window) : 0, start_b = window > 0 ? max(0, pos_b + 1 - window) : 0;
    const int start_w = window > 0 ? max(0, pos_w0 + 1 - window) : 0;
    const bool has_rows = warp * 16 < rows;
    const bool one_page = page_size % BKEYS == 0;             // a tile of keys lies in one page: one look-up, not one a row
    float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f}, o[HD / 8][4];
#pragma unroll
    for (int j = 0; j < HD / 8; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) o[j][e] = 0.f;
    const int a_row = warp * 16 + (lane & 15), a_c = lane >> 4;                                // ldmatrix addresses: queries,
    const int b_row = ((lane >> 4) << 3) + (lane & 7), b_c = (lane >> 3) & 1;                  // keys,
    const int v_row = lane & 15, v_c = lane >> 4;                                              // values

    constexpr int EACH = BKEYS / (WARPS * RPW);              // rows of a tile that a thread brings four elements of
    auto bring = [&](int k0) {
        if (k0 <= k_hi) {
            const int p0 = max(k0, k_lo);
            const float* tile = one_page ? key_row(p0) - (ptrdiff_t)(p0 - k0) * HD : nullptr;
#pragma unroll
            for (int i = 0; i < EACH; ++i) {
                const int p = k0 + (i * WARPS + warp) * RPW + sub;
                const bool there = p >= k_lo && p <= k_hi;
                const float* at = !there ? cache : (one_page ? tile + (size_t)(p - k0) * HD : key_row(p)) + d4;
                cp16(raw + i * (32 * WARPS * 16), at, there);
                cp16(raw + (EACH + i) * (32 * WARPS * 16), there ? at + v_plane : cache, there);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    const int k_first = k_lo / BKEYS * BKEYS + half * BKEYS;
    bring(k_first);
    __syncthreads();                   // the queries are there
    for (int k0 = k_first; k0 <= k_hi; k0 += HALVES * BKEYS) {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        half_sync(half);               // the previous keys and values have been used
#pragma unroll
        for (int i = 0; i < 2 * EACH; ++i) {
            float4 v;
            asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(raw + i * (32 * WARPS * 16)) : "memory");
            tq_put4<HD>(i < EACH ? sk : sv, C::K_PART, (i % EACH * WARPS + warp) * RPW + sub, d4, v);
        }
        bring(k0 + HALVES * BKEYS);
        half_sync(half);
        if (!has_rows || k0 > pos_w1 || k0 + BKEYS <= start_w) continue;     // nothing the warp's rows see
        float s[4][4];                 // scores of 16 rows and four groups of eight keys
        {
            float rest[4][4], first[4][4];
#pragma unroll
            for (int k = 0; k < HD / 16; ++k) {
                if (k == 4) {
#pragma unroll
                    for (int j = 0; j < 4; ++j)
#pragma unroll
                        for (int e = 0; e < 4; ++e) first[j][e] = s[j][e];
                }
                uint32_t a[3][4], b[3][2][4];
#pragma unroll
                for (int part = 0; part < 3; ++part) {
                    tq_ldm4(a[part], sq + part * C::Q_PART + tq_piece<HD>(a_row, 2 * k + a_c));
#pragma unroll
                    for (int jp = 0; jp < 2; ++jp) tq_ldm4(b[part][jp], sk + part * C::K_PART + tq_piece<HD>(16 * jp + b_row, 2 * k + b_c));
                }
                if (k == 0) tq_six<4, true, true>(s, rest, a, b);
                else if (k == 4) tq_six<4, true, false>(s, rest, a, b);
                else tq_six<4, false, false>(s, rest, a, b);
            }
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
                for (int e = 0; e < 4; ++e) s[j][e] = (HD > 64 ? first[j][e] + s[j][e] : s[j][e]) + rest[j][e];
        }
        // what a row does not see; maxima; exponentials
        if (k0 + BKEYS - 1 > pos_w0 || k0 < max(0, start_w + 15))
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int p = k0 + 8 * j + 2 * (lane & 3) + (e & 1);
                const bool sees = e < 2 ? p <= pos_a && p >= start_a : p <= pos_b && p >= start_b;
                if (!sees) s[j][e] = -INFINITY;
            }
        float top[2] = {m[0], m[1]};
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) top[e >> 1] = fmaxf(top[e >> 1], s[j][e]);
        float corr[2];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            top[r] = fmaxf(top[r], __shfl_xor_sync(0xffffffffu, top[r], 1));
            top[r] = fmaxf(top[r], __shfl_xor_sync(0xffffffffu, top[r], 2));
            corr[r] = top[r] == -INFINITY ? 1.f : expf(m[r] - top[r]);          // exp(-inf) = 0 the first time
            l[r] *= corr[r];
            m[r] = top[r];
        }
        uint32_t p[2][3][4];                                                     // weights as left operands, 16 keys each
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const float e0 = top[r] == -INFINITY ? 0.f : expf(s[j][2 * r] - top[r]), e1 = top[r] == -INFINITY ? 0.f : expf(s[j][2 * r + 1] - top[r]);
                l[r] += e0 + e1;
                const int at = 2 * (j & 1) + r;
                tq_split2(e0, e1, p[j >> 1][0][at], p[j >> 1][1][at], p[j >> 1][2][at]);
            }
#pragma unroll
        for (int j4 = 0; j4 < HD / 32; ++j4) {                                   // 32 elements of the output at a time
            float t[4][4], rest[4][4];
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                uint32_t b[3][2][4];
#pragma unroll
                for (int part = 0; part < 3; ++part)
#pragma unroll
                    for (int jp = 0; jp < 2; ++jp) tq_ldm4t(b[part][jp], sv + part * C::K_PART + tq_piece<HD>(16 * k + v_row, 4 * j4 + 2 * jp + v_c));
                if (k == 0) tq_six<4, true, true>(t, rest, p[k], b);
                else tq_six<4, false, false>(t, rest, p[k], b);
            }
#pragma unroll
            for (int u = 0; u < 4; ++u)
#pragma unroll
                for (int e = 0; e < 4; ++e) o[4 * j4 + u][e] = o[4 * j4 + u][e] * corr[e >> 1] + (t[u][e] + rest[u][e]);
        }
    }
    // the second half's sums to the first, by way of its keys' place: [row][HD], then maxima and totals
    __syncthreads();
    float* theirs = reinterpret_cast<float*>(smem + 3 * C::Q_PART + C::HALF);
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        l[r] += __shfl_xor_sync(0xffffffffu, l[r], 1);
        l[r] += __shfl_xor_sync(0xffffffffu, l[r], 2);
    }
    if (half == 1) {
#pragma unroll
        for (int r = 0; r < 2; ++r) {
#pragma unroll
            for (int j = 0; j < HD / 8; ++j)
                *reinterpret_cast<float2*>(theirs + (row_a + 8 * r) * HD + 8 * j + 2 * (lane & 3)) = make_float2(o[j][2 * r], o[j][2 * r + 1]);
            theirs[BQ * HD + row_a + 8 * r] = m[r];
            theirs[BQ * HD + BQ + row_a + 8 * r] = l[r];
        }
    }
    __syncthreads();
    if (half == 1) return;
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const float m1 = theirs[BQ * HD + row_a + 8 * r], l1 = theirs[BQ * HD + BQ + row_a + 8 * r], top = fmaxf(m[r], m1);
        const float c0 = m[r] == -INFINITY ? 0.f : expf(m[r] - top), c1 = m1 == -INFINITY ? 0.f : expf(m1 - top);
        l[r] = l[r] * c0 + l1 * c1;
#pragma unroll
        for (int j = 0; j < HD / 8; ++j) {
            const float2 v = *reinterpret_cast<const float2*>(theirs + (row_a + 8 * r) * HD + 8 * j + 2 * (lane & 3));
            o[j][2 * r] = o[j][2 * r] * c0 + v.x * c1;
            o[j][2 * r + 1] = o[j][2 * r + 1] * c0 + v.y * c1;
        }
    }
    bool fine[2] = {true, true};
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const float inv = 1.0f / l[r];
        float* op = out + ((size_t)(t_first + row_a + 8 * r) * nh + h) * HD + 2 * (lane & 3);
#pragma unroll
        for (int j = 0; j < HD / 8; ++j) {
            const float2 v = make_float2(o[j][2 * r] * inv, o[j][2 * r + 1] * inv);
            if (row_a + 8 * r < rows) *reinterpret_cast<float2*>(op + 8 * j) = v;
            fine[r] &= isfinite(v.x) && isfinite(v.y);
        }
    }
    // rows that met an infinity or a NaN, key by key: the parts of a value cannot say which it was
    unsigned again = 0;
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const unsigned b = __ballot_sync(0xffffffffu, !fine[r] && row_a + 8 * r < rows);
        for (int i = 0; i < 8; ++i)
            if (b >> (4 * i) & 15u) again |= 1u << (8 * r + i);
    }
    while (again) {
        const int row = warp * 16 + __ffs(again) - 1, pos = pos0 + row;
        again &= again - 1;
        float qr[HD / 32], acc[HD / 32], mx = -INFINITY, sum = 0.f;
        const size_t at = ((size_t)(t_first + row) * nh + h) * HD;
#pragma unroll
        for (int c = 0; c < HD / 32; ++c) { qr[c] = q[at + lane + 32 * c] * scale; acc[c] = 0.f; }
        for (int p = window > 0 ? max(0, pos + 1 - window) : 0; p <= pos; ++p) {
            const float* kr = key_row(p);
            float sc = 0.f;
#pragma unroll
            for (int c = 0; c < HD / 32; ++c) sc = fmaf(qr[c], kr[lane + 32 * c], sc);
            sc = tq_warp_sum(sc);
            const float up = fmaxf(mx, sc);
            const float c0 = up == -INFINITY ? 1.f : expf(mx - up), e = up == -INFINITY ? 0.f : expf(sc - up);
            sum = sum * c0 + e;
            mx = up;
#pragma unroll
            for (int c = 0; c < HD / 32; ++c) acc[c] = fmaf(e, kr[v_plane + lane + 32 * c], acc[c] * c0);
        }
#pragma unroll
        for (int c = 0; c < HD / 32; ++c) out[at + lane + 32 * c] = acc[c] * (1.0f / sum);
    }
}

template <int HD>
int launch(const float* q, const float* cache, const int* cu_seqlens, const int* seq_start, const int* page_table, int table_stride, int page_size,
           int window, float scale, float* out, int T, int n_seqs, int nh, int nkv, int n_pages, cudaStream_t stream) {
    static std::atomic<unsigned long long> asked{0};
    const cudaError_t e = tq_reserve_smem(attention_f32_kernel<HD>, Cfg<HD>::SMEM_BYTES, asked);
    if (e != cudaSuccess) TQ_FAIL(-1, "attention_f32: %d bytes of shared memory refused: %s", Cfg<HD>::SMEM_BYTES, cudaGetErrorString(e));
    tq_launch(nh * (T / BQ + n_seqs), THREADS, Cfg<HD>::SMEM_BYTES, stream)(attention_f32_kernel<HD>, q, cache, cu_seqlens, seq_start, page_table,
        table_stride, page_size, window, scale, out, n_seqs, nh, nkv, n_pages);
    TQ_CHECK_LAUNCH("attention_f32");
    return 0;
}

}  // namespace

// q, out [T, nh, hd], cache [pages, 2, nkv, page_size, hd], float32 on 16-byte boundaries; hd 64 or 128.  Sequence i's rows are
// cu_seqlens[i] .. cu_seqlens[i + 1], the first at position seq_start[i]; the step's keys and values are in the cache.
TQ_EXPORT int tq_attention_f32(const float* q, const float* cache, const int* cu_seqlens, const int* seq_start, const int* page_table, int table_stride,
                               int page_size, int window, float scale, float* out, int T, int n_seqs, int nh, int nkv, int hd, int n_pages,
                               cudaStream_t stream) {
    if (T == 0) return 0;
    TQ_REQUIRE(hd == 64 || hd == 128, "attention_f32: head size %d is not 64 or 128", hd);
    TQ_REQUIRE(nkv >= 1 && nh >= 1 && nh % nkv == 0, "attention_f32: %d heads are not a multiple of %d key/value heads", nh, nkv);
    TQ_REQUIRE(n_seqs >= 1 && (long long)nh * (T / BQ + n_seqs) < (1ll << 31), "attention_f32: bad grid (%d tokens, %d sequences)", T, n_seqs);
    TQ_REQUIRE(window >= 0 && page_size >= 1, "attention_f32: window %d, pages of %d", window, page_size);
    TQ_REQUIRE(((uintptr_t)q & 15) == 0 && ((uintptr_t)cache & 15) == 0 && ((uintptr_t)out & 7) == 0, "attention_f32: operands are not aligned to 16 bytes");
#define ATT_ARGS q, cache, cu_seqlens, seq_start, page_table, table_stride, page_size, window, scale, out, T, n_seqs, nh, nkv, n_pages, stream
    return hd == 64 ? launch<64>(ATT_ARGS) : launch<128>(ATT_ARGS);
#undef ATT_ARGS
}
