// Runs of many tokens in chunks of 64: which tokens a chunk holds, its decays, and where the lanes' shares of its products lie.
#pragma once
#include "common.cuh"

namespace tq_recurrence {

constexpr int L = 64;          // tokens of a chunk
constexpr int LD = 65;         // row stride of a 64 x 64 float32 matrix in shared memory

// Chunks are numbered sequence after sequence; a sequence has ceil(run / 64).
struct Chunk { int seq, t0, n; };      // n = 0: there is no such chunk
__device__ __forceinline__ Chunk find_chunk(int chunk, const int* __restrict__ cu_seqlens, int n_seqs, Chunk* s_chunk) {
    if (threadIdx.x < 32) {
        const int lane = threadIdx.x;
        int before = 0;
        Chunk c = {0, 0, 0};
        for (int base = 0; base < n_seqs; base += 32) {
            const int s = base + lane;
            const int t0 = s < n_seqs ? cu_seqlens[s] : 0, run = s < n_seqs ? cu_seqlens[s + 1] - t0 : 0;
            const int k = (run + L - 1) / L;
            int upto = k;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) { const int v = __shfl_up_sync(0xffffffffu, upto, o); if (lane >= o) upto += v; }
            const int i = chunk - before - (upto - k);
            const unsigned mine = __ballot_sync(0xffffffffu, i >= 0 && i < k);
            if (mine) {
                if (i >= 0 && i < k) *s_chunk = Chunk{s, t0 + i * L, min(L, run - i * L)};
                break;
            }
            before += __shfl_sync(0xffffffffu, upto, 31);
            if (base + 32 >= n_seqs && lane == 0) *s_chunk = c;
        }
    }
    __syncthreads();
    return *s_chunk;
}

__device__ __forceinline__ float4 zero4() { return make_float4(0.f, 0.f, 0.f, 0.f); }
// NaN if one of the four is not finite, else 0
__device__ __forceinline__ float odd(float4 v) { return fmaf(v.x, 0.f, fmaf(v.y, 0.f, fmaf(v.z, 0.f, v.w * 0.f))); }
// row of an accumulator's or left operand's lane, right operand's address parts: [n][k] rows, [k][n] rows
struct Lane {
    int a_row, a_c, b_row, b_c, t_row, t_c, v_row, v_c, r, c;
    __device__ __forceinline__ explicit Lane(int lane)
        : a_row(lane & 15), a_c(lane >> 4),                                      // left operand [m][k]
          b_row(((lane >> 4) << 3) + (lane & 7)), b_c((lane >> 3) & 1),          // right operand lying as [n][k]
          t_row(lane & 15), t_c(lane >> 4),                                      // right operand lying as [k][n]
          v_row(((lane >> 4) << 3) + (lane & 7)), v_c((lane >> 3) & 1),          // left operand lying as [k][m]
          r(lane >> 2), c(2 * (lane & 3)) {}
};

// D[t][s] (zero for s > t) to m, A_t to s_A, D[last] to s_D; g beyond the chunk's tokens is one
__device__ __forceinline__ void decays(float* m, const float* s_g, float* s_A, float* s_D) {
    const int t = threadIdx.x;
    if (t < L) {
        float d = 1.f;
        for (int s = L - 1; s >= 0; --s) {
            if (s < t) d *= s_g[s + 1];
            m[t * LD + s] = s <= t ? d : 0.f;
            if (t == L - 1 && s_D) s_D[s] = d;
        }
    } else if (t == L) {
        float d = 1.f;
        for (int i = 0; i < L; ++i) { d *= s_g[i]; s_A[i] = d; }
    }
}

}  // namespace tq_recurrence
