// Runs of many tokens in chunks of 64: which tokens a chunk holds.
#pragma once
#include "common.cuh"

namespace tq_recurrence {

constexpr int L = 64;          // tokens of a chunk

// Chunks are numbered sequence after sequence; a sequence has ceil(run / 64).
struct Chunk { int seq, t0, n, in_seq; };      // in_seq: its place among the sequence's; n = 0: there is no such chunk
__device__ __forceinline__ Chunk find_chunk(int chunk, const int* __restrict__ cu_seqlens, int n_seqs, Chunk* s_chunk) {
    if (threadIdx.x < 32) {
        const int lane = threadIdx.x;
        int before = 0;
        Chunk c = {0, 0, 0, 0};
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
                if (i >= 0 && i < k) *s_chunk = Chunk{s, t0 + i * L, min(L, run - i * L), i};
                break;
            }
            before += __shfl_sync(0xffffffffu, upto, 31);
            if (base + 32 >= n_seqs && lane == 0) *s_chunk = c;
        }
    }
    __syncthreads();
    return *s_chunk;
}

}  // namespace tq_recurrence
