// Which chunk of a batch a block has: the tokens of the segments of more than `from` tokens in chunks of ROWS, numbered one after another, segment by segment.
#pragma once

#include <stdint.h>

namespace vk {

struct Chunk { int seg, first, rows, start; };      // segment (-1: there is no such chunk), first token, rows, the segment's first token

// sh: four ints of shared memory; every thread of the block calls it and gets the answer.
template <int ROWS>
__device__ __forceinline__ Chunk find_chunk(int n, const int32_t* __restrict__ seg_starts, int segments, int* sh, int from = 0) {
    if (threadIdx.x < 32) {
        const int lane = threadIdx.x;
        int base = 0, found = 0;
        for (int s0 = 0; s0 < segments && !found; s0 += 32) {
            const int s = s0 + lane;
            const int a = s < segments ? seg_starts[s] : 0, b = s < segments ? seg_starts[s + 1] : 0;
            const int mine = b - a > from ? (b - a + ROWS - 1) / ROWS : 0;
            int upto = mine;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, upto, o);
                if (lane >= o) upto += v;
            }
            const int lo = base + upto - mine;
            const bool here = n >= lo && n < lo + mine;
            if (here) {
                sh[0] = s;
                sh[1] = a + (n - lo) * ROWS;
                sh[2] = min(ROWS, b - sh[1]);
                sh[3] = a;
            }
            found = __any_sync(0xffffffffu, here);
            base += __shfl_sync(0xffffffffu, upto, 31);
        }
        if (!found && lane == 0) sh[0] = -1;
    }
    __syncthreads();
    return Chunk{sh[0], sh[1], sh[2], sh[3]};
}

// The number of the first chunk of segment `seg`; the first warp of the block calls it.
template <int ROWS>
__device__ __forceinline__ int first_chunk_of(int seg, const int32_t* __restrict__ seg_starts, int from = 0) {
    int n = 0;
    for (int s = threadIdx.x & 31; s < seg; s += 32) {
        const int len = seg_starts[s + 1] - seg_starts[s];
        n += len > from ? (len + ROWS - 1) / ROWS : 0;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) n += __shfl_xor_sync(0xffffffffu, n, o);
    return n;
}

// The most chunks of a step of `tokens` tokens in `segments` segments.
inline int most_chunks(int rows, int tokens, int segments, int from) {
    const int longer = tokens / (from + 1);             // segments of more than `from` tokens at most, each with one chunk that is not full
    return tokens / rows + (segments < longer ? segments : longer);
}

}  // namespace vk
