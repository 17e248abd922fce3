// The true 32-bit path's attention for prompt portions: 32 neighbouring tokens of one request and one head a block.
//
// attention_rows.cu states the arithmetic, a block a token and head.  This kernel does the SAME operations in the same order for every query
// (runs of 128 keys at absolute positions; a score is one fmaf chain over the head's values in order, times the scale; a run's sum of
// probabilities meets in the same tree: lanes 32 keys wide, then the four groups as (0 + 2) + (1 + 3); an output is one fmaf chain over a run's keys in
// order), so a token's output is the same bytes whether it came in a portion (here) or alone (there).  What changes is who does it: a block brings
// 128 keys and values into shared memory once for its 32 queries, and a thread works out 4 x 4 scores from 16-byte loads.
//
// The one-token form reads every key once a query, a cache line a lane, and its outputs' chain stands on 4-byte loads from memory; here a block is
// bound by its multiply-adds and by shared memory (two 16-byte loads a thread for 16 products).  Measured, 512 tokens of 9 heads of 64: 382 us a token
// a block, 45 us here (144 blocks of one to four runs; the multiply-adds alone would be 8 us on all multiprocessors, and the longest block's four
// runs 10 us each).  Tiles of 32 and not 64 queries, because a prompt of 512 tokens would be 72 blocks for 148 multiprocessors.
#include "common.cuh"

namespace vk {

constexpr int RT_THREADS = 256, RT_Q = 32, RT_KEYS = 128;

// HD: the head size rounded up to 64 or 128 (sizes that are multiples of 4); warp w has queries 4 w .. 4 w + 3, lane l keys l, l + 32, l + 64, l + 96
// of a run and, for the outputs, values (HD / 32) l ..
template <int HD>
__global__ void __launch_bounds__(RT_THREADS) attention_rows_tile_kernel(
    const float* __restrict__ q, const float* __restrict__ cache, const int32_t* __restrict__ block_tables, const int32_t* __restrict__ tiles,
    float* __restrict__ out, int nh, int nkv, int hd, int vd, int page_size, int max_blocks, float scale, int window,
    const float* __restrict__ dist_bias, int max_dist, int v_in_key, int v_share, int out_ld, const float* __restrict__ gate, int gate_ld) {
    constexpr int LDK = HD + 4, LDP = RT_KEYS + 4, DV = HD / 32;
    extern __shared__ __align__(16) float rt_smem[];
    float* ks = rt_smem;                        // [128][LDK]
    float* vs = ks + RT_KEYS * LDK;             // [128][HD]
    float* qs = vs + RT_KEYS * HD;              // [32][LDK]
    float* ps = qs + RT_Q * LDK;                // [32][LDP]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, h = blockIdx.y;
    // the longest walks stand last in the list of tiles (64 tokens each, two blocks)
    const int32_t* tile = tiles + 4 * (gridDim.x / 2 - 1 - blockIdx.x / 2);
    const int half = (blockIdx.x & 1) ? 0 : RT_Q;
    const int first = tile[0] + half, rows = min(RT_Q, tile[1] - half), pos0 = tile[2] + half;
    if (rows <= 0) return;
    const int32_t* bt = block_tables + (size_t)tile[3] * max_blocks;
    const int kvh = h / (nh / nkv);
    const size_t page_stride = (size_t)page_size * (v_in_key ? nkv * hd : nkv * hd + nkv / v_share * vd);
    const size_t v_base = v_in_key ? 0 : (size_t)nkv * page_size * hd;
    const int v_stride = v_in_key ? hd : vd;
    for (int e = tid; e < RT_Q * (HD / 4); e += RT_THREADS) {
        const int r = e / (HD / 4), d = 4 * (e % (HD / 4));
        copy16_or_zero(qs + r * LDK + d, q + ((size_t)(first + (r < rows ? r : 0)) * nh + h) * hd + (d < hd ? d : 0), r < rows && d < hd);
    }
    float m[4], l[4], acc[4][DV];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        m[i] = -INFINITY;
        l[i] = 0.0f;
#pragma unroll
        for (int d = 0; d < DV; d++) acc[i][d] = 0.0f;
    }
    const int last = pos0 + rows - 1;
    const int lo_first = (window > 0 && pos0 - window + 1 > 0) ? pos0 - window + 1 : 0;       // the first key any of the queries sees
    for (int c0 = (lo_first / RT_KEYS) * RT_KEYS; c0 <= last; c0 += RT_KEYS) {
        for (int e = tid; e < RT_KEYS * (HD / 4); e += RT_THREADS) {
            const int j = e / (HD / 4), d = 4 * (e % (HD / 4)), key = c0 + j;
            const bool there = key >= lo_first && key <= last;
            const int page = there ? bt[key / page_size] : 0, at = there ? key % page_size : 0;
            const float* base = cache + (size_t)page * page_stride;
            copy16_or_zero(ks + j * LDK + d, base + ((size_t)kvh * page_size + at) * hd + (d < hd ? d : 0), there && d < hd);
            copy16_or_zero(vs + j * HD + d, base + v_base + ((size_t)(kvh / v_share) * page_size + at) * v_stride + (d < vd ? d : 0), there && d < vd);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
        float s[4][4];
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int j = 0; j < 4; j++) s[i][j] = 0.0f;
        const float* qp = qs + 4 * warp * LDK;
        const float* kp = ks + lane * LDK;
#pragma unroll 4
        for (int d = 0; d < hd; d += 4) {
            float4 a[4], b[4];
#pragma unroll
            for (int i = 0; i < 4; i++) a[i] = *reinterpret_cast<const float4*>(qp + i * LDK + d);
#pragma unroll
            for (int j = 0; j < 4; j++) b[j] = *reinterpret_cast<const float4*>(kp + j * 32 * LDK + d);
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    s[i][j] = fmaf(a[i].x, b[j].x, s[i][j]);
                    s[i][j] = fmaf(a[i].y, b[j].y, s[i][j]);
                    s[i][j] = fmaf(a[i].z, b[j].z, s[i][j]);
                    s[i][j] = fmaf(a[i].w, b[j].w, s[i][j]);
                }
        }
        int j0[4], j1[4];                       // the run's keys that a query sees: j0 .. j1 (none: j1 < j0, and the run does not count for it)
        bool all = true;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int pos = pos0 + 4 * warp + i;
            const int lo = (window > 0 && pos - window + 1 > 0) ? pos - window + 1 : 0;
            j0[i] = max(lo, c0) - c0;
            j1[i] = 4 * warp + i < rows ? min(pos, c0 + RT_KEYS - 1) - c0 : -1;
            all = all && j0[i] == 0 && j1[i] == RT_KEYS - 1;
            if (j1[i] < j0[i]) {
#pragma unroll
                for (int j = 0; j < 4; j++) ps[(4 * warp + i) * LDP + lane + 32 * j] = 0.0f;
                continue;
            }
            float mx = -INFINITY;
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const int k = lane + 32 * j;
                float v = __fmul_rn(s[i][j], scale);
                if (dist_bias) {
                    const int n = max(0, pos - (c0 + k));
                    v += dist_bias[(size_t)(n < max_dist ? n : max_dist - 1) * nh + h];
                }
                s[i][j] = (k >= j0[i] && k <= j1[i]) ? v : -INFINITY;
                mx = fmaxf(mx, s[i][j]);
            }
            mx = warp_max(mx);
            const float m_new = fmaxf(m[i], mx);
            float part[4];
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const int k = lane + 32 * j;
                const float p = (k >= j0[i] && k <= j1[i]) ? expf(s[i][j] - m_new) : 0.0f;
                ps[(4 * warp + i) * LDP + k] = p;
                part[j] = warp_sum(p);
            }
            const float corr = expf(m[i] - m_new);          // 0 on the first run, where m is -inf
            l[i] = l[i] * corr + ((part[0] + part[2]) + (part[1] + part[3]));
            m[i] = m_new;
#pragma unroll
            for (int d = 0; d < DV; d++) acc[i][d] *= corr;
        }
        __syncwarp();                           // a warp reads its own four rows of probabilities
        const float* pp = ps + 4 * warp * LDP;
        const float* vp = vs + lane * DV;
        if (all) {
#pragma unroll 2
            for (int j = 0; j < RT_KEYS; j += 4) {
                float4 p[4];
#pragma unroll
                for (int i = 0; i < 4; i++) p[i] = *reinterpret_cast<const float4*>(pp + i * LDP + j);
#pragma unroll
                for (int jj = 0; jj < 4; jj++) {
                    float v[DV];
#pragma unroll
                    for (int d = 0; d < DV; d += 2) { const float2 t = *reinterpret_cast<const float2*>(vp + (j + jj) * HD + d); v[d] = t.x; v[d + 1] = t.y; }
#pragma unroll
                    for (int i = 0; i < 4; i++) {
                        const float w = jj == 0 ? p[i].x : jj == 1 ? p[i].y : jj == 2 ? p[i].z : p[i].w;
#pragma unroll
                        for (int d = 0; d < DV; d++) acc[i][d] = fmaf(w, v[d], acc[i][d]);
                    }
                }
            }
        } else {                                // a run at the diagonal or at a window's edge: a query adds the keys it sees and no others
            int a = RT_KEYS, b = -1;
#pragma unroll
            for (int i = 0; i < 4; i++)
                if (j1[i] >= j0[i]) { a = min(a, j0[i]); b = max(b, j1[i]); }
            for (int j = a; j <= b; j++) {
                float v[DV];
#pragma unroll
                for (int d = 0; d < DV; d += 2) { const float2 t = *reinterpret_cast<const float2*>(vp + j * HD + d); v[d] = t.x; v[d + 1] = t.y; }
#pragma unroll
                for (int i = 0; i < 4; i++)
                    if (j >= j0[i] && j <= j1[i]) {
                        const float w = pp[i * LDP + j];
#pragma unroll
                        for (int d = 0; d < DV; d++) acc[i][d] = fmaf(w, v[d], acc[i][d]);
                    }
            }
        }
        __syncthreads();                        // the next run's keys and values take their place
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int r = 4 * warp + i;
        if (r >= rows) continue;
        const float inv = 1.0f / l[i];
        float* orow = out + (size_t)(first + r) * out_ld + (size_t)h * vd;
#pragma unroll
        for (int d = 0; d < DV; d++)
            if (lane * DV + d < vd) orow[lane * DV + d] = gated(acc[i][d] * inv, gate, gate_ld, first + r, h);
    }
}

}  // namespace vk

using namespace vk;

// Whether the kernel takes these sizes: heads and values of multiples of four up to 128, so that every piece is 16 bytes.
VK_API int vk_attention_rows_tile_takes(int hd, int vd) { return hd > 0 && vd > 0 && hd % 4 == 0 && vd % 4 == 0 && hd <= 128 && vd <= 128; }

// The arguments of vk_attention_rows_biased, float32 alone, with tiles int32 [ntiles][4] (first token, rows up to 64, position of the first token,
// segment) in the place of the tokens' lists.
VK_API int vk_attention_rows_tile(const float* q, const float* cache, const int32_t* block_tables, const int32_t* tiles, float* out, int ntiles, int nh,
                                  int nkv, int hd, int vd, int page_size, int max_blocks, float scale, int window, const float* dist_bias, int max_dist,
                                  int v_in_key, int v_share, int out_ld, const float* gate, int gate_ld, cudaStream_t stream) {
    if (ntiles <= 0) return VK_OK;
    if (nh <= 0 || nkv <= 0 || nh % nkv != 0 || page_size <= 0 || max_blocks <= 0 || window < 0) return VK_BAD_SHAPE;
    if (!vk_attention_rows_tile_takes(hd, vd)) return VK_BAD_SHAPE;
    if (dist_bias && max_dist <= 0) return VK_BAD_SHAPE;
    if (v_in_key && vd > hd) return VK_BAD_SHAPE;
    if (v_share < 1 || nkv % v_share != 0 || (v_in_key && v_share != 1)) return VK_BAD_SHAPE;
    if (out_ld < nh * vd) return VK_BAD_SHAPE;
    if (nh > 65535) return VK_TOO_LARGE;
    if ((uintptr_t)q % 16 || (uintptr_t)cache % 16) return VK_BAD_ALIGNMENT;
    const int HD = (hd > vd ? hd : vd) <= 64 ? 64 : 128;
    const int smem = (RT_KEYS * (HD + 4) + RT_KEYS * HD + RT_Q * (HD + 4) + RT_Q * (RT_KEYS + 4)) * (int)sizeof(float);
    auto kern = HD == 64 ? attention_rows_tile_kernel<64> : attention_rows_tile_kernel<128>;
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return (int)e;
    kern<<<dim3(2 * ntiles, nh), RT_THREADS, smem, stream>>>(q, cache, block_tables, tiles, out, nh, nkv, hd, vd, page_size, max_blocks, scale, window, dist_bias,
                                                             max_dist, v_in_key, v_share, out_ld, gate, gate_ld);
    return launch_status();
}
