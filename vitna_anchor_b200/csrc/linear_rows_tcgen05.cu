// The matrix product of a few dozen rows in bfloat16 on the fifth-generation tensor cores: out[M, N] = x[M, K] * W[N, K]^T, M <= 64, with the weights as
// the 128-row operand.
//
// Decoding a few dozen requests together streams every weight once; what bounds it is how many bytes of weights are on their way.  A tile is 128 rows of the
// weights (tensor-core rows) by all batch rows (its 16, 32 or 64 columns), so that a stage of the ring is 16 KB of weights and at most 8 KB of x, and a
// block needs no register and no issue slot for a weight.  Where the tiles are fewer than the multiprocessors, K is split over a cluster's blocks: each
// leaves its float32 sums in its shared memory, and every block of the cluster adds up a share of the batch rows over all of them, in the order of the
// splits, and finishes it.  The first four stages' weights are asked for before the wait on the kernel before this one.
//
//   warp 0   one lane: TMA copies into a ring of four stages (64 columns of K each)
//   warp 1   one lane: tcgen05.mma, 128 x NB x 16, to the tile's accumulators in turn
//   warps 2-5  the accumulators out of tensor memory, added up in float32, into shared memory, [batch row][weight row]
//   all      the sums over the cluster, and the epilogue: a thread has four neighbouring output columns of a batch row
//
// Measured over weights that are not in the second-level cache, 64 rows, what stands in otherwise (mma.sync with the weights through registers up to 8,192 columns, else
// tiles of 128 batch rows) / this: 6,144 x 2,048 26.8 / 10.4 us (2.4 TB/s), 2,048 x 8,192 into a sum 33.2 / 12.8 (2.6 TB/s), 16,384 x 2,048 gated 22.1 / 18.6 (3.6 TB/s; 128 tiles
// are what 128 multiprocessors pull), 5,120 x 960 gated 15.5 / 8.5; 16 rows of 49,152 x 2,048 57.6 / 33.4 (6.0 TB/s), one of 49,152 x 576 18.8 / 10.9 (5.2 TB/s).  About 3.4 us of
// a launch are not the stream: set-up, the first copies' way, the cluster's meeting and the epilogue; that is why small matrices stay with linear_skinny_mma.cu.
//
// The tensor core cuts off what a sum in tensor memory has no bits for, every time that it adds to it, so that an error grows with the products that are added to
// one accumulator one after another.  The mma.sync kernels split K over a block's eight warps; here the blocks of a cluster and the accumulators that a block's
// products go to in turn (`accs`) make as many such chains of an output.  Error against 64 bits over the result's size (2-norms, random operands), the mma.sync kernel / one
// accumulator a block / as here, in 1e-7: 49,152 x 576 1.09 / 5.5 / 1.00, 5,120 x 960 1.53 / 2.9 / 1.14, 6,144 x 2,048 2.36 / 6.5 / 2.1, 2,048 x 8,192 9.96 / 9.95 / 9.95 (eight blocks
// share K there); 16,384 x 2,048, in tiles of 128 rows otherwise, 21 / 21 / 4.7.
//
// An output does not depend on M or on the other batch rows: the splits of K and the accumulators depend on N and K alone.  Every wait on an mbarrier is bounded (see
// tcgen05_common.cuh); a block that gave up still meets its cluster.
#include "tcgen05_common.cuh"

namespace vk {

constexpr int RT_BM = 128, RT_BK = 64, RT_STAGES = 4, RT_THREADS = 192, RT_MAX_SPLIT = 8, RT_CHAINS = 8;
enum { RT_SAME = 0, RT_F32 = 1, RT_ACC = 2, RT_SWIGLU = 3, RT_ROPE = 4 };

struct RtArgs {
    void* out;
    int M, N, K, splits, accs;   // accs: accumulators that a block's products go to in turn
    int act;                     // RT_SAME: an activation on the float32 sums (activate_dense; 0 none); RT_SWIGLU: the gate's function (0: silu)
    const int32_t* positions;
    const float* cos_t;
    const float* sin_t;
    const int32_t* slot;
    __nv_bfloat16* cache;
    int nh, nkv, hd, page_size;
};

__device__ __forceinline__ float4 ld_peer4(uint32_t local, int rank) {
    uint32_t at;
    float4 v;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(local), "r"(rank));
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(at) : "memory");
    return v;
}
// The sums of four neighbouring weight rows for a batch row, over the cluster's blocks in their order.
__device__ __forceinline__ float4 rt_sum4(const float* red, int m, int c, int splits) {
    const uint32_t at = smem_u32(red + m * RT_BM + c);
    if (splits == 1) return *reinterpret_cast<const float4*>(red + m * RT_BM + c);
    float4 v[RT_MAX_SPLIT];
#pragma unroll
    for (int s = 0; s < RT_MAX_SPLIT; s++)
        if (s < splits) v[s] = ld_peer4(at, s);
    float4 t = v[0];
#pragma unroll
    for (int s = 1; s < RT_MAX_SPLIT; s++)
        if (s < splits) { t.x += v[s].x; t.y += v[s].y; t.z += v[s].z; t.w += v[s].w; }
    return t;
}
__device__ __forceinline__ uint2 rt_pack4(float a, float b, float c, float d) {
    __nv_bfloat162 lo = __floats2bfloat162_rn(a, b), hi = __floats2bfloat162_rn(c, d);
    return make_uint2(*reinterpret_cast<uint32_t*>(&lo), *reinterpret_cast<uint32_t*>(&hi));
}
__device__ __forceinline__ float rt_round(float v) { return __bfloat162float(__float2bfloat16_rn(v)); }

// 16 or 32 columns of this thread's lane of tensor memory.
template <int COLS>
__device__ __forceinline__ void rt_load(uint32_t taddr, uint32_t* r) {
    if constexpr (COLS == 16) {
        tmem_ld16(taddr, r);
    } else {
        tmem_ld32(taddr, r);
        tmem_loaded(r);
    }
}

// Columns of tensor memory for `accs` accumulators of nb columns: a power of two, at least 32.
__host__ __device__ __forceinline__ uint32_t rt_tmem_columns(int nb, int accs) {
    uint32_t c = 32;
    while (c < (uint32_t)(nb * accs)) c *= 2;
    return c;
}

// grid (tiles * splits), a cluster of `splits` blocks a tile
template <int NB, int EPI>
__global__ void __launch_bounds__(RT_THREADS) linear_rows_tcgen05_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w,
                                                                         const RtArgs p, const WaitCtl wc) {
    constexpr uint32_t W_BYTES = RT_BM * RT_BK * 2, X_BYTES = NB * RT_BK * 2, STAGE_BYTES = W_BYTES + X_BYTES;
    static_assert(NB * RT_BM * 4 <= RT_STAGES * STAGE_BYTES, "the sums take the stages' place");
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + RT_STAGES * STAGE_BYTES);
    uint64_t* empty = full + RT_STAGES;
    uint64_t* acc_full = empty + RT_STAGES;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_full + 1);
    float* red = reinterpret_cast<float*>(smem);        // [NB][128], once every product has read its stage
    __shared__ int failed;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int splits = p.splits, tile = blockIdx.x / splits, rank = blockIdx.x % splits;
    const int n0 = tile * (EPI == RT_SWIGLU ? RT_BM / 2 : RT_BM);
    const uint32_t tm_cols = rt_tmem_columns(NB, p.accs);
    const int num_kb = (p.K + RT_BK - 1) / RT_BK, kb0 = rank * num_kb / splits, n_kb = (rank + 1) * num_kb / splits - kb0;      // at least one

    auto load_w = [&](int kb, int s) {
        uint8_t* dst = smem + s * STAGE_BYTES;
        if (EPI == RT_SWIGLU) {                // 64 gate rows and the same 64 up rows: the map's box is 64 rows
            tma_load_2d(dst, &map_w, (kb0 + kb) * RT_BK, n0, &full[s]);
            tma_load_2d(dst + W_BYTES / 2, &map_w, (kb0 + kb) * RT_BK, p.N / 2 + n0, &full[s]);
        } else {
            tma_load_2d(dst, &map_w, (kb0 + kb) * RT_BK, n0, &full[s]);
        }
    };
    // (a stage named by wc.skip_stage is left unarmed and unfilled: a test of the give-up path)
    const int early = n_kb < RT_STAGES ? n_kb : RT_STAGES;
    if (threadIdx.x == 0) {
        failed = 0;
        for (int s = 0; s < RT_STAGES; s++) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
        mbar_init(acc_full, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        // the first weights, before the block has its tensor memory: under the end of a kernel whose blocks hold the multiprocessor's, that is a long wait
        for (int kb = 0; kb < early; kb++) {
            if (kb == wc.skip_stage) continue;
            mbar_expect_tx(&full[kb], STAGE_BYTES);
            load_w(kb, kb);
        }
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(tm_cols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    if (warp == 0) {
        if (lane == 0) {
            dependency_wait();
            for (int kb = 0; kb < early; kb++)
                if (kb != wc.skip_stage) tma_load_2d(smem + kb * STAGE_BYTES + W_BYTES, &map_x, (kb0 + kb) * RT_BK, 0, &full[kb]);
            for (int kb = early; kb < n_kb; kb++) {
                const int s = kb % RT_STAGES;
                if (!mbar_wait(&empty[s], ((kb / RT_STAGES) & 1) ^ 1, wc.cycles)) { give_up(wc.error, &failed, 71); break; }
                if (kb == wc.skip_stage) continue;
                mbar_expect_tx(&full[s], STAGE_BYTES);
                load_w(kb, s);
                tma_load_2d(smem + s * STAGE_BYTES + W_BYTES, &map_x, (kb0 + kb) * RT_BK, 0, &full[s]);
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            const uint32_t idesc = umma_idesc_bf16(RT_BM, NB);
            const uint32_t w_lo0 = umma_desc_lo(smem_u32(smem)), acc_end = tmem + NB * p.accs;
            uint32_t acc = tmem, add = 0;              // the first product of an accumulator writes it; half a stage's products go to one
            for (int kb = 0; kb < n_kb; kb++) {
                const int s = kb % RT_STAGES;
                if (!mbar_wait(&full[s], (kb / RT_STAGES) & 1, wc.cycles)) { give_up(wc.error, &failed, 72); break; }
                tc_fence_after();
                const uint32_t w_lo = w_lo0 + s * (STAGE_BYTES >> 4), x_lo = w_lo + (W_BYTES >> 4);
#pragma unroll
                for (int k = 0; k < RT_BK / 16; k += 2) {
                    umma_bf16_lo(acc, w_lo + 2 * k, x_lo + 2 * k, idesc, add);
                    umma_bf16_lo(acc, w_lo + 2 * k + 2, x_lo + 2 * k + 2, idesc, 1);
                    acc += NB;
                    if (acc == acc_end) { acc = tmem; add = 1; }
                }
                umma_commit(&empty[s]);
            }
            umma_commit(acc_full);                     // arrives when every instruction has written the accumulator
        }
    } else {
        if (!mbar_wait(acc_full, 0, wc.cycles)) { if (lane == 0) give_up(wc.error, &failed, 73); }
        __syncwarp();
        const int quarter = warp & 3;
        const uint32_t acc = tmem + ((uint32_t)(quarter * 32) << 16);
        // after a failed wait a copy may still be on its way into the stages: the sums are not written, what is added up is not valid
        const bool ok = *reinterpret_cast<volatile int*>(&failed) == 0;
        tc_fence_after();
        if (__all_sync(0xffffffffu, ok)) {
            float* mine = red + quarter * 32 + lane;
            const int used = min(p.accs, n_kb * (RT_BK / 32));
            constexpr int COLS = NB < 32 ? NB : 32;
#pragma unroll
            for (int c = 0; c < NB; c += COLS) {
                uint32_t sum[COLS];
                rt_load<COLS>(acc + c, sum);
#pragma unroll 1
                for (int a = 1; a < used; a++) {
                    uint32_t r[COLS];
                    rt_load<COLS>(acc + a * NB + c, r);
#pragma unroll
                    for (int j = 0; j < COLS; j++) sum[j] = __float_as_uint(__uint_as_float(sum[j]) + __uint_as_float(r[j]));
                }
#pragma unroll
                for (int j = 0; j < COLS; j++) mine[(c + j) * RT_BM] = __uint_as_float(sum[j]);
            }
        }
        tc_fence_before();
    }
    __syncwarp();
    dependency_wait();                                 // what is read and written from here on is after the kernel before this one
    let_dependents_start();
    if (splits > 1) cluster_meet();
    else __syncthreads();

    // the batch rows rank, rank + splits, ..: a thread takes four neighbouring columns of one at a time
    constexpr int PIECES = EPI == RT_SWIGLU || EPI == RT_ROPE ? RT_BM / 8 : RT_BM / 4;
    const int my_rows = (p.M - rank + splits - 1) / splits;
    for (int it = threadIdx.x; it < my_rows * PIECES; it += RT_THREADS) {
        const int m = rank + (it / PIECES) * splits, piece = it % PIECES;
        if (EPI == RT_SWIGLU) {
            const int inter = p.N / 2, col = n0 + 4 * piece;
            const float4 g = rt_sum4(red, m, 4 * piece, splits), u = rt_sum4(red, m, RT_BM / 2 + 4 * piece, splits);
            const float gv[4] = {g.x, g.y, g.z, g.w}, uv[4] = {u.x, u.y, u.z, u.w};
            float v[4];
#pragma unroll
            for (int e = 0; e < 4; e++) {
                const float a = rt_round(gv[e]), b = rt_round(uv[e]);
                v[e] = (p.act ? activate_rt(p.act, a) : a / (1.0f + expf(-a))) * b;
            }
            if (col < inter) *reinterpret_cast<uint2*>(reinterpret_cast<__nv_bfloat16*>(p.out) + (size_t)m * inter + col) = rt_pack4(v[0], v[1], v[2], v[3]);
        } else if (EPI == RT_ROPE) {
            const int half = p.hd / 2, per_head = half / 4;                // pieces of four pairs a head
            const int hh = piece / per_head, j = 4 * (piece % per_head), head = n0 / p.hd + hh;
            if (head >= p.nh + 2 * p.nkv) continue;
            const float4 a4 = rt_sum4(red, m, hh * p.hd + j, splits), b4 = rt_sum4(red, m, hh * p.hd + half + j, splits);
            const bool is_q = head < p.nh, is_k = !is_q && head < p.nh + p.nkv;
            __nv_bfloat16* dst = nullptr;
            if (is_q) dst = reinterpret_cast<__nv_bfloat16*>(p.out) + ((size_t)m * p.nh + head) * p.hd;
            else {
                const int sl = p.slot[m], kvh = is_k ? head - p.nh : head - p.nh - p.nkv;
                if (sl >= 0)
                    dst = p.cache + (size_t)(sl / p.page_size) * 2 * p.nkv * p.page_size * p.hd + (is_k ? 0 : (size_t)p.nkv * p.page_size * p.hd) +
                          ((size_t)kvh * p.page_size + sl % p.page_size) * p.hd;
            }
            if (!dst) continue;
            const float av[4] = {rt_round(a4.x), rt_round(a4.y), rt_round(a4.z), rt_round(a4.w)}, bv[4] = {rt_round(b4.x), rt_round(b4.y), rt_round(b4.z), rt_round(b4.w)};
            float ra[4], rb[4];
            if (is_q || is_k) {
                const int pos = p.positions[m];
                const float4 c4 = *reinterpret_cast<const float4*>(p.cos_t + (size_t)pos * half + j), s4 = *reinterpret_cast<const float4*>(p.sin_t + (size_t)pos * half + j);
                const float cs[4] = {c4.x, c4.y, c4.z, c4.w}, sn[4] = {s4.x, s4.y, s4.z, s4.w};
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    ra[e] = av[e] * cs[e] - bv[e] * sn[e];
                    rb[e] = bv[e] * cs[e] + av[e] * sn[e];
                }
            } else {
#pragma unroll
                for (int e = 0; e < 4; e++) { ra[e] = av[e]; rb[e] = bv[e]; }
            }
            *reinterpret_cast<uint2*>(dst + j) = rt_pack4(ra[0], ra[1], ra[2], ra[3]);
            *reinterpret_cast<uint2*>(dst + half + j) = rt_pack4(rb[0], rb[1], rb[2], rb[3]);
        } else {
            const int col = n0 + 4 * piece;
            if (col >= p.N) continue;                  // (N is a multiple of four)
            const size_t at = (size_t)m * p.N + col;
            float4 old = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (EPI == RT_ACC) old = *reinterpret_cast<const float4*>(reinterpret_cast<float*>(p.out) + at);
            float4 v = rt_sum4(red, m, 4 * piece, splits);
            if (EPI == RT_SAME) {
                if (p.act) { v.x = activate_dense(p.act, v.x); v.y = activate_dense(p.act, v.y); v.z = activate_dense(p.act, v.z); v.w = activate_dense(p.act, v.w); }
                *reinterpret_cast<uint2*>(reinterpret_cast<__nv_bfloat16*>(p.out) + at) = rt_pack4(v.x, v.y, v.z, v.w);
            } else {
                *reinterpret_cast<float4*>(reinterpret_cast<float*>(p.out) + at) = make_float4(old.x + v.x, old.y + v.y, old.z + v.z, old.w + v.w);
            }
        }
    }
    __syncwarp();
    tc_fence_before();
    if (splits > 1) cluster_meet();                    // the others have read this block's sums
    else __syncthreads();
    if (warp == 1) {
        if (failed) __nanosleep(200000);               // after a failed wait: let copies in flight land
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(tm_cols) : "memory");
    }
}

static bool rt_make_map(CUtensorMap* map, const void* base, int rows, int cols, int ld, int box_rows) {
    EncodeTiledFn enc = encode_tiled();
    if (!enc) return false;
    cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
    cuuint32_t box[2] = {(cuuint32_t)RT_BK, (cuuint32_t)box_rows};
    cuuint32_t elem[2] = {1, 1};
    return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
               CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Blocks that share a tile's K: as many as the multiprocessors have room for, at most eight (a cluster anywhere), at least one step of 64 columns each.
static int rt_splits(int tiles, int K) {
    const int num_kb = (K + RT_BK - 1) / RT_BK;
    int s = sm_count() / tiles;
    if (s > RT_MAX_SPLIT) s = RT_MAX_SPLIT;
    if (s > num_kb) s = num_kb;
    return s < 1 ? 1 : s;
}

// Accumulators of a block: with the splits of K, RT_CHAINS chains of an output's products; but four where K is long and not split (matrices of more than 8,192 columns,
// which tiles of 128 rows with one accumulator have otherwise): eight of 64 columns are all of a multiprocessor's tensor memory, and the next launch's blocks
// cannot begin beside them (a layer of 1.7B with 64 decoding requests 224.8 us with four for gate and up, 233.5 with eight).
static int rt_accs(int splits, int K) {
    const int a = (RT_CHAINS + splits - 1) / splits;
    return K >= 2048 && a > 4 ? 4 : a;
}

template <int NB, int EPI>
static int rt_launch(const CUtensorMap& mx, const CUtensorMap& mw, RtArgs p, int* error, cudaStream_t stream) {
    const WaitCtl wc = wait_ctl(error, WAIT_FAMILY_LINEAR);
    const size_t smem = (size_t)RT_STAGES * (RT_BM + NB) * RT_BK * 2 + 1024 + 128;
    auto kern = linear_rows_tcgen05_kernel<NB, EPI>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
    const int per_tile = EPI == RT_SWIGLU ? RT_BM / 2 : RT_BM, cols = EPI == RT_SWIGLU ? p.N / 2 : p.N;
    const int tiles = (cols + per_tile - 1) / per_tile;
    p.splits = rt_splits(tiles, p.K);
    p.accs = rt_accs(p.splits, p.K);
    return launch_dependent_cluster(kern, dim3(tiles * p.splits), dim3(RT_THREADS), p.splits, smem, stream, mx, mw, p, wc);
}

}  // namespace vk

using namespace vk;

// x [M, K] bfloat16 with row stride ldx, M <= 64; w [N, K] bfloat16; epi 0 out bfloat16 (act: activate_dense's number), 1 float32, 2 float32 +=,
// 3 [M, N / 2] bfloat16 = f(first half) * second half (act 0 silu, else activate_rt's number), 4 rotated q, with k and v into the cache (hd 64 or 128).
// K and ldx multiples of 8, N of 4 (3: of 8), x, w, out (and cache, cos, sin) 16-byte aligned.  error: a word the kernel sets if a bounded wait ran out.
VK_API int vk_linear_rows_tcgen05(const void* x, const void* w, void* out, int M, int N, int K, int ldx, int epi, int act, const int32_t* positions,
                                  const float* cos_t, const float* sin_t, const int32_t* slot, void* cache, int nh, int nkv, int hd, int page_size, int* error,
                                  cudaStream_t stream) {
    if (M <= 0 || N <= 0) return VK_OK;
    if (M > 64) return VK_TOO_LARGE;
    if (K <= 0 || ldx < K || K % 8 != 0 || ldx % 8 != 0 || N % 4 != 0 || epi < 0 || epi > 4 || !error || act < 0 || act > 4 ||
        (act && epi != RT_SAME && (epi != RT_SWIGLU || act > 3)))
        return VK_BAD_SHAPE;
    if (((uintptr_t)x % 16) || ((uintptr_t)w % 16) || ((uintptr_t)out % 16)) return VK_BAD_ALIGNMENT;
    if (epi == RT_SWIGLU && N % 8 != 0) return VK_BAD_SHAPE;
    if (epi == RT_ROPE) {
        if (nh <= 0 || nkv <= 0 || (hd != 64 && hd != 128) || page_size <= 0 || N != (nh + 2 * nkv) * hd || !positions || !cos_t || !sin_t || !slot || !cache)
            return VK_BAD_SHAPE;
        if (((uintptr_t)cache % 16) || ((uintptr_t)cos_t % 16) || ((uintptr_t)sin_t % 16)) return VK_BAD_ALIGNMENT;
    }
    const int nb = M <= 16 ? 16 : M <= 32 ? 32 : 64;
    CUtensorMap mx, mw;
    if (!rt_make_map(&mx, x, M, K, ldx, nb) || !rt_make_map(&mw, w, N, K, K, epi == RT_SWIGLU ? RT_BM / 2 : RT_BM)) return VK_BAD_SHAPE;
    RtArgs p{out, M, N, K, 1, 1, act, positions, cos_t, sin_t, slot, (__nv_bfloat16*)cache, nh, nkv, hd, page_size};
#define GO(NB)                                                              \
    switch (epi) {                                                          \
        case RT_SAME: return rt_launch<NB, RT_SAME>(mx, mw, p, error, stream);     \
        case RT_F32: return rt_launch<NB, RT_F32>(mx, mw, p, error, stream);       \
        case RT_ACC: return rt_launch<NB, RT_ACC>(mx, mw, p, error, stream);       \
        case RT_SWIGLU: return rt_launch<NB, RT_SWIGLU>(mx, mw, p, error, stream); \
        default: return rt_launch<NB, RT_ROPE>(mx, mw, p, error, stream);          \
    }
    if (nb == 16) GO(16)
    if (nb == 32) GO(32)
    GO(64)
#undef GO
}
