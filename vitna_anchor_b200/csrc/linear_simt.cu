// Matrix products on CUDA cores: out[M, N] = x[M, K] * W[N, K]^T.
//
// These are the engine's true-32-bit products and the bfloat16 path's
// products at sizes its tensor-core kernels do not take.  Inputs are widened
// exactly, every product and sum is float32 (fmaf), and the order in which an
// output element's K terms are added depends only on K and on which of the two
// kernels runs, never on M, on the position of the row in the batch, or on
// the grid: a row's result does not change with what else is in the batch.
//
// Output modes: 0 = store in the input type, 1 = store float32,
//               2 = add into a float32 output (the residual sum).
#include "common.cuh"

namespace vk {

enum { OUT_SAME = 0, OUT_F32 = 1, OUT_ACC_F32 = 2 };

template <typename T, int MODE>
__device__ __forceinline__ void store_out(void* out, size_t idx, float v) {
    if (MODE == OUT_SAME) ((T*)out)[idx] = from_f32<T>(v);
    else if (MODE == OUT_F32) ((float*)out)[idx] = v;
    else ((float*)out)[idx] += v;
}

// 64x64 output tile, K in slabs of 16, 256 threads, 4x4 outputs per thread.
// (The reference's prompt GEMM has the same tile shape, engine/src/model_cuda.cu:2579-2641.)
constexpr int TM = 64, TN = 64, TK = 16;

template <typename T, int MODE>
__global__ void __launch_bounds__(256) gemm_tile_kernel(const T* __restrict__ x, const T* __restrict__ w, void* __restrict__ out,
                                                        int M, int N, int K, int ldx) {
    __shared__ float xs[TK][TM + 4];
    __shared__ float ws[TK][TN + 4];
    const int m0 = blockIdx.y * TM, n0 = blockIdx.x * TN;
    const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
    float acc[4][4] = {};
    for (int k0 = 0; k0 < K; k0 += TK) {
        // 64 rows x 16 k of each operand: 1024 elements, 4 per thread
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int e = threadIdx.x + i * 256;
            const int r = e / TK, kk = e % TK;
            const int gm = m0 + r, gn = n0 + r, gk = k0 + kk;
            xs[kk][r] = (gm < M && gk < K) ? to_f32<T>(x[(size_t)gm * ldx + gk]) : 0.0f;
            ws[kk][r] = (gn < N && gk < K) ? to_f32<T>(w[(size_t)gn * K + gk]) : 0.0f;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < TK; kk++) {
            float a[4], b[4];
#pragma unroll
            for (int i = 0; i < 4; i++) a[i] = xs[kk][ty * 4 + i];
#pragma unroll
            for (int j = 0; j < 4; j++) b[j] = ws[kk][tx * 4 + j];
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int gm = m0 + ty * 4 + i;
        if (gm >= M) continue;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int gn = n0 + tx * 4 + j;
            if (gn < N) store_out<T, MODE>(out, (size_t)gm * N + gn, acc[i][j]);
        }
    }
}

// The float32 product of whole 16-byte pieces: BM x BN outputs a block, RM x RN a thread (rows and columns a thread grid apart, so that
// neighbouring lanes read neighbouring rows), K in slabs of 32 that cp.async brings GT_STAGES - 1 slabs ahead.  Operands stay as they lie in
// memory (k along a row, rows 36 floats apart: eight lanes' 16-byte loads meet no bank twice).  An output is ONE fmaf chain over k in increasing
// order whatever the tile, so every tile, and the kernel above, give the same bits and the tile may follow the launch's size.
constexpr int GT_K = 32, GT_LD = GT_K + 4, GT_STAGES = 4;

template <int MODE, int BM, int BN, int RM, int RN>
__global__ void __launch_bounds__((BM / RM) * (BN / RN)) gemm_async_kernel(const float* __restrict__ x, const float* __restrict__ w, void* __restrict__ out,
                                                                           int M, int N, int K, int ldx) {
    constexpr int TX = BN / RN, TY = BM / RM, NT = TX * TY, STAGE = (BM + BN) * GT_LD, PIECES = (BM + BN) * (GT_K / 4);
    extern __shared__ __align__(16) float gt_smem[];
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN, tid = threadIdx.x;
    const int tx = tid % TX, ty = tid / TX;
    float acc[RM][RN] = {};
    const int slabs = (K + GT_K - 1) / GT_K;
    auto issue = [&](int s) {
        if (s < slabs) {
            float* st = gt_smem + (s % GT_STAGES) * STAGE;
#pragma unroll
            for (int e = tid; e < PIECES; e += NT) {
                const int r = e / (GT_K / 4), k = s * GT_K + 4 * (e % (GT_K / 4));
                const bool isx = r < BM;
                const int g = isx ? m0 + r : n0 + r - BM;
                const bool there = k < K && g < (isx ? M : N);
                copy16_or_zero(st + r * GT_LD + 4 * (e % (GT_K / 4)), there ? (isx ? x + (size_t)g * ldx + k : w + (size_t)g * K + k) : x, there);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
#pragma unroll
    for (int s = 0; s < GT_STAGES - 1; s++) issue(s);
    for (int s = 0; s < slabs; s++) {
        asm volatile("cp.async.wait_group %0;" ::"n"(GT_STAGES - 2) : "memory");
        __syncthreads();                                    // slab s is there for everybody, and everybody has left slab s - 1
        issue(s + GT_STAGES - 1);
        const float* xs = gt_smem + (s % GT_STAGES) * STAGE + ty * GT_LD;
        const float* ws = gt_smem + (s % GT_STAGES) * STAGE + (BM + tx) * GT_LD;
#pragma unroll
        for (int k = 0; k < GT_K; k += 4) {
            float4 a[RM], b[RN];
#pragma unroll
            for (int i = 0; i < RM; i++) a[i] = *reinterpret_cast<const float4*>(xs + i * TY * GT_LD + k);
#pragma unroll
            for (int j = 0; j < RN; j++) b[j] = *reinterpret_cast<const float4*>(ws + j * TX * GT_LD + k);
#pragma unroll
            for (int i = 0; i < RM; i++)
#pragma unroll
                for (int j = 0; j < RN; j++) {
                    acc[i][j] = fmaf(a[i].x, b[j].x, acc[i][j]);
                    acc[i][j] = fmaf(a[i].y, b[j].y, acc[i][j]);
                    acc[i][j] = fmaf(a[i].z, b[j].z, acc[i][j]);
                    acc[i][j] = fmaf(a[i].w, b[j].w, acc[i][j]);
                }
        }
    }
#pragma unroll
    for (int i = 0; i < RM; i++) {
        const int gm = m0 + ty + i * TY;
        if (gm >= M) continue;
#pragma unroll
        for (int j = 0; j < RN; j++) {
            const int gn = n0 + tx + j * TX;
            if (gn < N) store_out<float, MODE>(out, (size_t)gm * N + gn, acc[i][j]);
        }
    }
}

template <int MODE, int BM, int BN, int RM, int RN>
static int launch_async(const float* x, const float* w, void* out, int M, int N, int K, int ldx, cudaStream_t stream) {
    auto kern = gemm_async_kernel<MODE, BM, BN, RM, RN>;
    constexpr int smem = GT_STAGES * (BM + BN) * GT_LD * (int)sizeof(float);
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return (int)e;
    dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
    if (grid.y > 65535) return VK_TOO_LARGE;
    kern<<<grid, (BM / RM) * (BN / RN), smem, stream>>>(x, w, out, M, N, K, ldx);
    return launch_status();
}

// The tile by the number of blocks it would make (all give the same bits).  Measured, us a product (128 x 128 / 64 x 64 / 32 x 32 / 16 x 16 tiles; the kernel
// above takes 31 to 80 for the first three): 512 x 3072 x 576: 66 / 53 / 64 / 115;  512 x 576 x 576: 64 / 25 / 16.5 / 27;  512 x 576 x 1536: 162 / 58 / 37 / 63;
// 2048 x 576 x 576 (288 tiles of 64): 66 / 39 / 47 / 88;  64 x 576 x 1536 (36 tiles of 32): 158 / 58 / 27 / 14.5;  16 x 576 x 576: 62 / 23 / 12 / 8.
// 2048 x 6144 x 2048: 1270 / 1183 / 1575 (61 % of the multiply-add rate in tiles of 64): more blocks than a multiprocessor holds gain nothing more.
template <int MODE>
static int launch_async_tile(const float* x, const float* w, void* out, int M, int N, int K, int ldx, cudaStream_t stream) {
    auto tiles = [&](int bm, int bn) { return (long long)((M + bm - 1) / bm) * ((N + bn - 1) / bn); };
    if (M > 16 && tiles(64, 64) >= 200) return launch_async<MODE, 64, 64, 8, 4>(x, w, out, M, N, K, ldx, stream);
    if (M > 16 && tiles(32, 32) >= 100) return launch_async<MODE, 32, 32, 4, 2>(x, w, out, M, N, K, ldx, stream);
    if (tiles(16, 32) >= 148) return launch_async<MODE, 16, 32, 2, 2>(x, w, out, M, N, K, ldx, stream);
    return launch_async<MODE, 16, 16, 2, 1>(x, w, out, M, N, K, ldx, stream);
}

// Few rows (M <= ROWS): a warp per output column streams that column's weight
// row once, 16 bytes per lane per load, and keeps one sum per input row.
// Each lane's partial sum runs over k = lane*VEC + 32*VEC*i (+0..VEC-1) in
// increasing order; the 32 partial sums meet in a fixed shuffle tree.
template <typename T, int MODE, int ROWS, bool VECTOR>
__global__ void __launch_bounds__(256) gemv_rows_kernel(const T* __restrict__ x, const T* __restrict__ w, void* __restrict__ out,
                                                        int M, int N, int K, int ldx) {
    constexpr int V = Vec16<T>::N;
    const int lane = threadIdx.x & 31;
    const int warps_per_block = blockDim.x >> 5;
    for (int n = blockIdx.x * warps_per_block + (threadIdx.x >> 5); n < N; n += gridDim.x * warps_per_block) {
        const T* wr = w + (size_t)n * K;
        float acc[ROWS];
#pragma unroll
        for (int m = 0; m < ROWS; m++) acc[m] = 0.0f;
        if (VECTOR) {
            for (int k = lane * V; k < K; k += 32 * V) {
                float wf[V];
                load16<T>(wr + k, wf);
#pragma unroll
                for (int m = 0; m < ROWS; m++) {
                    if (m < M) {
                        float xf[V];
                        load16<T>(x + (size_t)m * ldx + k, xf);
#pragma unroll
                        for (int i = 0; i < V; i++) acc[m] = fmaf(xf[i], wf[i], acc[m]);
                    }
                }
            }
        } else {
            for (int k = lane; k < K; k += 32) {
                const float wv = to_f32<T>(wr[k]);
#pragma unroll
                for (int m = 0; m < ROWS; m++)
                    if (m < M) acc[m] = fmaf(to_f32<T>(x[(size_t)m * ldx + k]), wv, acc[m]);
            }
        }
#pragma unroll
        for (int m = 0; m < ROWS; m++) {
            const float s = warp_sum(acc[m]);
            if (lane == 0 && m < M) store_out<T, MODE>(out, (size_t)m * N + n, s);
        }
    }
}

template <typename T, int MODE>
static int launch_linear(const T* x, const T* w, void* out, int M, int N, int K, int ldx, int few_rows, cudaStream_t stream) {
    if (M <= few_rows) {
        constexpr int V = Vec16<T>::N;
        const bool vec = (K % V == 0) && (ldx % V == 0) && ((uintptr_t)x % 16 == 0) && ((uintptr_t)w % 16 == 0);
        const int blocks = (N + 7) / 8 < 148 * 8 ? (N + 7) / 8 : 148 * 8;
        if (M <= 4) {
            if (vec) gemv_rows_kernel<T, MODE, 4, true><<<blocks, 256, 0, stream>>>(x, w, out, M, N, K, ldx);
            else gemv_rows_kernel<T, MODE, 4, false><<<blocks, 256, 0, stream>>>(x, w, out, M, N, K, ldx);
        } else {
            if (vec) gemv_rows_kernel<T, MODE, 8, true><<<blocks, 256, 0, stream>>>(x, w, out, M, N, K, ldx);
            else gemv_rows_kernel<T, MODE, 8, false><<<blocks, 256, 0, stream>>>(x, w, out, M, N, K, ldx);
        }
    } else {
        if (sizeof(T) == 4 && K % 4 == 0 && ldx % 4 == 0 && (uintptr_t)x % 16 == 0 && (uintptr_t)w % 16 == 0)
            return launch_async_tile<MODE>((const float*)x, (const float*)w, out, M, N, K, ldx, stream);
        dim3 grid((N + TN - 1) / TN, (M + TM - 1) / TM);
        if (grid.y > 65535) return VK_TOO_LARGE;
        gemm_tile_kernel<T, MODE><<<grid, 256, 0, stream>>>(x, w, out, M, N, K, ldx);
    }
    return launch_status();
}

}  // namespace vk

using namespace vk;

// x [M, K] with row stride ldx, w [N, K], out [M, N]; dtype 0 = float32, 1 = bfloat16.
// few_rows: batches of at most this many rows (<= 8) take the column-per-warp kernel; 0 sends
// everything through the tile kernel.
VK_API int vk_linear_simt(const void* x, const void* w, void* out, int M, int N, int K, int ldx, int dtype, int mode,
                          int few_rows, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return VK_OK;
    if (K <= 0 || ldx < K || mode < 0 || mode > 2 || few_rows < 0 || few_rows > 8) return VK_BAD_SHAPE;
#define GO(T, MODE) return launch_linear<T, MODE>((const T*)x, (const T*)w, out, M, N, K, ldx, few_rows, stream)
    if (dtype == 0) {
        if (mode == 0) GO(float, OUT_SAME);
        if (mode == 1) GO(float, OUT_F32);
        GO(float, OUT_ACC_F32);
    } else {
        if (mode == 0) GO(__nv_bfloat16, OUT_SAME);
        if (mode == 1) GO(__nv_bfloat16, OUT_F32);
        GO(__nv_bfloat16, OUT_ACC_F32);
    }
#undef GO
}
