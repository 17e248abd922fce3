// The gated delta rule over a prompt's portion in chunks of 64 tokens: what can be worked out without the state is worked out for all
// chunks at once, only a short pass per chunk runs in order, and the outputs follow for all chunks at once again.
//
// For a chunk with the state S before it, L_t = ln(g_1 .. g_t) (the decays up to t, inside the chunk):
//     A[t][i] = beta_t e^(L_t - L_i) (k_t . k_i)   (i < t)          the updates u_t solve  (I + A) U = diag(beta) V - diag(beta e^L) K S
//     so with  U' = (I + A)^-1 diag(beta) V   and   W = (I + A)^-1 diag(beta e^L) K :     U = U' - W S
//     P[t][i] = e^(L_t - L_i) (q_t . k_i)          (i <= t)         O = diag(e^L) Q S + P U
//     S <- e^(L_64) S + (diag(e^(L_64 - L)) K)^T U
//
//  delta_chunk_prepare   a block a chunk and head, all chunks side by side: A, P, T = (I + A)^-1 (the four 16 x 16 blocks on the diagonal by substitution, the
//                        others from them), W and U' as products with T, and the scaled Q and K.
//  delta_chunk_scan      a block a request, head and 8 or 16 columns of the state walks the request's chunks in order: two small products a chunk, the state's
//                        slice in registers and, as an operand, in shared memory; leaves U and the state before every chunk.  A chunk's two operands are one bulk
//                        copy into a ring of three stages, two chunks ahead (asked for piece by piece with cp.async they cost the block 890 of a chunk's 2,900 cycles);
//                        every wait for one is bounded.
//  delta_chunk_out       a block a chunk, head and 64 or 128 columns, all chunks side by side: O, and where a head's values are in one block and the decay is one
//                        a head, its norm and gate.
//
// The decays, beta, the unit vectors and the state are 32-bit quantities of this mixer: products take them as two tf32 parts (tf32.cuh), every other operation is
// float32.  The results equal the token-by-token recurrence up to the order of sums.  A chunk that reaches past its segment's end is filled
// with tokens that do nothing.  Inputs are the rows `delta_prepare` writes (q | k | v | log decay | beta).
//
// The form with a decay per head AND key channel (template flag CH; inputs are the rows `cdelta_prepare` writes, q | k | v | log decay [H][dk] | beta [H] | ..): L_t is a
// vector over the key channels, and the decays no longer leave the sums over dk: A[t][i] = beta_t sum_d k_t[d] k_i[d] e^(L_t[d] - L_i[d]), P likewise.  Pairs inside 16
// tokens are taken one by one; between different sixteens the exponential is split into what the row's sixteen leaves up to its token, what whole
// sixteens between leave, and what the column's sixteen leaves behind its token, each at most 1.  The state's rows decay by the vector e^(L_64[d]).
//
// What bounds it: the scan is a chain of 2 products, 2 barriers a chunk; the other two kernels the tensor cores' rate for three tf32 products.
#include "chunks.cuh"
#include "common.cuh"
#include "tcgen05_common.cuh"
#include "tf32.cuh"

namespace vk {

constexpr int DC_C = 64;                    // tokens of a chunk
constexpr int DC_MAX_TAPS = 16;
constexpr int DC_LDA = DC_C + 8;            // a padded row of a 64 x 64 matrix

// Floats of scratch for one (chunk, head):  W [64][LDQ] | Kg [64][LDQ] (rows as they lie in shared memory, dk of DKP = 64 or 128 columns used, LDQ = DKP + 8) |
// Qg [64][dk] | P [64][64] | U', then U [64][dv] | S before the chunk [dv][dk] | e^(L_64) (one, or one a channel), padded to a multiple of four.
__host__ __device__ __forceinline__ int dc_ldq(int dk) { return dk <= 64 ? 72 : 136; }
__host__ __device__ __forceinline__ size_t dc_q_off(int dk) { return (size_t)2 * DC_C * dc_ldq(dk); }
__host__ __device__ __forceinline__ size_t dc_p_off(int dk) { return dc_q_off(dk) + (size_t)DC_C * dk; }
__host__ __device__ __forceinline__ size_t dc_u_off(int dk) { return dc_p_off(dk) + DC_C * DC_C; }
__host__ __device__ __forceinline__ size_t dc_s_off(int dk, int dv) { return dc_u_off(dk) + (size_t)DC_C * dv; }
__host__ __device__ __forceinline__ size_t dc_e_off(int dk, int dv) { return dc_s_off(dk, dv) + (size_t)dk * dv; }
__host__ __device__ __forceinline__ size_t dc_stride(int dk, int dv, bool ch) { return dc_e_off(dk, dv) + (ch ? (dk + 3) / 4 * 4 : 4); }

struct DcArgs {
    const float* prep;
    int P;                                  // floats of a row of prep
    const int32_t* seg_starts;
    const int32_t* seg_slots;
    int segments, from;                     // segments of up to `from` tokens are left alone
    float* scratch;
    int G, H, dk, dv;
};

__host__ __device__ __forceinline__ int dc_ldv(int dv) { return (dv + 15) / 16 * 16 + 4; }

template <int DKP, bool CH>
__host__ __device__ constexpr int dc_prepare_floats_fixed() { return DC_C * (DKP + 8) * (CH ? 3 : 2) + 2 * DC_C * DC_LDA + (CH ? 4 * DKP : 0); }

// grid (chunks, H)
template <int DKP, bool CH>
__global__ void __launch_bounds__(256) delta_chunk_prepare_kernel(const DcArgs p) {
    constexpr int LDQ = DKP + 8;
    extern __shared__ __align__(16) float dp_smem[];
    __shared__ double L[CH ? 1 : DC_C];             // (float64: what counts are differences of neighbours, and behind a strongly decaying token the sum is in the thousands)
    __shared__ float beta[DC_C], factor[DC_C];
    __shared__ int find[4];
    const int LDV = dc_ldv(p.dv);
    float* sq = dp_smem;                            // [64][LDQ]
    float* sk = sq + DC_C * LDQ;                    // [64][LDQ]
    float* sA = sk + DC_C * LDQ;                    // [64][DC_LDA]
    float* sT = sA + DC_C * DC_LDA;                 // [64][DC_LDA]
    float* sl = sT + DC_C * DC_LDA;                 // CH: [64][LDQ] the decays' logarithms, then k times what its sixteen leaves behind it
    float* vec = sl + (CH ? DC_C * LDQ : 0);        // CH: [4][DKP] what whole sixteens leave
    float* sv = vec + (CH ? 4 * DKP : 0);           // [64][LDV]
    const Chunk ch = find_chunk<DC_C>(blockIdx.x, p.seg_starts, p.segments, find, p.from);
    if (ch.seg < 0 || p.seg_slots[ch.seg] < 0) return;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t4 = lane & 3, wm = warp & 1, wn = warp >> 1;
    const int h = blockIdx.y, dk = p.dk, dv = p.dv, rows = ch.rows, kh = h / (p.H / p.G), Cq = 2 * p.G * dk + p.H * dv;
    const float* row0 = p.prep + (size_t)ch.first * p.P;
    for (int e = tid; e < DC_C * (DKP / 4); e += 256) {
        const int r = e / (DKP / 4), d = 4 * (e % (DKP / 4));
        const bool on = r < rows && d < dk;
        const float* row = row0 + (size_t)(on ? r : 0) * p.P + (on ? d : 0);
        copy16_or_zero(sq + r * LDQ + d, row + kh * dk, on);
        copy16_or_zero(sk + r * LDQ + d, row + (p.G + kh) * dk, on);
        if (CH) copy16_or_zero(sl + r * LDQ + d, row + Cq + h * dk, on);
    }
    const int vp = (LDV - 4) / 4;
    for (int e = tid; e < DC_C * vp; e += 256) {
        const int r = e / vp, c = 4 * (e - r * vp);
        const bool on = r < rows && c < dv;
        copy16_or_zero(sv + r * LDV + c, row0 + (size_t)(on ? r : 0) * p.P + 2 * p.G * dk + h * dv + (on ? c : 0), on);
    }
    tf_commit();
    if (tid < 32) {                                 // beta, and the sums of the decays' logarithms
        double carry = 0.0;
#pragma unroll
        for (int u = 0; u < 2; u++) {
            const int r = 32 * u + tid;
            const float* row = row0 + (size_t)(r < rows ? r : 0) * p.P + Cq;
            beta[r] = r < rows ? row[(CH ? p.H * dk : p.H) + h] : 0.0f;
            if (!CH) {
                // (a token that leaves less than e^-10000 leaves nothing either way, and one that leaves e^-inf must not make the sums infinite)
                const float l = r < rows ? row[h] : 0.0f;
                double s = l < -1e4f ? -1e4 : (double)l;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const double v = __shfl_up_sync(0xffffffffu, s, o);
                    if (tid >= o) s += v;
                }
                L[r] = carry + s;
                carry += __shfl_sync(0xffffffffu, s, 31);
            }
        }
    }
    tf_wait<0>();
    __syncthreads();

    float* out = p.scratch + ((size_t)blockIdx.x * p.H + h) * dc_stride(dk, dv, CH);
    float* W_g = out;
    float* K_g = W_g + DC_C * LDQ;
    float* Q_g = out + dc_q_off(dk);
    float* P_g = out + dc_p_off(dk);
    float* U_g = out + dc_u_off(dk);
    float* E_g = out + dc_e_off(dk, dv);

    // k k^T and q k^T: a warp has the 16 x 16 pieces (rows 32 wm + 16 m .., columns 16 wn ..), m = 0, 1
    float kk[2][2][4], qk[2][2][4];
#pragma unroll
    for (int m = 0; m < 2; m++)
#pragma unroll
        for (int n = 0; n < 2; n++)
#pragma unroll
            for (int e = 0; e < 4; e++) kk[m][n][e] = qk[m][n][e] = 0.0f;
    if (CH) {
        // pairs inside sixteen tokens: four threads a row, a quarter of the channels each, walk back from the row's token with the sum of the logarithms so far
        const int r = tid >> 2, p0 = r & ~15;
        float pk[16], pq[16];
#pragma unroll
        for (int j = 0; j < 16; j++) pk[j] = pq[j] = 0.0f;
        for (int d = tid & 3; d < DKP; d += 4) {
            float sum = 0.0f;
            const float qv = sq[r * LDQ + d], kv = sk[r * LDQ + d];
#pragma unroll
            for (int j = 15; j >= 0; j--)
                if (p0 + j <= r) {
                    const float x = sk[(p0 + j) * LDQ + d] * expf(sum);
                    pk[j] = fmaf(kv, x, pk[j]);
                    pq[j] = fmaf(qv, x, pq[j]);
                    sum += sl[(p0 + j) * LDQ + d];
                }
        }
        float* tk = sA;                             // (sA and sT are free until the pieces are collected)
        float* tq = sT;
#pragma unroll
        for (int j = 0; j < 16; j++) {
            pk[j] += __shfl_xor_sync(0xffffffffu, pk[j], 1);
            pk[j] += __shfl_xor_sync(0xffffffffu, pk[j], 2);
            pq[j] += __shfl_xor_sync(0xffffffffu, pq[j], 1);
            pq[j] += __shfl_xor_sync(0xffffffffu, pq[j], 2);
            if ((tid & 3) == (j & 3)) { tk[r * 17 + j] = pk[j]; tq[r * 17 + j] = pq[j]; }
        }
        __syncthreads();
#pragma unroll
        for (int m = 0; m < 2; m++)
            if (2 * wm + m == wn) {
#pragma unroll
                for (int n = 0; n < 2; n++)
#pragma unroll
                    for (int e = 0; e < 4; e++) {
                        const int at = (16 * wn + g + (e >> 1) * 8) * 17 + n * 8 + 2 * t4 + (e & 1);
                        kk[m][n][e] = tk[at];
                        qk[m][n][e] = tq[at];
                    }
            }
        for (int e = tid; e < 4 * DKP; e += 256) {  // a channel of a sixteen a thread
            const int s = e / DKP, d = e % DKP;
            float l[16], k[16], sum = 0.0f;
#pragma unroll
            for (int j = 0; j < 16; j++) { l[j] = sl[(16 * s + j) * LDQ + d]; k[j] = sk[(16 * s + j) * LDQ + d]; }
#pragma unroll
            for (int j = 0; j < 16; j++) {
                sum += l[j];
                const float f = expf(sum);
                sq[(16 * s + j) * LDQ + d] *= f;
                sk[(16 * s + j) * LDQ + d] = k[j] * f;
            }
            vec[e] = expf(sum);
            sum = 0.0f;
#pragma unroll
            for (int j = 15; j >= 0; j--) {
                sl[(16 * s + j) * LDQ + d] = k[j] * expf(sum);
                sum += l[j];
            }
        }
        __syncthreads();
    }
    {
        const float* right = CH ? sl : sk;
#pragma unroll
        for (int m = 0; m < 2; m++) {
            const int I = 2 * wm + m;
            if (CH ? wn >= I : wn > I) continue;
#pragma unroll 2
            for (int ks = 0; ks < DKP / 8; ks++) {
                const int d = ks * 8 + 2 * t4;
                float2 x[4] = {*reinterpret_cast<const float2*>(sk + (16 * I + g) * LDQ + d), *reinterpret_cast<const float2*>(sk + (16 * I + g + 8) * LDQ + d),
                               *reinterpret_cast<const float2*>(sq + (16 * I + g) * LDQ + d), *reinterpret_cast<const float2*>(sq + (16 * I + g + 8) * LDQ + d)};
                if (CH) {
                    float f0 = 1.0f, f1 = 1.0f;
                    for (int u = wn + 1; u < I; u++) { f0 *= vec[u * DKP + d]; f1 *= vec[u * DKP + d + 1]; }
#pragma unroll
                    for (int i = 0; i < 4; i++) { x[i].x *= f0; x[i].y *= f1; }
                }
                const Tf a[2][4] = {{tf_split(x[0].x), tf_split(x[1].x), tf_split(x[0].y), tf_split(x[1].y)},
                                    {tf_split(x[2].x), tf_split(x[3].x), tf_split(x[2].y), tf_split(x[3].y)}};
                Tf b[2][2];
#pragma unroll
                for (int n = 0; n < 2; n++) {
                    const float2 kb = *reinterpret_cast<const float2*>(right + (16 * wn + n * 8 + g) * LDQ + d);
                    b[n][0] = tf_split(kb.x);
                    b[n][1] = tf_split(kb.y);
                }
                float* const d_[2][2] = {{kk[m][0], kk[m][1]}, {qk[m][0], qk[m][1]}};
                tf_mma3(d_, a, b);
            }
        }
    }
    if (CH) __syncthreads();                        // (the pieces that lay in sA and sT have been collected)
#pragma unroll
    for (int m = 0; m < 2; m++)
#pragma unroll
        for (int n = 0; n < 2; n++)
#pragma unroll
            for (int u = 0; u < 2; u++) {
                const int r = 32 * wm + 16 * m + g + 8 * u, i = 16 * wn + n * 8 + 2 * t4;
                float a[2], w[2];
#pragma unroll
                for (int e = 0; e < 2; e++) {
                    const float ratio = i + e <= r ? (CH ? 1.0f : expf((float)(L[r] - L[i + e]))) : 0.0f;
                    a[e] = i + e < r ? beta[r] * ratio * kk[m][n][2 * u + e] : 0.0f;
                    w[e] = i + e <= r ? ratio * qk[m][n][2 * u + e] : 0.0f;
                }
                *reinterpret_cast<float2*>(sA + r * DC_LDA + i) = make_float2(a[0], a[1]);
                *reinterpret_cast<float2*>(P_g + r * DC_C + i) = make_float2(w[0], w[1]);
            }
    // the scaled q and k; with a decay a channel k times e^L takes k's place
    for (int e = tid; e < DC_C * (DKP / 4); e += 256) {
        const int r = e / (DKP / 4), d = 4 * (e % (DKP / 4));      // (q and k are zero from dk on, and the scan reads Kg to DKP)
        float4 kq, kb;
        if (CH) {
            kq = *reinterpret_cast<const float4*>(sq + r * LDQ + d);
            kb = *reinterpret_cast<const float4*>(sl + r * LDQ + d);
            float4 kw = *reinterpret_cast<const float4*>(sk + r * LDQ + d);
            for (int u = 0; u < r / 16; u++) {
                const float4 f = *reinterpret_cast<const float4*>(vec + u * DKP + d);
                kq.x *= f.x; kq.y *= f.y; kq.z *= f.z; kq.w *= f.w;
                kw.x *= f.x; kw.y *= f.y; kw.z *= f.z; kw.w *= f.w;
            }
            for (int u = r / 16 + 1; u < 4; u++) {
                const float4 f = *reinterpret_cast<const float4*>(vec + u * DKP + d);
                kb.x *= f.x; kb.y *= f.y; kb.z *= f.z; kb.w *= f.w;
            }
            *reinterpret_cast<float4*>(sk + r * LDQ + d) = kw;
        } else {
            const float fq = expf((float)L[r]), fk = expf((float)(L[DC_C - 1] - L[r]));
            kq = *reinterpret_cast<const float4*>(sq + r * LDQ + d);
            kb = *reinterpret_cast<const float4*>(sk + r * LDQ + d);
            kq.x *= fq; kq.y *= fq; kq.z *= fq; kq.w *= fq;
            kb.x *= fk; kb.y *= fk; kb.z *= fk; kb.w *= fk;
        }
        if (d < dk) *reinterpret_cast<float4*>(Q_g + r * dk + d) = kq;
        *reinterpret_cast<float4*>(K_g + r * LDQ + d) = kb;
    }
    if (CH) {
        for (int d = tid; d < dk; d += 256) E_g[d] = (vec[d] * vec[DKP + d]) * (vec[2 * DKP + d] * vec[3 * DKP + d]);
    } else if (tid == 0) E_g[0] = expf((float)L[DC_C - 1]);
    __syncthreads();

    // T = (I + A)^-1.  The blocks on the diagonal, a column a thread ..
    if (tid < DC_C) {
        const int b = tid >> 4, j = tid & 15;
        const float* a = sA + 16 * b * DC_LDA + 16 * b;
        float x[16];
#pragma unroll
        for (int r = 0; r < 16; r++) {
            float s = 0.0f;
#pragma unroll
            for (int i = 0; i < r; i++) s = fmaf(a[r * DC_LDA + i], x[i], s);
            x[r] = r < j ? 0.0f : r == j ? 1.0f : -s;
            sT[(16 * b + r) * DC_LDA + 16 * b + j] = x[r];
        }
    }
    __syncthreads();
    // .. and T_ij = -T_ii sum_k A_ik T_kj below it, one step from the diagonal after the other (the sum waits in the block mirrored above the diagonal)
    {
        const int r = tid >> 4, c = tid & 15;
        for (int step = 1; step < 4; step++) {
            for (int j = 0; j + step < 4; j++) {
                const int i = j + step;
                float s0 = 0.0f, s1 = 0.0f;
                for (int k = 16 * j; k < 16 * i; k += 2) {
                    s0 = fmaf(sA[(16 * i + r) * DC_LDA + k], sT[k * DC_LDA + 16 * j + c], s0);
                    s1 = fmaf(sA[(16 * i + r) * DC_LDA + k + 1], sT[(k + 1) * DC_LDA + 16 * j + c], s1);
                }
                sT[(16 * j + r) * DC_LDA + 16 * i + c] = s0 + s1;
            }
            __syncthreads();
            for (int j = 0; j + step < 4; j++) {
                const int i = j + step;
                float s = 0.0f;
#pragma unroll
                for (int u = 0; u < 16; u++)
                    if (u <= r) s = fmaf(sT[(16 * i + r) * DC_LDA + 16 * i + u], sT[(16 * j + u) * DC_LDA + 16 * i + c], s);
                sT[(16 * i + r) * DC_LDA + 16 * j + c] = -s;
            }
            __syncthreads();
        }
    }
    // W = T diag(beta e^L) K and U' = T diag(beta) V, eight columns a warp at a time
    if (tid < DC_C) factor[tid] = CH ? beta[tid] : beta[tid] * expf((float)L[tid]);      // of k's rows
    __syncthreads();
    constexpr int nw = DKP / 8;
    const int nv = (dv + 7) / 8;
    for (int n = warp; n < nw + nv; n += 8) {
        const bool is_w = n < nw;
        const int c0 = (is_w ? n : n - nw) * 8, ld = is_w ? LDQ : LDV;
        const float* src = (is_w ? sk : sv) + c0 + g;
        const float* fac = is_w ? factor : beta;
        float acc[4][4];
#pragma unroll
        for (int m = 0; m < 4; m++)
#pragma unroll
            for (int e = 0; e < 4; e++) acc[m][e] = 0.0f;
#pragma unroll
        for (int ks = 0; ks < 8; ks++) {
            const int k = ks * 8 + 2 * t4;
            const Tf b[2] = {tf_split(fac[k] * src[k * ld]), tf_split(fac[k + 1] * src[(k + 1) * ld])};
            Tf a[4][4];
#pragma unroll
            for (int m = ks / 2; m < 4; m++) {      // T is lower triangular
                const float2 x = *reinterpret_cast<const float2*>(sT + (16 * m + g) * DC_LDA + k), y = *reinterpret_cast<const float2*>(sT + (16 * m + g + 8) * DC_LDA + k);
                a[m][0] = tf_split(x.x); a[m][1] = tf_split(y.x); a[m][2] = tf_split(x.y); a[m][3] = tf_split(y.y);
            }
            float t[4][4];
#pragma unroll
            for (int m = ks / 2; m < 4; m++) {
                t[m][0] = t[m][1] = t[m][2] = t[m][3] = 0.0f;
                tf_mma(t[m], a[m][0].lo, a[m][1].lo, a[m][2].lo, a[m][3].lo, b[0].hi, b[1].hi);
            }
#pragma unroll
            for (int m = ks / 2; m < 4; m++) tf_mma(t[m], a[m][0].hi, a[m][1].hi, a[m][2].hi, a[m][3].hi, b[0].lo, b[1].lo);
#pragma unroll
            for (int m = ks / 2; m < 4; m++) tf_mma(t[m], a[m][0].hi, a[m][1].hi, a[m][2].hi, a[m][3].hi, b[0].hi, b[1].hi);
#pragma unroll
            for (int m = ks / 2; m < 4; m++)
#pragma unroll
                for (int e = 0; e < 4; e++) acc[m][e] += t[m][e];
        }
        // a sum that is not finite again, term by term: zeros above T's diagonal meet what stands in the tokens behind (0 times a NaN), and the parts' products make a
        // NaN of an infinity
        float all = 0.0f;
#pragma unroll
        for (int m = 0; m < 4; m++) all += (acc[m][0] + acc[m][1]) + (acc[m][2] + acc[m][3]);
        if (!tf_finite(all)) {
#pragma unroll
            for (int m = 0; m < 4; m++)
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    const int r = 16 * m + g + 8 * (e >> 1);
                    acc[m][e] = 0.0f;
#pragma unroll 1
                    for (int k = 0; k <= r; k++) acc[m][e] = fmaf(sT[r * DC_LDA + k], fac[k] * src[k * ld + 2 * t4 + (e & 1) - g], acc[m][e]);
                }
        }
        float* dst = is_w ? W_g : U_g;
        const int width = is_w ? LDQ : dv, c = c0 + 2 * t4;
        if (is_w || c < dv) {
#pragma unroll
            for (int m = 0; m < 4; m++) {
                *reinterpret_cast<float2*>(dst + (size_t)(16 * m + g) * width + c) = make_float2(acc[m][0], acc[m][1]);
                *reinterpret_cast<float2*>(dst + (size_t)(16 * m + g + 8) * width + c) = make_float2(acc[m][2], acc[m][3]);
            }
        }
    }
}

// grid (segments, H, slices of COLS columns); DKP / 16 warps: warp w has rows 16 w .. of the state's slice, and in the first product rows 16 (w & 3) .. of U and, with
// 16 columns, the 8 columns w >> 2.
constexpr int DC_STAGES = 3;

template <int DKP, int COLS, bool CH>
__global__ void __launch_bounds__(DKP * 2) delta_chunk_scan_kernel(const DcArgs p, const float* __restrict__ proj, int N, float* __restrict__ state,
                                                                   size_t state_stride, size_t conv_off, int taps, const WaitCtl wc) {
    constexpr int NTH = DKP * 2, LDQ = DKP + 8, LDS = DKP + 4, LDU = DC_C + 4, NT = COLS / 8, STAGE = 2 * DC_C * LDQ;
    static_assert(NT == DKP / 64, "the warps of the first product");
    extern __shared__ __align__(128) float ds_smem[];
    __shared__ __align__(8) uint64_t full[DC_STAGES];
    __shared__ int base_sh, failed;
    float* ring = ds_smem;
    float* sS = ring + DC_STAGES * STAGE;           // [COLS][LDS]
    float* sU = sS + COLS * LDS;                    // [COLS][LDU]
    const int seg = blockIdx.x, h = blockIdx.y, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t4 = lane & 3;
    const int slot = p.seg_slots[seg], start = p.seg_starts[seg], n = p.seg_starts[seg + 1] - start;
    if (slot < 0 || n <= p.from) return;
    if (warp == 0) {
        const int b = first_chunk_of<DC_C>(seg, p.seg_starts, p.from);
        if (lane == 0) {
            base_sh = b;
            failed = 0;
            for (int i = 0; i < DC_STAGES; i++) mbar_init(&full[i], 1);
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        }
    }
    const int dk = p.dk, dv = p.dv, H = p.H, c0 = blockIdx.z * COLS, chunks = (n + DC_C - 1) / DC_C;
    float* row = state + (size_t)slot * state_stride;
    for (int e = tid; e < COLS * DKP; e += NTH) {
        const int c = e / DKP, d = e % DKP;
        sS[c * LDS + d] = (c0 + c < dv && d < dk) ? row[((size_t)h * dv + c0 + c) * dk + d] : 0.0f;
    }
    __syncthreads();
    const size_t stride = dc_stride(dk, dv, CH);
    float* mine = p.scratch + ((size_t)base_sh * H + h) * stride;
    const size_t u_off = dc_u_off(dk), s_off = dc_s_off(dk, dv), e_off = dc_e_off(dk, dv);
    auto issue = [&](int c) {                       // thread 0: chunk c's W and Kg, one copy
        if (c >= chunks || c == wc.skip_stage) return;          // (a chunk named by wc.skip_stage is left out: a test of the give-up path)
        uint64_t* bar = &full[c % DC_STAGES];
        mbar_expect_tx(bar, STAGE * 4);
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                     ::"r"(smem_u32(ring + (c % DC_STAGES) * STAGE)), "l"(mine + (size_t)c * H * stride), "r"(STAGE * 4), "r"(smem_u32(bar)) : "memory");
    };
    float s[NT][4];                                 // this warp's rows of the state: rows d, d + 8, columns 8 i + 2 t4, + 1
    const int d = 16 * warp + g;
#pragma unroll
    for (int i = 0; i < NT; i++)
#pragma unroll
        for (int e = 0; e < 4; e++) s[i][e] = sS[(8 * i + 2 * t4 + (e & 1)) * LDS + d + 8 * (e >> 1)];
    const int ur = 16 * (warp & 3) + g, uc = 8 * (warp >> 2) + 2 * t4;          // this thread's places in U: rows ur, ur + 8, columns uc, + 1
    float2 up[2];
    float dec[2];
    auto fetch = [&](int c) {                       // U' and the decays of chunk c
        const float* in = mine + (size_t)(c < chunks ? c : 0) * H * stride;
        const bool on = c < chunks && c0 + uc < dv;
        up[0] = on ? *reinterpret_cast<const float2*>(in + u_off + (size_t)ur * dv + c0 + uc) : make_float2(0.0f, 0.0f);
        up[1] = on ? *reinterpret_cast<const float2*>(in + u_off + (size_t)(ur + 8) * dv + c0 + uc) : make_float2(0.0f, 0.0f);
        dec[0] = CH ? (d < dk ? in[e_off + d] : 0.0f) : in[e_off];
        dec[1] = CH ? (d + 8 < dk ? in[e_off + d + 8] : 0.0f) : dec[0];
    };
    if (tid == 0) {
        issue(0);
        issue(1);
    }
    fetch(0);
    for (int c = 0; c < chunks; c++) {
        if (!mbar_wait(&full[c % DC_STAGES], (c / DC_STAGES) & 1, wc.cycles)) give_up(wc.error, &failed, 61);
        __syncthreads();                            // the chunk's operands are there, the state's slice is written, and everybody has left the chunk before
        if (*reinterpret_cast<volatile int*>(&failed)) {        // the same for every thread: all have written it before the barrier or nobody has
            // this chunk's copy and the next one's may be in flight: they land before the block's memory goes, or the limit runs out again
            for (int d = c; d < chunks && d < c + 2; d++)
                if (d != wc.skip_stage) mbar_wait(&full[d % DC_STAGES], (d / DC_STAGES) & 1, wc.cycles);
            return;
        }
        if (tid == 0) issue(c + 2);
        float* in = mine + (size_t)c * H * stride;
        const float* sW = ring + (c % DC_STAGES) * STAGE;
        const float* sK = sW + DC_C * LDQ;
        for (int e = tid; e < COLS * (DKP / 4); e += NTH) {                     // the state before the chunk
            const int cc = e / (DKP / 4), dd = 4 * (e % (DKP / 4));
            if (c0 + cc < dv && dd < dk) *reinterpret_cast<float4*>(in + s_off + (size_t)(c0 + cc) * dk + dd) = *reinterpret_cast<const float4*>(sS + cc * LDS + dd);
        }
        // (a product of one sum waits some 70 cycles for the one before it: every step has sums of its own for the large products, added up in float32 (tf32.cuh says why),
        // and the small ones of all steps take turns on two sets each)
        float x[2][2][4], ws[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
        for (int j = 0; j < 2; j++)
#pragma unroll
            for (int i = 0; i < 2; i++)
#pragma unroll
                for (int e = 0; e < 4; e++) x[j][i][e] = 0.0f;
        const float* wa = sW + ur * LDQ + 2 * t4;
        const float* sb = sS + (8 * (warp >> 2) + g) * LDS + 2 * t4;
#pragma unroll
        for (int ks = 0; ks < DKP / 8; ks++) {
            const float2 a0 = *reinterpret_cast<const float2*>(wa + ks * 8), a1 = *reinterpret_cast<const float2*>(wa + 8 * LDQ + ks * 8);
            const float2 b0 = *reinterpret_cast<const float2*>(sb + ks * 8);
            const Tf a[4] = {tf_split(a0.x), tf_split(a1.x), tf_split(a0.y), tf_split(a1.y)}, b[2] = {tf_split(b0.x), tf_split(b0.y)};
            float t[4] = {0.0f, 0.0f, 0.0f, 0.0f};
            tf_mma(t, a[0].hi, a[1].hi, a[2].hi, a[3].hi, b[0].hi, b[1].hi);
            tf_mma(x[ks & 1][0], a[0].lo, a[1].lo, a[2].lo, a[3].lo, b[0].hi, b[1].hi);
            tf_mma(x[ks & 1][1], a[0].hi, a[1].hi, a[2].hi, a[3].hi, b[0].lo, b[1].lo);
#pragma unroll
            for (int e = 0; e < 4; e++) ws[e] += t[e];
        }
#pragma unroll
        for (int e = 0; e < 4; e++) ws[e] += (x[0][0][e] + x[1][0][e]) + (x[0][1][e] + x[1][1][e]);
        const float2 u[2] = {make_float2(up[0].x - ws[0], up[0].y - ws[1]), make_float2(up[1].x - ws[2], up[1].y - ws[3])};
        sU[uc * LDU + ur] = u[0].x;
        sU[(uc + 1) * LDU + ur] = u[0].y;
        sU[uc * LDU + ur + 8] = u[1].x;
        sU[(uc + 1) * LDU + ur + 8] = u[1].y;
        if (c0 + uc < dv) {
            *reinterpret_cast<float2*>(in + u_off + (size_t)ur * dv + c0 + uc) = u[0];
            *reinterpret_cast<float2*>(in + u_off + (size_t)(ur + 8) * dv + c0 + uc) = u[1];
        }
        const float da = dec[0], db = dec[1];
        fetch(c + 1);
        __syncthreads();                            // U is there, and nobody reads the old state any more
        constexpr int SETS = 2 / NT;
        float y[NT][SETS][2][4], z[NT][4];
#pragma unroll
        for (int i = 0; i < NT; i++)
#pragma unroll
            for (int e = 0; e < 4; e++) {
                z[i][e] = 0.0f;
#pragma unroll
                for (int q = 0; q < SETS; q++) y[i][q][0][e] = y[i][q][1][e] = 0.0f;
            }
#pragma unroll
        for (int ks = 0; ks < DC_C / 8; ks++) {
            const float* ka = sK + (ks * 8 + t4) * LDQ + d;
            const Tf a[4] = {tf_split(ka[0]), tf_split(ka[8]), tf_split(ka[4 * LDQ]), tf_split(ka[4 * LDQ + 8])};
#pragma unroll
            for (int i = 0; i < NT; i++) {
                const float* ub = sU + (8 * i + g) * LDU + ks * 8 + t4;
                const Tf b[2] = {tf_split(ub[0]), tf_split(ub[4])};
                float t[4] = {0.0f, 0.0f, 0.0f, 0.0f};
                tf_mma(t, a[0].hi, a[1].hi, a[2].hi, a[3].hi, b[0].hi, b[1].hi);
                tf_mma(y[i][ks % SETS][0], a[0].lo, a[1].lo, a[2].lo, a[3].lo, b[0].hi, b[1].hi);
                tf_mma(y[i][ks % SETS][1], a[0].hi, a[1].hi, a[2].hi, a[3].hi, b[0].lo, b[1].lo);
#pragma unroll
                for (int e = 0; e < 4; e++) z[i][e] += t[e];
            }
        }
#pragma unroll
        for (int i = 0; i < NT; i++)
#pragma unroll
            for (int e = 0; e < 4; e++) {
                float add = z[i][e];
#pragma unroll
                for (int q = 0; q < SETS; q++) add += y[i][q][0][e] + y[i][q][1][e];
                s[i][e] = fmaf(e < 2 ? da : db, s[i][e], add);
                sS[(8 * i + 2 * t4 + (e & 1)) * LDS + d + 8 * (e >> 1)] = s[i][e];
            }
    }
    __syncthreads();
    for (int e = tid; e < COLS * DKP; e += NTH) {
        const int c = e / DKP, dd = e % DKP;
        if (c0 + c < dv && dd < dk) row[((size_t)h * dv + c0 + c) * dk + dd] = sS[c * LDS + dd];
    }
    // the convolution's memory: the last taps-1 inputs of the request, this step's tokens included
    if (taps > 1) {
        const int Cq = 2 * p.G * dk + H * dv;
        float* cs = row + conv_off;
        const int nb = gridDim.y * gridDim.z, bi = h * gridDim.z + blockIdx.z;
        for (int chn = bi * NTH + tid; chn < Cq; chn += nb * NTH) {
            float keep[DC_MAX_TAPS];
#pragma unroll
            for (int rr = 0; rr < DC_MAX_TAPS; rr++)
                if (rr < taps - 1) {
                    const int src = n - (taps - 1) + rr;
                    keep[rr] = src >= 0 ? proj[(size_t)(start + src) * N + chn] : cs[(size_t)(rr + n) * Cq + chn];
                }
#pragma unroll
            for (int rr = 0; rr < DC_MAX_TAPS; rr++)
                if (rr < taps - 1) cs[(size_t)rr * Cq + chn] = keep[rr];
        }
    }
}

// grid (chunks, H, slices of COLS columns); 256 threads: warp w has rows 16 (w & 3) .. and half of the slice's columns, w >> 2.  norm_w (null: o [tokens][H dv] gets the
// outputs as they are): out [tokens][H dv] in T gets o / rms(o) over the head's dv <= COLS values * norm_w * silu(gate), the gate at gate_off of proj's rows.
template <int DKP, int COLS, typename T>
__global__ void __launch_bounds__(256) delta_chunk_out_kernel(const DcArgs p, bool ch_decay, float* __restrict__ o, const float* __restrict__ proj, int N, int gate_off,
                                                              const float* __restrict__ norm_w, float eps, T* __restrict__ out) {
    constexpr int LDQ = DKP + 8, LDU = COLS + 4, NT = COLS / 16;
    extern __shared__ __align__(16) float do_smem[];
    __shared__ int find[4];
    __shared__ float squares[2][DC_C];
    float* sQ = do_smem;                            // [64][LDQ]
    float* sS = sQ + DC_C * LDQ;                    // [COLS columns][LDQ]
    float* sP = sS + COLS * LDQ;                    // [64][DC_LDA]
    float* sU = sP + DC_C * DC_LDA;                 // [64][LDU]
    const Chunk ch = find_chunk<DC_C>(blockIdx.x, p.seg_starts, p.segments, find, p.from);
    if (ch.seg < 0 || p.seg_slots[ch.seg] < 0) return;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t4 = lane & 3, m = warp & 3, half = warp >> 2, cw = (COLS / 2) * half;
    const int h = blockIdx.y, c0 = blockIdx.z * COLS, dk = p.dk, dv = p.dv;
    const float* in = p.scratch + ((size_t)blockIdx.x * p.H + h) * dc_stride(dk, dv, ch_decay);
    for (int e = tid; e < DC_C * (DKP / 4); e += 256) {
        const int r = e / (DKP / 4), d = 4 * (e % (DKP / 4));
        copy16_or_zero(sQ + r * LDQ + d, in + dc_q_off(dk) + (d < dk ? (size_t)r * dk + d : 0), d < dk);
    }
    for (int e = tid; e < COLS * (DKP / 4); e += 256) {
        const int r = e / (DKP / 4), d = 4 * (e % (DKP / 4));
        const bool on = d < dk && c0 + r < dv;
        copy16_or_zero(sS + r * LDQ + d, in + dc_s_off(dk, dv) + (on ? (size_t)(c0 + r) * dk + d : 0), on);
    }
    for (int e = tid; e < DC_C * 16; e += 256) {
        const int r = e / 16, c = 4 * (e % 16);
        copy16_or_zero(sP + r * DC_LDA + c, in + dc_p_off(dk) + r * DC_C + c, true);
    }
    for (int e = tid; e < DC_C * (COLS / 4); e += 256) {
        const int r = e / (COLS / 4), c = 4 * (e % (COLS / 4));
        const bool on = c0 + c < dv;
        copy16_or_zero(sU + r * LDU + c, in + dc_u_off(dk) + (on ? (size_t)r * dv + c0 + c : 0), on);
    }
    tf_commit();
    // the gate's values are asked for with the operands
    float2 gt[2][NT];
    if (norm_w) {
#pragma unroll
        for (int u = 0; u < 2; u++) {
            const int r = 16 * m + g + 8 * u;
            const float* gate = proj + (size_t)(ch.first + (r < ch.rows ? r : 0)) * N + gate_off + (size_t)h * dv;
#pragma unroll
            for (int i = 0; i < NT; i++) {
                const int c = cw + 8 * i + 2 * t4;
                gt[u][i] = c < dv ? make_float2(gate[c], gate[c + 1]) : make_float2(0.0f, 0.0f);
            }
        }
    }
    tf_wait<0>();
    __syncthreads();
    float acc[NT][4];
#pragma unroll
    for (int i = 0; i < NT; i++)
#pragma unroll
        for (int e = 0; e < 4; e++) acc[i][e] = 0.0f;
    auto step = [&](const float* pa, int lda, auto&& right) {
        const float2 x = *reinterpret_cast<const float2*>(pa), y = *reinterpret_cast<const float2*>(pa + 8 * lda);
        const Tf a[1][4] = {{tf_split(x.x), tf_split(y.x), tf_split(x.y), tf_split(y.y)}};
#pragma unroll
        for (int i0 = 0; i0 < NT; i0 += 4) {
            Tf b[4][2];
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const float2 v = right(i0 + i);
                b[i][0] = tf_split(v.x);
                b[i][1] = tf_split(v.y);
            }
            float* const d_[1][4] = {{acc[i0], acc[i0 + 1], acc[i0 + 2], acc[i0 + 3]}};
            tf_mma3(d_, a, b);
        }
    };
    if (16 * m < ch.rows) {
#pragma unroll 2
        for (int ks = 0; ks < DKP / 8; ks++) {
            const int k = ks * 8 + 2 * t4;
            step(sQ + (16 * m + g) * LDQ + k, LDQ, [&](int i) { return *reinterpret_cast<const float2*>(sS + (cw + 8 * i + g) * LDQ + k); });
        }
#pragma unroll 2
        for (int ks = 0; ks < 2 * (m + 1); ks++) {  // (P is lower triangular)
            const int k = ks * 8 + 2 * t4;
            step(sP + (16 * m + g) * DC_LDA + k, DC_LDA, [&](int i) { const float* ub = sU + k * LDU + cw + 8 * i + g; return make_float2(ub[0], ub[LDU]); });
        }
    }
    // an output that is not finite again, term by term, without the tokens behind it (see delta_chunk_prepare)
    float all = 0.0f;
#pragma unroll
    for (int i = 0; i < NT; i++) all += (acc[i][0] + acc[i][1]) + (acc[i][2] + acc[i][3]);
    if (!tf_finite(all)) {
        auto again = [&](int r, int c) {
            float s = 0.0f;
#pragma unroll 1
            for (int d = 0; d < dk; d++) s = fmaf(sQ[r * LDQ + d], sS[c * LDQ + d], s);
#pragma unroll 1
            for (int k = 0; k <= r; k++) s = fmaf(sP[r * DC_LDA + k], sU[k * LDU + c], s);
            return s;
        };
#pragma unroll
        for (int i = 0; i < NT; i++)
#pragma unroll
            for (int e = 0; e < 4; e++) acc[i][e] = again(16 * m + g + 8 * (e >> 1), cw + 8 * i + 2 * t4 + (e & 1));
    }
    if (!norm_w) {
#pragma unroll
        for (int i = 0; i < NT; i++)
#pragma unroll
            for (int u = 0; u < 2; u++) {
                const int r = 16 * m + g + 8 * u, c = c0 + cw + 8 * i + 2 * t4;
                if (r < ch.rows && c < dv) *reinterpret_cast<float2*>(o + ((size_t)(ch.first + r) * p.H + h) * dv + c) = make_float2(acc[i][2 * u], acc[i][2 * u + 1]);
            }
        return;
    }
#pragma unroll
    for (int u = 0; u < 2; u++) {
        float ss = 0.0f;
#pragma unroll
        for (int i = 0; i < NT; i++) {
            ss = fmaf(acc[i][2 * u], acc[i][2 * u], ss);
            ss = fmaf(acc[i][2 * u + 1], acc[i][2 * u + 1], ss);
        }
        ss += __shfl_xor_sync(0xffffffffu, ss, 1);
        ss += __shfl_xor_sync(0xffffffffu, ss, 2);
        if (t4 == 0) squares[half][16 * m + g + 8 * u] = ss;
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < 2; u++) {
        const int r = 16 * m + g + 8 * u;
        if (r >= ch.rows) continue;
        const float inv = 1.0f / sqrtf((squares[0][r] + squares[1][r]) / (float)dv + eps);
        T* orow = out + ((size_t)(ch.first + r) * p.H + h) * dv;
#pragma unroll
        for (int i = 0; i < NT; i++) {
            const int c = cw + 8 * i + 2 * t4;
            if (c >= dv) continue;
            float v[2];
#pragma unroll
            for (int e = 0; e < 2; e++) {
                const float x = e ? gt[u][i].y : gt[u][i].x;
                v[e] = ((acc[i][2 * u + e] * inv) * norm_w[c + e]) * (x / (1.0f + expf(-x)));
            }
            if (sizeof(T) == 2) *reinterpret_cast<__nv_bfloat162*>(orow + c) = __floats2bfloat162_rn(v[0], v[1]);
            else { orow[c] = from_f32<T>(v[0]); orow[c + 1] = from_f32<T>(v[1]); }
        }
    }
}

}  // namespace vk

using namespace vk;

static int dc_chunks(int tokens, int segments, int from) { return most_chunks(DC_C, tokens, segments, from); }

// Whether the chunked kernels take these sizes (else the token-by-token kernel does the work).
VK_API int vk_delta_chunked_takes(int G, int H, int dk, int dv, int taps) {
    return G > 0 && H > 0 && H % G == 0 && dk % 4 == 0 && dk >= 8 && dk <= 128 && dv > 0 && dv % 4 == 0 && dv <= 256 && taps >= 1 && taps <= DC_MAX_TAPS;
}

// Bytes of scratch for a step of `tokens` tokens in `segments` segments (from: as for the kernels; the larger it is, the fewer chunks a step of many segments can
// have, each with its operands and a head's whole state: 0.22 MB a head of 128 x 128).
VK_API size_t vk_delta_chunked_scratch_bytes(int tokens, int segments, int H, int dk, int dv, int from) {
    return (size_t)dc_chunks(tokens, segments, from) * H * dc_stride(dk, dv, false) * sizeof(float);
}

// Whether delta_chunk_out norms and gates the outputs itself (else the gate kernel follows): a head's values lie in one of its blocks.
VK_API int vk_delta_chunked_gates(int dv) { return dv <= 128; }

struct DcOut {
    float* o;
    const float* proj;
    int N, gate_off;
    const float* norm_w;                    // null: o
    float eps;
    void* out;
    int dtype;
};

template <int DKP, int COLS, typename T>
static int delta_out_launch(const DcArgs& p, bool ch, const DcOut& f, int chunks, cudaStream_t stream) {
    auto kern = delta_chunk_out_kernel<DKP, COLS, T>;
    const int smem = (DC_C * (DKP + 8) + COLS * (DKP + 8) + DC_C * DC_LDA + DC_C * (COLS + 4)) * (int)sizeof(float);
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return (int)e;
    return launch_plain(kern, dim3(chunks, p.H, (p.dv + COLS - 1) / COLS), dim3(256), smem, stream, p, ch, f.o, f.proj, f.N, f.gate_off, f.norm_w, f.eps, (T*)f.out);
}

template <int DKP, bool CH>
static int delta_chunked_launch(const DcArgs& p, const float* proj, int proj_width, float* state, size_t state_stride, const DcOut& f, int tokens, int taps,
                                int* error, cudaStream_t stream) {
    constexpr int COLS = DKP / 8;
    const int chunks = dc_chunks(tokens, p.segments, p.from);
    const int smem1 = (dc_prepare_floats_fixed<DKP, CH>() + DC_C * dc_ldv(p.dv)) * (int)sizeof(float);
    const int smem2 = (DC_STAGES * 2 * DC_C * (DKP + 8) + COLS * (DKP + 4) + COLS * (DC_C + 4)) * (int)sizeof(float);
    auto k1 = delta_chunk_prepare_kernel<DKP, CH>;
    auto k2 = delta_chunk_scan_kernel<DKP, COLS, CH>;
    cudaError_t e = cudaFuncSetAttribute(k1, cudaFuncAttributeMaxDynamicSharedMemorySize, smem1);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k2, cudaFuncAttributeMaxDynamicSharedMemorySize, smem2);
    if (e != cudaSuccess) return (int)e;
    int rc = launch_plain(k1, dim3(chunks, p.H), dim3(256), smem1, stream, p);
    if (rc != VK_OK) return rc;
    rc = launch_plain(k2, dim3(p.segments, p.H, (p.dv + COLS - 1) / COLS), dim3(DKP * 2), smem2, stream, p, proj, proj_width, state, state_stride,
                      (size_t)p.H * p.dv * p.dk, taps, wait_ctl(error, WAIT_FAMILY_DELTA));
    if (rc != VK_OK) return rc;
    // slices of 128 columns only where a head's outputs are normed here: the smaller block's two a multiprocessor are otherwise the better
    if (f.norm_w && p.dv > 64)
        return f.dtype == 0 ? delta_out_launch<DKP, 128, float>(p, CH, f, chunks, stream) : delta_out_launch<DKP, 128, __nv_bfloat16>(p, CH, f, chunks, stream);
    return f.dtype == 0 ? delta_out_launch<DKP, 64, float>(p, CH, f, chunks, stream) : delta_out_launch<DKP, 64, __nv_bfloat16>(p, CH, f, chunks, stream);
}

template <bool CH>
static int delta_chunked(const float* prep, int prep_width, const float* proj, int proj_width, const int32_t* seg_starts, const int32_t* seg_slots, float* state,
                         size_t state_stride, const DcOut& f, float* scratch, int segments, int from, int tokens, int G, int H, int dk, int dv, int taps,
                         int* error, cudaStream_t stream) {
    if (segments <= 0 || tokens <= 0) return VK_OK;
    if (!vk_delta_chunked_takes(G, H, dk, dv, taps) || prep_width % 4 || from < 0 || !error || (f.norm_w && !vk_delta_chunked_gates(dv))) return VK_BAD_SHAPE;
    if ((uintptr_t)scratch % 16 || (uintptr_t)prep % 16 || (uintptr_t)f.o % 8 || (f.norm_w && (uintptr_t)f.out % 4)) return VK_BAD_ALIGNMENT;
    if (H > 65535) return VK_TOO_LARGE;
    const DcArgs p = {prep, prep_width, seg_starts, seg_slots, segments, from, scratch, G, H, dk, dv};
    return dk <= 64 ? delta_chunked_launch<64, CH>(p, proj, proj_width, state, state_stride, f, tokens, taps, error, stream)
                    : delta_chunked_launch<128, CH>(p, proj, proj_width, state, state_stride, f, tokens, taps, error, stream);
}

// prep [tokens][prep width] as delta_prepare leaves it; proj as for the token-by-token kernel; three kernels.  norm_w null: o [tokens][H*dv] float32 gets the outputs.
// Segments of up to `from` tokens are left alone: their states and rows are for the token-by-token kernels.  norm_w given (sizes that vk_delta_chunked_gates): out [tokens][H*dv] in dtype gets them as vk_delta_gate makes them.  error: as for vk_linear_tcgen05.
VK_API int vk_delta_chunked(const float* prep, int prep_width, const float* proj, const int32_t* seg_starts, const int32_t* seg_slots, float* state,
                            size_t state_stride, float* o, float* scratch, const float* norm_w, float eps, void* out, int dtype, int segments, int from,
                            int tokens, int G, int H, int dk, int dv, int taps, int* error, cudaStream_t stream) {
    const int N = 2 * G * dk + 2 * H * dv + 2 * H;
    const DcOut f = {o, proj, N, 2 * G * dk + H * dv, norm_w, eps, out, dtype};
    return delta_chunked<false>(prep, prep_width, proj, N, seg_starts, seg_slots, state, state_stride, f, scratch, segments, from, tokens, G, H, dk, dv, taps, error, stream);
}

// The form with a decay per head and key channel: prep as cdelta_prepare leaves it, proj rows of proj_width floats (the
// convolution's inputs first).  The sizes are those vk_delta_chunked_takes.
VK_API size_t vk_cdelta_chunked_scratch_bytes(int tokens, int segments, int H, int dk, int dv, int from) {
    return (size_t)dc_chunks(tokens, segments, from) * H * dc_stride(dk, dv, true) * sizeof(float);
}

VK_API int vk_cdelta_chunked(const float* prep, int prep_width, const float* proj, int proj_width, const int32_t* seg_starts,
                             const int32_t* seg_slots, float* state, size_t state_stride, float* o, float* scratch, int segments, int from, int tokens,
                             int G, int H, int dk, int dv, int taps, int* error, cudaStream_t stream) {
    const DcOut f = {o, nullptr, 0, 0, nullptr, 0.0f, nullptr, 0};
    return delta_chunked<true>(prep, prep_width, proj, proj_width, seg_starts, seg_slots, state, state_stride, f, scratch, segments, from, tokens, G, H, dk, dv, taps,
                               error, stream);
}
