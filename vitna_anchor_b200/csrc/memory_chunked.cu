// The matrix memories' recurrences over a prompt's portion in chunks of 64 tokens on the tensor cores: mLSTM (mlstm.cu states it) and gated linear
// attention (gla.cu states it).  A request's state S [dim][vdim] before a chunk is all that the chunk needs of the tokens before it:
//
//   gated linear attention, L_t[d] = sum of ln a up to and with token t of the chunk:
//     o_t = sum_d q_t[d] e^(L_t[d]) S[d] + sum_(i <= t) (sum_d q_t[d] k_i[d] e^(L_t[d] - L_i[d])) v_i,     S' = diag(e^(L_64)) S + sum_i (e^(L_64 - L_i) k_i) v_i^T
//   mLSTM, F_t = sum of f up to t, A_i = i_i - F_i, N_t = max(m, max_(i <= t) A_i), m the running maximum before the chunk (m_t = F_t + N_t):
//     numerators = e^(m - N_t) S^T q_t + sum_(i <= t) e^(A_i - N_t) (q_t . k_i) v_i,     S' = e^(m - N_64) S + sum_i e^(A_i - N_64) k_i v_i^T,   n likewise with 1 for v
//
//   mlstm_chunk_gates   a block a head and segment: the gates, F, A and N's running maxima in float64 (a sum of 64 logarithms may be hundreds, and what counts
//                       are differences of neighbours), m before every chunk, the tokens' weights in what a chunk adds, and the m after the last token.
//   gla_chunk_decays    16 tokens a block: log2 a of every channel.  Wherever a weight spans several tokens their logarithms are added up for that very span, at
//                       most 16 of them; longer spans are products of such factors, each at most 1.  No difference of two sums is ever taken.
//   cm_add              what a chunk adds to a head's state, all chunks side by side, 64 x 64 of it a block.
//   cm_scan             the states before every chunk, in the place of what the chunk before added: four elements a thread, a request's chunks in order.
//   cm_out              a block a chunk and head, all chunks side by side: the weighted q k^T, its product with v, q with the state, and the norm and gate of
//                       the head's outputs, in the compute dtype.
//
// Why chunks: token after token the recurrence is a chain of 2,048 steps of 0.24 us in at most 136 blocks.  Every exponent here is at most 0.
//
// Products take float32 operands as two tf32 parts (tf32.cuh).
//
// Measured, a whole mixer with its two products: mLSTM, one request of 2,048 tokens, 8 heads of 128 x 256: 599 us token after token, 200 us here (gates 14,
// cm_add 26, cm_scan 10, cm_out 64 to 70: the tensor cores' rate for three tf32 products is 23 us of it on the multiprocessors that have two of its blocks);
// gated linear attention, 1,204 + 807 tokens, 4 heads of 64 x 256: 279 and 110 us (decays 7, cm_add 9, cm_scan 8, cm_out 39: 128 blocks of one wave).  A first form
// whose blocks walked the chunks in order with their tile of the state in the accumulators took 2.9 us a chunk, 90 us for cm_add's and cm_scan's work.
#include "chunks.cuh"
#include "common.cuh"
#include "tf32.cuh"

namespace vk {

constexpr int CM_Q = 64;                    // tokens of a chunk
constexpr int CM_LOCAL = 16;                // tokens over which a channel's logarithms are added up (gated linear attention)
constexpr int CM_T = 64, CM_LD = CM_T + 8;   // the tile of the state that a block of cm_add works out, and a padded row of one of its operands

struct CmArgs {
    const float* proj;              // [tokens][N]: q | k | v | ..
    int N, H, dk, dv, segments, from;       // segments of up to `from` tokens are left alone
    const int32_t* seg_starts;
    const int32_t* seg_slots;
    float* state;                   // [slots][state_floats]
    size_t state_floats;
    float* before;                  // scratch, [chunks][H][dk][dv]: what the chunks add, then the states before them
    float* decay;                   // [chunks][H] (mLSTM) or [chunks][H][dk]: what a chunk leaves of the state before it
    // mLSTM
    float* n_before;                // [chunks][H][dk], as `before`
    float* weight;                  // [tokens][H]: e^(A - N of the chunk's last token)
    double* A;                      // [tokens][H] each
    double* G;                      // the largest A up to a token, inside its chunk
    double* F;
    double* m_before;               // [chunks][H]
    // gated linear attention
    float* logs;                    // [tokens][H dk]: log2 of the decays
};

// -- mLSTM: the gates -----------------------------------------------------------------------------------------------------------------------

constexpr int MG_THREADS = 512, MG_BATCH = 128;     // chunks whose maxima meet at a time

__global__ void __launch_bounds__(MG_THREADS) mlstm_chunk_gates_kernel(const CmArgs p, const float* __restrict__ gate_bias, float cap) {
    __shared__ double sF[MG_BATCH], sG[MG_BATCH], sM[MG_BATCH];
    __shared__ int base_sh;
    const int h = blockIdx.x, seg = blockIdx.y, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, H = p.H;
    const int first = p.seg_starts[seg], end = p.seg_starts[seg + 1], slot = p.seg_slots[seg];
    if (end - first <= p.from) return;
    if (warp == 0) {
        const int b = first_chunk_of<CM_Q>(seg, p.seg_starts, p.from);
        if (lane == 0) base_sh = b;
    }
    const int chunks = (end - first + CM_Q - 1) / CM_Q;
    float* m_st = slot >= 0 ? p.state + (size_t)slot * p.state_floats + (size_t)H * p.dk * p.dv + (size_t)H * p.dk + h : nullptr;
    double m = m_st ? (double)*m_st : 0.0;                            // carried by thread 0
    const int i_off = 2 * H * p.dk + 2 * H * p.dv + h, f_off = i_off + H;
    const float bi = gate_bias[h], bf = gate_bias[H + h];
    for (int c0 = 0; c0 < chunks; c0 += MG_BATCH) {
        const int cnt = min(MG_BATCH, chunks - c0);
        __syncthreads();
        for (int c = warp; c < cnt; c += MG_THREADS / 32) {
            const int t0 = first + (c0 + c) * CM_Q + 2 * lane;
            double f[2], a[2];
            float gi[2];
#pragma unroll
            for (int u = 0; u < 2; u++) {
                const bool on = t0 + u < end;
                const float* row = p.proj + (size_t)(on ? t0 + u : first) * p.N;
                gi[u] = on ? cap * tanhf((row[i_off] + bi) / cap) : -INFINITY;
                f[u] = on ? (double)log_sigmoid(cap * tanhf((row[f_off] + bf) / cap)) : 0.0;
            }
            double sum = f[0] + f[1];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const double v = __shfl_up_sync(0xffffffffu, sum, o);
                if (lane >= o) sum += v;
            }
            const double f1 = sum, f0 = sum - f[1];
            a[0] = (double)gi[0] - f0;
            a[1] = (double)gi[1] - f1;
            double g = fmax(a[0], a[1]);
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const double v = __shfl_up_sync(0xffffffffu, g, o);
                if (lane >= o) g = fmax(g, v);
            }
            const double before = __shfl_up_sync(0xffffffffu, g, 1);
            const double g0 = lane > 0 ? fmax(before, a[0]) : a[0];
            if (t0 < end) {
                const size_t at = (size_t)t0 * H + h;
                p.A[at] = a[0]; p.G[at] = g0; p.F[at] = f0;
            }
            if (t0 + 1 < end) {
                const size_t at = (size_t)(t0 + 1) * H + h;
                p.A[at] = a[1]; p.G[at] = g; p.F[at] = f1;
            }
            if (lane == 31) { sF[c] = f1; sG[c] = g; }
        }
        __syncthreads();
        if (tid == 0) {
            for (int c = 0; c < cnt; c++) {
                sM[c] = m;
                m = sF[c] + fmax(m, sG[c]);
            }
        }
        __syncthreads();
        for (int c = warp; c < cnt; c += MG_THREADS / 32) {
            const double N = fmax(sM[c], sG[c]);
            const int t0 = first + (c0 + c) * CM_Q + 2 * lane;        // (a thread reads the A that it wrote)
#pragma unroll
            for (int u = 0; u < 2; u++)
                if (t0 + u < end) p.weight[(size_t)(t0 + u) * H + h] = expf((float)(p.A[(size_t)(t0 + u) * H + h] - N));
            if (lane == 0) {
                p.m_before[(size_t)(base_sh + c0 + c) * H + h] = sM[c];
                p.decay[(size_t)(base_sh + c0 + c) * H + h] = expf((float)(sM[c] - N));
            }
        }
    }
    if (tid == 0 && m_st) *m_st = (float)m;
}

// -- gated linear attention: the decays -------------------------------------------------------------------------------------------------------

constexpr int GD_THREADS = 128;

// grid (chunks x 4, channels / 128)
__global__ void __launch_bounds__(GD_THREADS) gla_chunk_decays_kernel(const CmArgs p, int a_off, int rank, const float* __restrict__ a2t,
                                                                      const float* __restrict__ bias, float inv_tau) {
    extern __shared__ float gd_sh[];                    // [rank][16]
    __shared__ int find[4];
    const Chunk ch = find_chunk<CM_Q>(blockIdx.x / 4, p.seg_starts, p.segments, find, p.from);
    const int r0 = (blockIdx.x & 3) * CM_LOCAL, cnt = ch.seg < 0 ? 0 : min(CM_LOCAL, ch.rows - r0);
    if (cnt <= 0) return;
    const int first = ch.first + r0, c = blockIdx.y * GD_THREADS + threadIdx.x, C = p.H * p.dk;
    for (int i = threadIdx.x; i < rank * CM_LOCAL; i += GD_THREADS) {
        const int t = i / rank, j = i - t * rank;
        gd_sh[j * CM_LOCAL + t] = t < cnt ? p.proj[(size_t)(first + t) * p.N + a_off + j] : 0.0f;
    }
    __syncthreads();
    if (c >= C) return;
    float z[CM_LOCAL];
#pragma unroll
    for (int t = 0; t < CM_LOCAL; t++) z[t] = 0.0f;
    for (int j = 0; j < rank; j++) {
        const float w = a2t[(size_t)j * C + c];
#pragma unroll
        for (int t = 0; t < CM_LOCAL; t++) z[t] = fmaf(gd_sh[j * CM_LOCAL + t], w, z[t]);
    }
    const float b = bias[c];
#pragma unroll
    for (int t = 0; t < CM_LOCAL; t++)
        if (t < cnt) p.logs[(size_t)(first + t) * C + c] = log_sigmoid(z[t] + b) * inv_tau * 1.4426950408889634f;
}

// -- the states before the chunks ---------------------------------------------------------------------------------------------------------------

// grid (chunks, H, tiles of 64 x 64); warp w has rows 32 (w & 1) .. and columns 32 (w >> 1) ..
template <bool MLSTM>
__global__ void __launch_bounds__(128) cm_add_kernel(const CmArgs p, int col_tiles) {
    extern __shared__ __align__(16) float ca_smem[];
    __shared__ float wt[CM_Q];                      // mLSTM: the tokens' weights
    __shared__ int find[4];
    float* sk = ca_smem;                            // [64][CM_LD] k
    float* sv = sk + CM_Q * CM_LD;                  // [64][CM_LD] v
    float* sl = sv + CM_Q * CM_LD;                  // [64][CM_LD] the decays' logarithms (gated linear attention)
    const Chunk ch = find_chunk<CM_Q>(blockIdx.x, p.seg_starts, p.segments, find, p.from);
    if (ch.seg < 0) return;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t4 = lane & 3, wd = (warp & 1) * 32, wv = (warp >> 1) * 32;
    const int h = blockIdx.y, H = p.H, dk = p.dk, dv = p.dv, rows = ch.rows;
    const int d0 = (blockIdx.z / col_tiles) * CM_T, v0 = (blockIdx.z % col_tiles) * CM_T;
    for (int e = tid; e < CM_Q * (CM_T / 4); e += 128) {
        const int r = e / (CM_T / 4), c = 4 * (e % (CM_T / 4));
        const bool onk = r < rows && d0 + c < dk, onv = r < rows && v0 + c < dv;
        const float* row = p.proj + (size_t)(ch.first + (r < rows ? r : 0)) * p.N;
        copy16_or_zero(sk + r * CM_LD + c, onk ? row + H * dk + h * dk + d0 + c : p.proj, onk);
        copy16_or_zero(sv + r * CM_LD + c, onv ? row + 2 * H * dk + h * dv + v0 + c : p.proj, onv);
        if (!MLSTM) copy16_or_zero(sl + r * CM_LD + c, onk ? p.logs + (size_t)(ch.first + r) * H * dk + h * dk + d0 + c : p.proj, onk);
    }
    tf_commit();
    if (MLSTM && tid < CM_Q) wt[tid] = tid < rows ? p.weight[(size_t)(ch.first + tid) * H + h] : 0.0f;
    tf_wait<0>();
    __syncthreads();
    const size_t at = (size_t)blockIdx.x * H + h;
    if (!MLSTM) {
        // k times what the tokens behind it leave of it: a thread has a channel of two pieces of 16 tokens (rows and channels that are not there hold zeros)
        const int d = tid & (CM_T - 1), part = tid / CM_T;
        float total[CM_Q / CM_LOCAL];
#pragma unroll
        for (int s = 0; s < CM_Q / CM_LOCAL; s++) {
            total[s] = 0.0f;
#pragma unroll
            for (int r = 0; r < CM_LOCAL; r++) total[s] += sl[(s * CM_LOCAL + r) * CM_LD + d];
            total[s] = tf_exp2(total[s]);
        }
        if (part == 0 && v0 == 0 && d0 + d < dk) p.decay[at * dk + d0 + d] = total[0] * total[1] * total[2] * total[3];
#pragma unroll
        for (int s = 0; s < CM_Q / CM_LOCAL; s++) {
            if (s / 2 != part) continue;
            float after = 1.0f, sum = 0.0f;
#pragma unroll
            for (int u = s + 1; u < CM_Q / CM_LOCAL; u++) after *= total[u];
#pragma unroll
            for (int r = CM_LOCAL - 1; r >= 0; r--) {
                float* k = sk + (s * CM_LOCAL + r) * CM_LD + d;
                *k *= tf_exp2(sum) * after;
                sum += sl[(s * CM_LOCAL + r) * CM_LD + d];
            }
        }
        __syncthreads();
    }
    float acc[2][4][4];
#pragma unroll
    for (int m = 0; m < 2; m++)
#pragma unroll
        for (int n = 0; n < 4; n++)
#pragma unroll
            for (int e = 0; e < 4; e++) acc[m][n][e] = 0.0f;
    float* const d_[2][4] = {{acc[0][0], acc[0][1], acc[0][2], acc[0][3]}, {acc[1][0], acc[1][1], acc[1][2], acc[1][3]}};
    const int steps = (rows + 7) / 8;
#pragma unroll 2
    for (int ks = 0; ks < steps; ks++) {
        Tf a[2][4], b[4][2];
#pragma unroll
        for (int m = 0; m < 2; m++) {
            const float* ka = sk + (ks * 8 + t4) * CM_LD + wd + 16 * m + g;
            a[m][0] = tf_split(ka[0]); a[m][1] = tf_split(ka[8]); a[m][2] = tf_split(ka[4 * CM_LD]); a[m][3] = tf_split(ka[4 * CM_LD + 8]);
        }
        const float w0 = MLSTM ? wt[ks * 8 + t4] : 1.0f, w1 = MLSTM ? wt[ks * 8 + t4 + 4] : 1.0f;
#pragma unroll
        for (int n = 0; n < 4; n++) {
            const float* vb = sv + (ks * 8 + t4) * CM_LD + wv + n * 8 + g;
            b[n][0] = tf_split(MLSTM ? w0 * vb[0] : vb[0]);
            b[n][1] = tf_split(MLSTM ? w1 * vb[4 * CM_LD] : vb[4 * CM_LD]);
        }
        tf_mma3(d_, a, b);
    }
    // a sum that is not finite again, term by term: the parts' products make a NaN of an infinity
    float all = 0.0f;
#pragma unroll
    for (int m = 0; m < 2; m++)
#pragma unroll
        for (int n = 0; n < 4; n++) all += (acc[m][n][0] + acc[m][n][1]) + (acc[m][n][2] + acc[m][n][3]);
    if (!tf_finite(all)) {
#pragma unroll
        for (int m = 0; m < 2; m++)
#pragma unroll
            for (int n = 0; n < 4; n++)
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    const int d = wd + 16 * m + g + 8 * (e >> 1), v = wv + n * 8 + 2 * t4 + (e & 1);
                    acc[m][n][e] = 0.0f;
#pragma unroll 1
                    for (int r = 0; r < rows; r++) acc[m][n][e] = fmaf(sk[r * CM_LD + d], (MLSTM ? wt[r] : 1.0f) * sv[r * CM_LD + v], acc[m][n][e]);
                }
    }
    float* out = p.before + at * dk * dv;
#pragma unroll
    for (int m = 0; m < 2; m++)
#pragma unroll
        for (int n = 0; n < 4; n++)
#pragma unroll
            for (int u = 0; u < 2; u++) {
                const int d = d0 + wd + 16 * m + g + 8 * u, v = v0 + wv + n * 8 + 2 * t4;
                if (d < dk && v < dv) *reinterpret_cast<float2*>(out + (size_t)d * dv + v) = make_float2(acc[m][n][2 * u], acc[m][n][2 * u + 1]);
            }
    if (MLSTM && v0 == 0 && tid < CM_T && d0 + tid < dk) {
        float s0 = 0.0f, s1 = 0.0f, s2 = 0.0f, s3 = 0.0f;
#pragma unroll 4
        for (int r = 0; r < CM_Q; r += 4) {
            s0 = fmaf(wt[r], sk[r * CM_LD + tid], s0);
            s1 = fmaf(wt[r + 1], sk[(r + 1) * CM_LD + tid], s1);
            s2 = fmaf(wt[r + 2], sk[(r + 2) * CM_LD + tid], s2);
            s3 = fmaf(wt[r + 3], sk[(r + 3) * CM_LD + tid], s3);
        }
        p.n_before[at * dk + d0 + tid] = (s0 + s1) + (s2 + s3);
    }
}

// grid (blocks of 1,024 elements of S, and with MLSTM one more for n; H; segments).  What the chunks add is read eight at a time.
template <bool MLSTM>
__global__ void __launch_bounds__(256) cm_scan_kernel(const CmArgs p) {
    __shared__ int base_sh;
    const int seg = blockIdx.z, h = blockIdx.y, H = p.H, dk = p.dk, dv = p.dv;
    const int first = p.seg_starts[seg], end = p.seg_starts[seg + 1], slot = p.seg_slots[seg];
    if (end - first <= p.from) return;
    if (threadIdx.x < 32) {
        const int b = first_chunk_of<CM_Q>(seg, p.seg_starts, p.from);
        if (threadIdx.x == 0) base_sh = b;
    }
    __syncthreads();
    const int base = base_sh, chunks = (end - first + CM_Q - 1) / CM_Q;
    float* st = slot >= 0 ? p.state + (size_t)slot * p.state_floats : nullptr;
    if (MLSTM && (int)blockIdx.x * 1024 >= (dk * dv + 1023) / 1024 * 1024) {
        const int d = threadIdx.x;
        if (d >= dk) return;
        float* n_st = st ? st + (size_t)H * dk * dv + (size_t)h * dk + d : nullptr;
        float n = n_st ? *n_st : 0.0f;
        for (int c = 0; c < chunks; c++) {
            const size_t at = (size_t)(base + c) * H + h;
            const float add = p.n_before[at * dk + d];
            p.n_before[at * dk + d] = n;
            n = fmaf(p.decay[at], n, add);
        }
        if (n_st) *n_st = n;
        return;
    }
    const int i = (blockIdx.x * 256 + threadIdx.x) * 4;
    if (i >= dk * dv) return;
    float* mine = st ? st + (size_t)h * dk * dv + i : nullptr;      // (a slot need not begin on 16 bytes)
    float4 s = mine ? make_float4(mine[0], mine[1], mine[2], mine[3]) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    constexpr int AHEAD = 8;
    for (int c0 = 0; c0 < chunks; c0 += AHEAD) {
        float4 v[AHEAD];
        float w[AHEAD];
#pragma unroll
        for (int u = 0; u < AHEAD; u++)
            if (c0 + u < chunks) {
                const size_t at = (size_t)(base + c0 + u) * H + h;
                v[u] = *reinterpret_cast<const float4*>(p.before + at * dk * dv + i);
                w[u] = MLSTM ? p.decay[at] : p.decay[at * dk + i / dv];
            }
#pragma unroll
        for (int u = 0; u < AHEAD; u++)
            if (c0 + u < chunks) {
                *reinterpret_cast<float4*>(p.before + ((size_t)(base + c0 + u) * H + h) * dk * dv + i) = s;
                s = make_float4(fmaf(w[u], s.x, v[u].x), fmaf(w[u], s.y, v[u].y), fmaf(w[u], s.z, v[u].z), fmaf(w[u], s.w, v[u].w));
            }
    }
    if (mine) { mine[0] = s.x; mine[1] = s.y; mine[2] = s.z; mine[3] = s.w; }
}

// -- the outputs ----------------------------------------------------------------------------------------------------------------------------------

template <int DKP, int DVP>
struct CmOut {
    static constexpr int LDQ = DKP + 8, LDB = DVP + 4, LDP = CM_Q + 8;
    // floats of a slot: 32 rows of the state or of v, or the chunk's k, or the decays' logarithms
    static constexpr int SLOT = (CM_Q * LDQ > 32 * LDB ? CM_Q * LDQ : 32 * LDB);
    static constexpr int FLOATS = CM_Q * LDQ + 2 * SLOT;
    static_assert(CM_Q * LDP <= CM_Q * LDQ, "the weights take q's place");
};

// grid (chunks, H); 256 threads: warp w has rows 32 (w & 1) .. + 31 and columns (w >> 1) DVP / 4 ..; out [tokens][H dv] in T; gate at gate_off of proj's rows
template <bool MLSTM, int DKP, int DVP, typename T>
__global__ void __launch_bounds__(256, 2) cm_out_kernel(const CmArgs p, int gate_off, const float* __restrict__ norm_w, float eps, T* __restrict__ out) {
    using L = CmOut<DKP, DVP>;
    constexpr int LDQ = L::LDQ, LDB = L::LDB, LDP = L::LDP, NT = DVP / 32, KS = DKP / 32;       // NT: tiles of 8 columns a warp; KS: slices of 32 rows of the state
    extern __shared__ __align__(16) float co_smem[];
    __shared__ int find[4];
    __shared__ float misc[MLSTM ? 10 * CM_Q : 17 * CM_Q];
    __shared__ double sA[MLSTM ? CM_Q : 1], sN[MLSTM ? CM_Q : 1];
    float (*squares)[CM_Q] = reinterpret_cast<float (*)[CM_Q]>(misc);                           // [4][64]
    float (*sums)[CM_Q] = reinterpret_cast<float (*)[CM_Q]>(misc + (MLSTM ? 4 * CM_Q : 0));     // [4][64], mLSTM
    float* row_n = misc + (MLSTM ? 8 * CM_Q : 0);
    float* row_f = misc + (MLSTM ? 9 * CM_Q : 0);
    __shared__ float vec[MLSTM ? DKP : 4 * DKP];        // MLSTM: n before the chunk; else the decays over each 16 tokens
    float* sq = co_smem;
    float* ring = co_smem + CM_Q * LDQ;
    float* sk = ring + L::SLOT;                         // k waits in the second slot
    const Chunk ch = find_chunk<CM_Q>(blockIdx.x, p.seg_starts, p.segments, find, p.from);
    if (ch.seg < 0) return;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t4 = lane & 3, wm = warp & 1, wn = warp >> 1;
    const int h = blockIdx.y, H = p.H, dk = p.dk, dv = p.dv, rows = ch.rows;
    const size_t at = (size_t)blockIdx.x * H + h;
    const float qscale = 1.0f / sqrtf((float)dk);
    const int col0 = wn * (DVP / 4);
    float o[2][NT][4];
    // The second time (where an output came out as no finite number): the outputs term by term, so that a token's NaN or infinity stays out of the tokens before it
    // (a weight of zero times a NaN is one) and an infinity is not made a NaN by its parts.
#pragma unroll 1
    for (bool careful = false;; careful = true) {
        for (int e = tid; e < CM_Q * (DKP / 4); e += 256) {
            const int r = e / (DKP / 4), d = 4 * (e % (DKP / 4));
            const bool on = r < rows && d < dk;
            const float* src = p.proj + (size_t)(ch.first + (on ? r : 0)) * p.N + h * dk + (on ? d : 0);
            copy16_or_zero(sq + r * LDQ + d, src, on);
            copy16_or_zero(sk + r * LDQ + d, src + H * dk, on);
            // the decays' logarithms lie in the first slot until the weights of the chunk are known
            if (!MLSTM) copy16_or_zero(ring + r * LDQ + d, p.logs + (size_t)(ch.first + (on ? r : 0)) * H * dk + h * dk + (on ? d : 0), on);
        }
        tf_commit();
        auto issue = [&](int s) {                           // slice s: 32 rows of the state, then of v
            if (s < KS + 2) {
                float* dst = ring + (s & 1) * L::SLOT;
                for (int e = tid; e < 32 * (DVP / 4); e += 256) {
                    const int r = e / (DVP / 4), v = 4 * (e % (DVP / 4)), row = (s < KS ? s : s - KS) * 32 + r;
                    const bool on = v < dv && row < (s < KS ? dk : rows);
                    const float* src = s < KS ? p.before + (at * dk + row) * dv + v : p.proj + (size_t)(ch.first + row) * p.N + 2 * H * dk + h * dv + v;
                    copy16_or_zero(dst + r * LDB + v, on ? src : p.proj, on);
                }
            }
            tf_commit();
        };
        if (MLSTM) {
            issue(0);
            if (tid < CM_Q) {
                const double mb = p.m_before[at];
                const size_t i = (size_t)(ch.first + (tid < rows ? tid : 0)) * H + h;
                const double Nt = fmax(mb, p.G[i]);
                sA[tid] = tid < rows ? p.A[i] : 0.0;
                sN[tid] = Nt;
                row_f[tid] = expf((float)(mb - Nt));
                row_n[tid] = expf(-(float)(p.F[i] + Nt));   // e^-m
            }
            for (int d = tid; d < DKP; d += 256) vec[d] = d < dk ? p.n_before[at * dk + d] : 0.0f;
            tf_wait<1>();
        } else {
            tf_wait<0>();
        }
        __syncthreads();

        // the chunk's weights, 16 x 16 of them a warp and m: rows 32 wm + 16 m .., columns 16 wn ..
        float w[2][2][4];
#pragma unroll
        for (int m = 0; m < 2; m++)
#pragma unroll
            for (int n = 0; n < 2; n++)
#pragma unroll
                for (int e = 0; e < 4; e++) w[m][n][e] = 0.0f;
        if (!MLSTM) {
            // Pairs inside a piece of 16 tokens by themselves, before q and k are scaled: four threads a row, a quarter of the channels each, walk from the row's
            // token back to the piece's first with the sum of the logarithms so far.
            const float* sl = ring;
            float* sw = misc;                               // [64][17]
            const int r = tid >> 2, p0 = r & ~15;
            float pw[CM_LOCAL];
#pragma unroll
            for (int i = 0; i < CM_LOCAL; i++) pw[i] = 0.0f;
            for (int d = tid & 3; d < DKP; d += 4) {
                float sum = 0.0f;
                const float qv = sq[r * LDQ + d];
#pragma unroll
                for (int j = CM_LOCAL - 1; j >= 0; j--)
                    if (p0 + j <= r) {
                        pw[j] = fmaf(qv * sk[(p0 + j) * LDQ + d], tf_exp2(sum), pw[j]);
                        sum += sl[(p0 + j) * LDQ + d];
                    }
            }
#pragma unroll
            for (int j = 0; j < CM_LOCAL; j++) {
                pw[j] += __shfl_xor_sync(0xffffffffu, pw[j], 1);
                pw[j] += __shfl_xor_sync(0xffffffffu, pw[j], 2);
                if ((tid & 3) == (j & 3)) sw[r * 17 + j] = pw[j];
            }
            __syncthreads();
#pragma unroll
            for (int m = 0; m < 2; m++)
                if (2 * wm + m == wn) {
#pragma unroll
                    for (int n = 0; n < 2; n++)
#pragma unroll
                        for (int e = 0; e < 4; e++) w[m][n][e] = sw[(16 * wn + g + (e >> 1) * 8) * 17 + n * 8 + 2 * t4 + (e & 1)];
                }
            // q times what its piece leaves up to it, k times what its piece leaves behind it, and what the whole pieces leave: a channel of a piece a thread
            for (int e = tid; e < 4 * DKP; e += 256) {
                const int s = e / DKP, d = e % DKP;
                float before = 0.0f, behind = 0.0f;
#pragma unroll
                for (int j = 0; j < CM_LOCAL; j++) {
                    before += sl[(16 * s + j) * LDQ + d];
                    sq[(16 * s + j) * LDQ + d] *= tf_exp2(before);
                }
                vec[e] = tf_exp2(before);
#pragma unroll
                for (int j = CM_LOCAL - 1; j >= 0; j--) {
                    sk[(16 * s + j) * LDQ + d] *= tf_exp2(behind);
                    behind += sl[(16 * s + j) * LDQ + d];
                }
            }
            __syncthreads();
            issue(0);
        }
        // q k^T: MLSTM every pair, else the pairs of different sixteens (q's factor takes what decays between the two)
#pragma unroll
        for (int m = 0; m < 2; m++) {
            const int I = 2 * wm + m;
            if (MLSTM ? wn > I : wn >= I) continue;
#pragma unroll 4
            for (int ks = 0; ks < DKP / 8; ks++) {
                const int d = ks * 8 + 2 * t4;
                const float* qa = sq + (16 * I + g) * LDQ + d;
                float2 x = *reinterpret_cast<const float2*>(qa), y = *reinterpret_cast<const float2*>(qa + 8 * LDQ);
                if (!MLSTM) {
                    float f0 = 1.0f, f1 = 1.0f;
                    for (int u = wn + 1; u < I; u++) { f0 *= vec[u * DKP + d]; f1 *= vec[u * DKP + d + 1]; }
                    x.x *= f0; x.y *= f1; y.x *= f0; y.y *= f1;
                }
                const Tf a[1][4] = {{tf_split(x.x), tf_split(y.x), tf_split(x.y), tf_split(y.y)}};
                Tf b[2][2];
#pragma unroll
                for (int n = 0; n < 2; n++) {
                    const float2 kb = *reinterpret_cast<const float2*>(sk + (16 * wn + n * 8 + g) * LDQ + d);
                    b[n][0] = tf_split(kb.x);
                    b[n][1] = tf_split(kb.y);
                }
                float* const d_[1][2] = {{w[m][0], w[m][1]}};
                tf_mma3(d_, a, b);
            }
        }
        if (MLSTM) {
            float part[2][2] = {{0.0f, 0.0f}, {0.0f, 0.0f}};
#pragma unroll
            for (int m = 0; m < 2; m++)
#pragma unroll
                for (int n = 0; n < 2; n++)
#pragma unroll
                    for (int e = 0; e < 4; e++) {
                        const int r = 32 * wm + 16 * m + g + (e >> 1) * 8, i = 16 * wn + n * 8 + 2 * t4 + (e & 1);
                        w[m][n][e] = (i <= r && i < rows) ? w[m][n][e] * expf((float)(sA[i] - sN[r])) : 0.0f;
                        part[m][e >> 1] += w[m][n][e];
                    }
#pragma unroll
            for (int m = 0; m < 2; m++)
#pragma unroll
                for (int u = 0; u < 2; u++) {
                    float v = part[m][u];
                    v += __shfl_xor_sync(0xffffffffu, v, 1);
                    v += __shfl_xor_sync(0xffffffffu, v, 2);
                    if (t4 == 0) sums[wn][32 * wm + 16 * m + g + u * 8] = v;
                }
            // q . n before the chunk: four threads a row
            const int r = tid >> 2;
            float s = 0.0f;
            for (int d = tid & 3; d < DKP; d += 4) s = fmaf(sq[r * LDQ + d], vec[d], s);
            s += __shfl_xor_sync(0xffffffffu, s, 1);
            s += __shfl_xor_sync(0xffffffffu, s, 2);
            if ((tid & 3) == 0) squares[0][r] = s;          // (until the squares are needed)
        }
        __syncthreads();                                    // nobody reads k any more
        issue(1);
        if (MLSTM && tid < CM_Q) {
            const float nq = fmaf(row_f[tid], squares[0][tid], (sums[0][tid] + sums[1][tid]) + (sums[2][tid] + sums[3][tid])) * qscale;
            row_n[tid] = 1.0f / (fmaxf(fabsf(nq), row_n[tid]) + 1e-6f);
        }
#pragma unroll
        for (int m = 0; m < 2; m++)
#pragma unroll
            for (int n = 0; n < NT; n++)
#pragma unroll
                for (int e = 0; e < 4; e++) o[m][n][e] = 0.0f;
#pragma unroll 1
        for (int s = 0; s < KS + 2; s++) {
            tf_wait<1>();
            __syncthreads();                                // slice s is there
            if (s == KS) {                                  // q with the state is done: the weights take q's place
#pragma unroll
                for (int m = 0; m < 2; m++)
#pragma unroll
                    for (int n = 0; n < 2; n++)
#pragma unroll
                        for (int u = 0; u < 2; u++)
                            *reinterpret_cast<float2*>(sq + (32 * wm + 16 * m + g + u * 8) * LDP + 16 * wn + n * 8 + 2 * t4) =
                                make_float2(w[m][n][2 * u], w[m][n][2 * u + 1]);
                if (MLSTM) {
#pragma unroll
                    for (int m = 0; m < 2; m++) {
                        const float fa = row_f[32 * wm + 16 * m + g], fb = row_f[32 * wm + 16 * m + g + 8];
#pragma unroll
                        for (int n = 0; n < NT; n++) { o[m][n][0] *= fa; o[m][n][1] *= fa; o[m][n][2] *= fb; o[m][n][3] *= fb; }
                    }
                }
                __syncthreads();
            }
            const float* sb = ring + (s & 1) * L::SLOT + col0 + g;
            if (s < KS || 32 * (s - KS) <= 32 * wm + 31) {  // (rows 0..31 do not see tokens 32..63)
                const int lda = s < KS ? LDQ : LDP;
                const float* pa = sq + (32 * wm + g) * lda + (s < KS ? 32 * s : 32 * (s - KS));
                if (careful) {
#pragma unroll 1
                    for (int i = 0; i < 32; i++)
#pragma unroll
                        for (int m = 0; m < 2; m++)
#pragma unroll
                            for (int u = 0; u < 2; u++) {
                                if (s >= KS && 32 * (s - KS) + i > 32 * wm + 16 * m + g + 8 * u) continue;
                                float x = pa[(16 * m + 8 * u) * lda + i];
                                if (!MLSTM && s < KS)
                                    for (int z = 0; z < 2 * wm + m; z++) x *= vec[z * DKP + 32 * s + i];
#pragma unroll
                                for (int n = 0; n < NT; n++)
#pragma unroll
                                    for (int e = 0; e < 2; e++) o[m][n][2 * u + e] = fmaf(x, sb[i * LDB + n * 8 + 2 * t4 - g + e], o[m][n][2 * u + e]);
                            }
                } else
#pragma unroll
                for (int ks = 0; ks < 4; ks++) {
                    Tf a[2][4];
#pragma unroll
                    for (int m = 0; m < 2; m++) {
                        const float* q0 = pa + 16 * m * lda + ks * 8 + 2 * t4;
                        float2 x = *reinterpret_cast<const float2*>(q0), y = *reinterpret_cast<const float2*>(q0 + 8 * lda);
                        if (!MLSTM && s < KS) {
                            const int d = 32 * s + ks * 8 + 2 * t4;
                            float f0 = 1.0f, f1 = 1.0f;
                            for (int u = 0; u < 2 * wm + m; u++) { f0 *= vec[u * DKP + d]; f1 *= vec[u * DKP + d + 1]; }
                            x.x *= f0; x.y *= f1; y.x *= f0; y.y *= f1;
                        }
                        a[m][0] = tf_split(x.x); a[m][1] = tf_split(y.x); a[m][2] = tf_split(x.y); a[m][3] = tf_split(y.y);
                    }
#pragma unroll
                    for (int n = 0; n < NT; n += 2) {
                        Tf b[2][2];
#pragma unroll
                        for (int u = 0; u < 2; u++) {
                            const float* vb = sb + (ks * 8 + 2 * t4) * LDB + (n + u) * 8;
                            b[u][0] = tf_split(vb[0]);
                            b[u][1] = tf_split(vb[LDB]);
                        }
                        float* const d_[2][2] = {{o[0][n], o[0][n + 1]}, {o[1][n], o[1][n + 1]}};
                        tf_mma3(d_, a, b);
                    }
                }
            }
            __syncthreads();
            issue(s + 2);
        }
        // the heads' norm and gate
        bool odd = false;
#pragma unroll
        for (int m = 0; m < 2; m++)
#pragma unroll
            for (int u = 0; u < 2; u++) {
                const int r = 32 * wm + 16 * m + g + u * 8;
                const float f = MLSTM ? qscale * row_n[r] : qscale;
                float ss = 0.0f;
#pragma unroll
                for (int n = 0; n < NT; n++)
#pragma unroll
                    for (int e = 0; e < 2; e++) {
                        o[m][n][2 * u + e] *= f;
                        ss = fmaf(o[m][n][2 * u + e], o[m][n][2 * u + e], ss);
                    }
                ss += __shfl_xor_sync(0xffffffffu, ss, 1);
                ss += __shfl_xor_sync(0xffffffffu, ss, 2);
                if (t4 == 0) squares[wn][r] = ss;
                odd = odd || (r < rows && !tf_finite(ss));
            }
        if (!__syncthreads_or(odd && !careful)) break;
    }
#pragma unroll
    for (int m = 0; m < 2; m++)
#pragma unroll
        for (int u = 0; u < 2; u++) {
            const int r = 32 * wm + 16 * m + g + u * 8;
            if (r >= rows) continue;
            const float inv = 1.0f / sqrtf(((squares[0][r] + squares[1][r]) + (squares[2][r] + squares[3][r])) / (float)dv + eps);
            const float* gate = p.proj + (size_t)(ch.first + r) * p.N + gate_off + (size_t)h * dv;
            T* orow = out + ((size_t)(ch.first + r) * H + h) * dv;
            const float* wrow = MLSTM ? norm_w + h * dv : norm_w;
#pragma unroll
            for (int n = 0; n < NT; n++) {
                const int c = col0 + n * 8 + 2 * t4;
                if (c >= dv) continue;
                const float2 gt = *reinterpret_cast<const float2*>(gate + c);
                const float a = (o[m][n][2 * u] * inv) * wrow[c], b = (o[m][n][2 * u + 1] * inv) * wrow[c + 1];      // (a weight may begin anywhere)
                const float ra = (MLSTM ? a : a * gt.x) / (1.0f + expf(-gt.x)), rb = (MLSTM ? b : b * gt.y) / (1.0f + expf(-gt.y));
                if (sizeof(T) == 2) *reinterpret_cast<__nv_bfloat162*>(orow + c) = __floats2bfloat162_rn(ra, rb);
                else { orow[c] = from_f32<T>(ra); orow[c + 1] = from_f32<T>(rb); }
            }
        }
}

}  // namespace vk

using namespace vk;

static int cm_chunks(int tokens, int segments, int from) { return most_chunks(CM_Q, tokens, segments, from); }
static size_t cm_up(size_t b) { return (b + 255) / 256 * 256; }

static size_t gla_decays_smem(int rank) { return (size_t)CM_LOCAL * rank * sizeof(float); }

// Whether the chunked kernels take these sizes: heads of up to 128 x 256 values in whole 16-byte pieces of the product's rows (N floats), and a decays' narrow half
// (rank values; none: 0) of which gla_chunk_decays has 16 tokens in the 48 KB that a block may have without asking, its own four numbers among them.
VK_API int vk_memory_chunked_takes(int N, int dk, int dv, int rank) {
    return N % 4 == 0 && dk > 0 && dk % 4 == 0 && dk <= 128 && dv > 0 && dv % 4 == 0 && dv <= 256 && rank >= 0 && gla_decays_smem(rank) + 4 * sizeof(int) <= 48 * 1024;
}

// (from: as for the kernels; the larger it is, the fewer chunks a step of many segments can have, each with a head's whole state)
VK_API size_t vk_mlstm_chunked_scratch_bytes(int tokens, int segments, int H, int dk, int dv, int from) {
    const size_t chunks = cm_chunks(tokens, segments, from);
    return cm_up(chunks * H * dk * dv * 4) + cm_up(chunks * H * dk * 4) + 2 * cm_up(chunks * H * 8) + 4 * cm_up((size_t)tokens * H * 8);
}
VK_API size_t vk_gla_chunked_scratch_bytes(int tokens, int segments, int H, int dk, int dv, int from) {
    const size_t chunks = cm_chunks(tokens, segments, from);
    return cm_up(chunks * H * dk * dv * 4) + cm_up(chunks * H * dk * 4) + cm_up((size_t)tokens * H * dk * 4);
}

template <bool MLSTM, int DK, int DV, typename T>
static int cm_launch_out(const CmArgs& p, int tokens, int gate_off, const float* norm_w, float eps, void* out, cudaStream_t stream) {
    auto kern = cm_out_kernel<MLSTM, DK, DV, T>;
    const int smem = CmOut<DK, DV>::FLOATS * (int)sizeof(float);
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return (int)e;
    return launch_plain(kern, dim3(cm_chunks(tokens, p.segments, p.from), p.H), dim3(256), smem, stream, p, gate_off, norm_w, eps, (T*)out);
}

template <bool MLSTM>
static int cm_launch(const CmArgs& p, int tokens, int gate_off, const float* norm_w, float eps, void* out, int dtype, cudaStream_t stream) {
    auto add = cm_add_kernel<MLSTM>;
    const int smem = CM_Q * CM_LD * (MLSTM ? 2 : 3) * (int)sizeof(float);
    const cudaError_t e = cudaFuncSetAttribute(add, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return (int)e;
    const int col_tiles = (p.dv + CM_T - 1) / CM_T, row_tiles = (p.dk + CM_T - 1) / CM_T;
    int s = launch_plain(add, dim3(cm_chunks(tokens, p.segments, p.from), p.H, row_tiles * col_tiles), dim3(128), smem, stream, p, col_tiles);
    if (s != VK_OK) return s;
    s = launch_plain(cm_scan_kernel<MLSTM>, dim3((p.dk * p.dv + 1023) / 1024 + (MLSTM ? 1 : 0), p.H, p.segments), dim3(256), 0, stream, p);
    if (s != VK_OK) return s;
#define GO(DK, DV)                                                                                                                       \
    return dtype == 0 ? cm_launch_out<MLSTM, DK, DV, float>(p, tokens, gate_off, norm_w, eps, out, stream)                               \
                      : cm_launch_out<MLSTM, DK, DV, __nv_bfloat16>(p, tokens, gate_off, norm_w, eps, out, stream)
    if (p.dk <= 64) {
        if (p.dv <= 64) GO(64, 64);
        if (p.dv <= 128) GO(64, 128);
        GO(64, 256);
    }
    if (p.dv <= 64) GO(128, 64);
    if (p.dv <= 128) GO(128, 128);
    GO(128, 256);
#undef GO
}

static int cm_check(const CmArgs& p, int gate_off, const void* out, const void* scratch) {
    if (p.H <= 0 || gate_off < 0 || gate_off % 2 || gate_off + p.H * p.dv > p.N || !vk_memory_chunked_takes(p.N, p.dk, p.dv, 0)) return VK_BAD_SHAPE;
    if (p.H > 65535 || p.segments > 65535) return VK_TOO_LARGE;
    if ((uintptr_t)p.proj % 16 || (uintptr_t)out % 4 || (uintptr_t)scratch % 16) return VK_BAD_ALIGNMENT;
    return VK_OK;
}

static CmArgs cm_args(const float* proj, int N, int H, int dk, int dv, const int32_t* seg_starts, const int32_t* seg_slots, float* state, void* scratch, int segments, int from) {
    CmArgs p = {};
    p.proj = proj; p.N = N; p.H = H; p.dk = dk; p.dv = dv; p.segments = segments; p.from = from;
    p.seg_starts = seg_starts; p.seg_slots = seg_slots; p.state = state; p.before = (float*)scratch;
    return p;
}

// proj, state and norm as for vk_mlstm_recurrence and vk_mlstm_gate; out [tokens][H dv] in dtype; four kernels.  Segments of up to `from` tokens are left alone: their
// states and their rows of out are for the token-by-token kernels.
VK_API int vk_mlstm_chunked(const float* proj, int N, int H, int dk, int dv, const float* gate_bias, float cap, int gate_off, const float* norm_w, float eps,
                            const int32_t* seg_starts, const int32_t* seg_slots, float* state, void* scratch, void* out, int tokens, int segments, int from,
                            int dtype, cudaStream_t stream) {
    if (segments <= 0 || tokens <= 0) return VK_OK;
    CmArgs p = cm_args(proj, N, H, dk, dv, seg_starts, seg_slots, state, scratch, segments, from);
    if (from < 0 || !(cap > 0.0f) || N < 2 * H * dk + 2 * H * dv + 2 * H) return VK_BAD_SHAPE;
    int s = cm_check(p, gate_off, out, scratch);
    if (s != VK_OK) return s;
    const size_t chunks = cm_chunks(tokens, segments, from), tok = cm_up((size_t)tokens * H * 8);
    char* at = (char*)scratch + cm_up(chunks * H * dk * dv * 4);
    p.state_floats = (size_t)H * dk * dv + (size_t)H * dk + H;
    p.n_before = (float*)at; at += cm_up(chunks * H * dk * 4);
    p.m_before = (double*)at; at += cm_up(chunks * H * 8);
    p.decay = (float*)at; at += cm_up(chunks * H * 8);
    p.A = (double*)at; at += tok;
    p.G = (double*)at; at += tok;
    p.F = (double*)at; at += tok;
    p.weight = (float*)at;
    s = launch_plain(mlstm_chunk_gates_kernel, dim3(H, segments), dim3(MG_THREADS), 0, stream, p, gate_bias, cap);
    if (s != VK_OK) return s;
    return cm_launch<true>(p, tokens, gate_off, norm_w, eps, out, dtype, stream);
}

// proj, decays and state as for vk_gla_prepare and vk_gla_recurrence, norm and gate as for vk_gla_gate; four kernels.
VK_API int vk_gla_chunked(const float* proj, int N, int H, int dk, int dv, int a_off, int rank, const float* a2t, const float* bias, float tau, int gate_off,
                          const float* norm_w, float eps, const int32_t* seg_starts, const int32_t* seg_slots, float* state, void* scratch, void* out,
                          int tokens, int segments, int from, int dtype, cudaStream_t stream) {
    if (segments <= 0 || tokens <= 0) return VK_OK;
    CmArgs p = cm_args(proj, N, H, dk, dv, seg_starts, seg_slots, state, scratch, segments, from);
    if (from < 0 || rank <= 0 || a_off < 0 || a_off + rank > N || !(tau > 0.0f) || N < 2 * H * dk + H * dv) return VK_BAD_SHAPE;
    const size_t smem = gla_decays_smem(rank);
    if (!vk_memory_chunked_takes(N, dk, dv, rank)) return VK_BAD_SHAPE;
    int s = cm_check(p, gate_off, out, scratch);
    if (s != VK_OK) return s;
    const int chunks = cm_chunks(tokens, segments, from);
    p.state_floats = (size_t)H * dk * dv;
    p.decay = (float*)((char*)scratch + cm_up((size_t)chunks * H * dk * dv * 4));
    p.logs = (float*)((char*)p.decay + cm_up((size_t)chunks * H * dk * 4));
    s = launch_plain(gla_chunk_decays_kernel, dim3(4 * chunks, (H * dk + GD_THREADS - 1) / GD_THREADS), dim3(GD_THREADS), smem, stream, p, a_off, rank, a2t, bias,
                         1.0f / tau);
    if (s != VK_OK) return s;
    return cm_launch<false>(p, tokens, gate_off, norm_w, eps, out, dtype, stream);
}
