// Causal attention of prompt portions over the paged cache on the fifth-generation tensor cores, keys and values of 64 or 128 values (bfloat16):
// softmax(q k^T * scale) v with float32 scores, running maxima and sums (the softmax of engine/src/model.c:932-956, computed tile by tile).
//
// A block takes a tile of up to 128 consecutive tokens of one request and one query head, and walks over the request's keys 64 at a time from absolute
// position 0 (or the window's first step).
//
//   GROUPS x 4 warps  the softmax, a thread a query row: group g takes the steps i with i mod GROUPS = g: 64 scores out of tensor memory, mask, maximum, 2^x, and
//              the probabilities as a high and a low bfloat16 part (p = hi + lo to about 2^-17, so that P V matches float32 probabilities) back into the
//              columns that the scores came from
//   one warp   TMA: the query tile once, and the keys, two stages of 64 at a time, straight from the pages (a box of one page's rows for one key-value head,
//              128-byte swizzle); another warp the values
//   one warp   tcgen05.mma, scores: S[128 x 64] = Q K^T into one of BUFS buffers in tensor memory, as soon as the product that read it last is done
//   one warp   tcgen05.mma, O[128 x VD] += P V in the order of the steps, P from tensor memory, the values as they lie in the cache (N-major)
//
// The tensor core cuts off what a sum in tensor memory has no bits for, every time that it adds to it; the form for launches of few blocks and long walks has two
// outputs, even and odd steps', which halves the products that are added to one.  (9 heads, 4,096 tokens: 8,187 of 2,359,296 results rounded to the wrong
// bfloat16 with one output, 6,533 with two.)
//
// O stays in tensor memory for the whole walk, and all groups share it and a row's reference maximum.  The maximum is only raised when a step's exceeds it by more
// than 2^8 (then the warp scales its rows of O, once every earlier product has landed); until then the probabilities are taken against the older maximum and may
// reach 256, which float32 sums and the two bfloat16 parts hold as well as values up to 1.  Every step settles the maximum for the next: a row's thread leaves it for
// the row's thread of the next group, in one word of shared memory with the step's number, long before its probabilities are done.  The groups' sums are added at
// the end, and the result is normalised.
//
// Why this form.  What a step cannot do without are 64 exponentials a row (512 cycles of the special-function units for 128 rows) and its products (450 cycles at
// VD = 64: an instruction of 128 x 64 x 16 takes 48 cycles with both operands in shared memory and 32 with P in tensor memory, if the issuing warp's operands are in
// uniform registers).  A step's own chain (scores, softmax, P V, each with a hand-over of 150 to 250 cycles) is 2,900 cycles, so steps must overlap, in a block
// and between two blocks.  32 heads, 8,192 tokens (275 GFLOP and, with the low parts, half as much again): 618 us with 32 keys a thread and the probabilities through
// shared memory (13 instructions a score, most of them waits and meetings of a row's two threads); 612 us with 128 keys a step, two groups with an output of their own
// and no overlap inside a block; 483 us with four blocks of one group; 442 us here (two groups, two blocks).  2,048 tokens: 62 -> 47 us; a mixed step of 15 heads (1,301
// tokens in three portions) 29.3 -> 21.3; 16 heads of 128 x 128, 2,048 tokens, a window of 1,024: 46 -> 37.
//
// In a launch with few blocks (a portion of a few hundred tokens far into a context) a long walk is cut: a block takes at most AP_PART steps of its tile (part p of a
// tile is steps 16p .. 16p+15 from the tile's first), so that more multiprocessors share the work.  A tile with one part is finished by its block; otherwise every part
// leaves its unnormalised output, reference maxima and sums in scratch memory, and the part that arrives last (a counter per tile and head, no waiting) adds them in
// part order and writes the result.
//
// A row's result does not depend on the other rows: its keys are walked in 64s from absolute position 0 (or the window's first tile), parts lie at fixed
// steps of that walk, and every decision above is the row's own.  What the launcher chooses by the size of the whole launch, the form (over how many groups a row's
// sum is added up, over how many outputs its products are) and whether walks are cut, does move its last bits.
//
// Every wait is bounded (see tcgen05_common.cuh); a thread that gave up keeps its appointments.
//
// tiles [n_tiles][4] int32: first token (flat index), rows (1..128), position of the first token, segment.
#include <cstdlib>

#include "tcgen05_common.cuh"

namespace vk {

constexpr int AP_BM = 128, AP_BN = 64;
constexpr int AP_PART = 16;          // steps of 64 keys a block walks at most, where walks are cut

// A form of the kernel: keys of HD and values of VD values (64 or 128), GROUPS groups of four softmax warps, BUFS buffers of scores and probabilities in tensor
// memory, STAGES of keys and of values in shared memory, BLOCKS a multiprocessor, OUTS outputs in tensor memory that the steps' products go to in turn.
template <int HD_, int VD_, int GROUPS_, int BUFS_, int STAGES_, int BLOCKS_, int OUTS_ = 1>
struct ApForm {
    static constexpr int HD = HD_, VD = VD_, GROUPS = GROUPS_, BUFS = BUFS_, STAGES = STAGES_, BLOCKS = BLOCKS_, OUTS = OUTS_;
    static constexpr int KP = HD / 64, VP = VD / 64;            // panels of 64 columns: rows of 128 bytes each
    static constexpr int SOFT = 4 * GROUPS, THREADS = 32 * (SOFT + 4);
    static constexpr uint32_t PANEL = AP_BN * 128, Q_PANEL = AP_BM * 128, Q_BYTES = KP * Q_PANEL, K_BYTES = KP * PANEL, V_BYTES = VP * PANEL;
    static constexpr uint32_t K_OFF = Q_BYTES, V_OFF = K_OFF + STAGES * K_BYTES, BAR_OFF = V_OFF + STAGES * V_BYTES, SMEM = BAR_OFF + 512 + 1024;
    static constexpr uint32_t O_COL = BUFS * AP_BN, O_END = O_COL + OUTS * VD, TMEM = O_END <= 128 ? 128 : O_END <= 256 ? 256 : 512;
    static_assert((HD == 64 || HD == 128) && (VD == 64 || VD == 128) && O_END <= 512 && TMEM * BLOCKS <= 512, "tensor memory");
    // A thread waits on a barrier's phases by parity, so it must never be two phases behind: a group takes every GROUPS-th step, a buffer every BUFS-th.
    static_assert(STAGES >= BUFS && BUFS >= GROUPS, "phases");
};

// A row's reference maximum (the low half) and the number of the step that settled it, in one 64-bit word of shared memory, stored and loaded as one scalar: nothing
// else orders the two halves (to the memory model a vector access is an access for each component).
__device__ __forceinline__ void ap_settle(unsigned long long* at, int step, float m) {
    asm volatile("{\n\t.reg .b64 w;\n\tmov.b64 w, {%1, %2};\n\tst.volatile.shared.b64 [%0], w;\n\t}" ::"r"(smem_u32(at)), "r"(__float_as_uint(m)), "r"(step) : "memory");
}
__device__ __forceinline__ bool ap_settled(const unsigned long long* at, int step, float& m, unsigned long long limit) {
    const uint32_t addr = smem_u32(at);
    long long start = 0;
    for (int tries = 0;; tries++) {
        uint32_t v, s;
        asm volatile("{\n\t.reg .b64 w;\n\tld.volatile.shared.b64 w, [%2];\n\tmov.b64 {%0, %1}, w;\n\t}" : "=r"(v), "=r"(s) : "r"(addr) : "memory");
        if ((int)s == step) { m = __uint_as_float(v); return true; }
        if (tries == 0) start = clock64();
        else if ((tries & 15) == 0 && (unsigned long long)(clock64() - start) > limit) return false;
    }
}

// Bounded wait for two barriers' phases at once (of an issuing warp: two waits one after another, of which each takes a hundred cycles and more when it is over
// already, were half of its time for a step).
__device__ __forceinline__ bool ap_wait_both(uint64_t* a, uint32_t parity_a, uint64_t* b, uint32_t parity_b, unsigned long long limit) {
    const uint32_t at_a = smem_u32(a), at_b = smem_u32(b);
    long long start = 0;
    for (int tries = 0;; tries++) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p, q;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %5;\n\tmbarrier.try_wait.parity.shared::cta.b64 q, [%3], %4, %5;\n\t"
            "and.pred p, p, q;\n\tselp.b32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(at_a), "r"(parity_a & 1), "r"(at_b), "r"(parity_b & 1), "r"(20000u)
            : "memory");
        if (__all_sync(0xffffffffu, done)) return true;
        if (tries == 0) start = clock64();
        else if (__any_sync(0xffffffffu, (unsigned long long)(clock64() - start) > limit)) return false;
    }
}

// Scratch of the parts: outputs [tiles][heads][parts][128][64] float32, then maxima and sums [tiles][heads][parts][128][2],
// then counters [tiles][heads] (zero before the first launch; the kernel leaves them zero).
struct ApScratch {
    float* part_o;
    float* part_ml;
    int* counters;
    int parts;                       // parts a tile can have in this launch (the grid's width is tiles * parts)
    int part_steps;                  // steps of a part (AP_PART; an experiment may set another through VITNA_ATT_PART)
    int n_tiles;
};

__device__ __forceinline__ float ap_ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ uint32_t ap_pack(float lo, float hi) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
}
// Two float32 values an instruction.
__device__ __forceinline__ uint64_t ap_two(float a, float b) {
    uint64_t v;
    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(a), "f"(b));
    return v;
}
__device__ __forceinline__ void ap_split2(uint64_t v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ uint64_t ap_fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t v;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(v) : "l"(a), "l"(b), "l"(c));
    return v;
}
__device__ __forceinline__ uint64_t ap_add2(uint64_t a, uint64_t b) {
    uint64_t v;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(v) : "l"(a), "l"(b));
    return v;
}
__device__ __forceinline__ float ap_max3(float a, float b, float c) {
    float v;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(v) : "f"(a), "f"(b), "f"(c));
    return v;
}
__device__ __forceinline__ float ap_largest32(const uint32_t* s) {
    float m[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
    for (int j = 0; j < 32; j += 8)
#pragma unroll
        for (int u = 0; u < 4; u++) m[u] = ap_max3(m[u], __uint_as_float(s[j + 2 * u]), __uint_as_float(s[j + 2 * u + 1]));
    return fmaxf(ap_max3(m[0], m[1], m[2]), m[3]);
}
__device__ __forceinline__ void ap_tmem_st16(uint32_t taddr, const uint32_t* r) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
                 ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]),
                 "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
                 : "memory");
}
// A box of one page's rows: column x, row y of the page's keys (or values), page z.
__device__ __forceinline__ void ap_load_page(void* dst, const CUtensorMap* map, int x, int y, int z, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
        ::"r"(smem_u32(dst)), "l"(map), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z)
        : "memory");
}
// The low word of a descriptor of an N-major operand whose columns lie in panels of 64: the panels' distance is its leading byte offset.
__device__ __forceinline__ uint32_t ap_desc_lo_panels(uint32_t smem_addr, uint32_t panel_bytes) { return ((smem_addr & 0x3FFFF) >> 4) | ((panel_bytes >> 4) << 16); }
// The product with the first operand in tensor memory (128 lanes, two bfloat16 values a column).
__device__ __forceinline__ void ap_umma_ts(uint32_t d, uint32_t a, uint32_t b_lo, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 db;\n\tmov.b64 db, {%2, %5};\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], db, %3, p;\n\t}"
        ::"r"(d), "r"(a), "r"(b_lo), "r"(idesc), "r"(accumulate), "r"(UMMA_DESC_HI_SW128));
}

template <typename F>
__global__ void __launch_bounds__(F::THREADS, F::BLOCKS) attention_prefill_tcgen05_kernel(
    const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v,
    const int32_t* __restrict__ block_tables, const int32_t* __restrict__ tiles, __nv_bfloat16* __restrict__ out, int nh, int nkv, int page_size, int max_blocks,
    float scale, int window, int out_ld, const float* __restrict__ gate, int gate_ld, const WaitCtl wc, const ApScratch sc) {
    constexpr int HD = F::HD, VD = F::VD, GROUPS = F::GROUPS, BUFS = F::BUFS, STAGES = F::STAGES, SOFT = F::SOFT, OUTS = F::OUTS, OUT = VD / GROUPS;
    constexpr float RAISE = 8.0f;                    // the reference maximum follows when a maximum exceeds it by 2^8
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint64_t* q_full = reinterpret_cast<uint64_t*>(smem + F::BAR_OFF);
    uint64_t* k_full = q_full + 1;
    uint64_t* k_empty = k_full + STAGES;
    uint64_t* v_full = k_empty + STAGES;
    uint64_t* v_empty = v_full + STAGES;
    uint64_t* s_full = v_empty + STAGES;             // [BUFS]: a step's scores lie in buffer step mod BUFS
    uint64_t* p_full = s_full + BUFS;                // [BUFS]: its probabilities do
    uint64_t* pv_done = p_full + BUFS;               // [BUFS]: their product with the values has been added into O
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(pv_done + BUFS);
    __shared__ int failed, is_last;
    __shared__ unsigned long long settled[AP_BM];    // a row's reference maximum (log2 units, the low word) and the step that settled it
    __shared__ float l_row[GROUPS][AP_BM];           // at the end the groups' sums

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // Blocks in the order of their tiles, last tile first, all heads and parts of a tile together: later tiles of a prompt walk over more keys, and a launch
    // ends sooner when its longest blocks start first.
    const int per_tile = sc.parts * nh;
    const int tile = sc.n_tiles - 1 - blockIdx.x / per_tile, part = (blockIdx.x % per_tile) / nh;
    const int h = blockIdx.x % nh, kvh = h / (nh / nkv);
    const int tok0 = tiles[tile * 4 + 0], rows = tiles[tile * 4 + 1], pos0 = tiles[tile * 4 + 2], seg = tiles[tile * 4 + 3];
    const int last_pos = pos0 + rows - 1;
    const int lo_first = (window > 0 && pos0 - window + 1 > 0) ? pos0 - window + 1 : 0;     // lowest key any row needs
    const int kt_first = lo_first / AP_BN, kt1 = last_pos / AP_BN;                          // the tile's walk: key steps kt_first .. kt1
    const int n_parts = (kt1 - kt_first) / sc.part_steps + 1;
    if (part >= n_parts) return;                                                            // the whole block: nothing to do
    const int kt0 = kt_first + part * sc.part_steps, n_it = min(sc.part_steps, kt1 - kt0 + 1);      // this block's steps: kt0 .. kt0 + n_it - 1

    if (threadIdx.x == 0) {
        failed = 0;
        mbar_init(q_full, 1);
        for (int s = 0; s < STAGES; s++) { mbar_init(&k_full[s], 1); mbar_init(&k_empty[s], 1); mbar_init(&v_full[s], 1); mbar_init(&v_empty[s], 1); }
        for (int b = 0; b < BUFS; b++) { mbar_init(&s_full[b], 1); mbar_init(&p_full[b], 4); mbar_init(&pv_done[b], 1); }      // p_full: one arrival a warp of the group
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (threadIdx.x < AP_BM) settled[threadIdx.x] = ~0ull;              // step -1
    if (warp == SOFT + 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(F::TMEM) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    auto got = [&](uint64_t* bar, int parity, int code) -> bool {
        if (__all_sync(0xffffffffu, mbar_wait(bar, (uint32_t)parity & 1, wc.cycles))) return true;
        if (lane == 0) give_up(wc.error, &failed, code);
        return false;
    };

    if (warp == SOFT || warp == SOFT + 3) {
        // ---- the copies: one warp the query tile and the keys, one the values ----------------------------------------------------------------------------
        const bool values = warp == SOFT + 3;
        uint64_t *full = values ? v_full : k_full, *empty = values ? v_empty : k_empty;
        uint8_t* ring = smem + (values ? F::V_OFF : F::K_OFF);
        const CUtensorMap* map = values ? &map_v : &map_k;
        const int panels = values ? F::VP : F::KP;
        const uint32_t stage_bytes = values ? F::V_BYTES : F::K_BYTES;
        if (!values && lane == 0) {
            mbar_expect_tx(q_full, F::Q_BYTES);
            for (int p = 0; p < F::KP; p++) tma_load_2d(smem + p * F::Q_PANEL, &map_q, h * HD + 64 * p, tok0, q_full);      // rows beyond the batch read as zero
        }
        const int32_t* bt = block_tables + (size_t)seg * max_blocks;
        const int box_rows = page_size < AP_BN ? page_size : AP_BN, boxes = AP_BN / box_rows;
        // Two steps at a time, lane b the box b of the two.  (A step at a time, the wait for its stage and what surrounds the copies took 1,000 cycles a step and paced
        // launches whose blocks have a multiprocessor to themselves.)  The pages come from the block table 32 at a time (lane l the l-th page from the batch's
        // first), a batch ahead of their use, and are handed round by shuffle.  A batch's steps lie in 32 pages whatever page they begin in.
        const int batch_steps = (31 * page_size / AP_BN) & ~1, last_page = last_pos / page_size;      // >= 2: pages hold at least 8 keys
        auto load_batch = [&](int i0) -> int {
            const int p0 = ((kt0 + i0) * AP_BN) / page_size;
            return (i0 < n_it && p0 + lane <= last_page) ? bt[p0 + lane] : 0;
        };
        int pages_now = load_batch(0), pages_next = load_batch(batch_steps), batch_first = 0, batch_page0 = (kt0 * AP_BN) / page_size;
        const int which = lane / boxes, box = lane - which * boxes;
        for (int i = 0; i < n_it; i += 2) {
            if (i - batch_first == batch_steps) {
                batch_first = i;
                batch_page0 = (kt0 + i) * AP_BN / page_size;
                pages_now = pages_next;
                pages_next = load_batch(i + batch_steps);
            }
            const int my = i + which, s = my % STAGES, key0 = (kt0 + my) * AP_BN, my_page_index = (key0 + box * box_rows) / page_size;
            const int page = __shfl_sync(0xffffffffu, pages_now, (my_page_index - batch_page0) & 31);
            // boxes that hold a key some row needs; the rows of the others are never counted (p = 0) and the values' rows beyond the last position are zeroed
            // by the softmax warps
            const int nb = which < 2 && my < n_it ? min((last_pos - key0) / box_rows + 1, boxes) : 0;
            const int row = kvh * page_size + key0 + box * box_rows - my_page_index * page_size;
            bool ok = true;
            if (i >= STAGES && i + 1 < n_it) ok = ap_wait_both(&empty[i % STAGES], i / STAGES - 1, &empty[(i + 1) % STAGES], (i + 1) / STAGES - 1, wc.cycles);
            else if (i >= STAGES) ok = __all_sync(0xffffffffu, mbar_wait(&empty[i % STAGES], (uint32_t)(i / STAGES - 1) & 1, wc.cycles));
            else if (i + 1 >= STAGES && i + 1 < n_it) ok = __all_sync(0xffffffffu, mbar_wait(&empty[(i + 1) % STAGES], (uint32_t)((i + 1) / STAGES - 1) & 1, wc.cycles));
            if (!ok) { if (lane == 0) give_up(wc.error, &failed, values ? 19 : 11); break; }
            const bool on = nb > 0 && (values || my != wc.skip_stage);          // (a step named by wc.skip_stage gets no keys: a test of the give-up path)
            if (on && box == 0) mbar_expect_tx(&full[s], (uint32_t)(nb * box_rows * panels) * 128);
            __syncwarp();
            if (on && box < nb)
                for (int p = 0; p < panels; p++) ap_load_page(ring + s * stage_bytes + p * F::PANEL + box * box_rows * 128, map, 64 * p, row, page, &full[s]);
        }
    } else if (warp == SOFT + 1) {
        // ---- tensor core: the scores, up to BUFS steps ahead of P V ----------------------------------------------------------------------------------------
        const uint32_t idesc = umma_idesc_bf16(AP_BM, AP_BN), q_lo = umma_desc_lo(smem_u32(smem)), k_lo0 = umma_desc_lo(smem_u32(smem + F::K_OFF));
        if (got(q_full, 0, 12)) {
            int b = 0, use = 0;                      // buffer i mod BUFS, i / BUFS
            for (int i = 0; i < n_it; i++) {
                const int s = i % STAGES;
                // the scores take the place of probabilities that the tensor core has read
                if (!(use > 0 ? ap_wait_both(&k_full[s], i / STAGES, &pv_done[b], use - 1, wc.cycles) : got(&k_full[s], i / STAGES, 13))) {
                    if (lane == 0) give_up(wc.error, &failed, 13);
                    break;
                }
                tc_fence_after();
                if (elect_one()) {
#pragma unroll
                    for (int k = 0; k < HD / 16; k++)
                        umma_bf16_lo(tmem + b * AP_BN, q_lo + (k / 4) * (F::Q_PANEL >> 4) + 2 * (k % 4), k_lo0 + s * (F::K_BYTES >> 4) + (k / 4) * (F::PANEL >> 4) + 2 * (k % 4),
                                     idesc, k != 0);
                    umma_commit(&s_full[b]);
                    umma_commit(&k_empty[s]);        // the keys' stage is free once these instructions have read it
                }
                __syncwarp();
                if (++b == BUFS) { b = 0; use++; }
            }
        }
    } else if (warp == SOFT + 2) {
        // ---- tensor core, the other issuer: P V in the order of the steps ----------------------------------------------------------------------------------
        const uint32_t idesc = umma_idesc_bf16(AP_BM, VD) | (1u << 16), v_lo0 = ap_desc_lo_panels(smem_u32(smem + F::V_OFF), F::PANEL);      // (the values are N-major)
        int b = 0, use = 0;
        for (int i = 0; i < n_it; i++) {
            const int s = i % STAGES;
            if (!ap_wait_both(&v_full[s], i / STAGES, &p_full[b], use, wc.cycles)) {
                if (lane == 0) give_up(wc.error, &failed, 14);
                break;
            }
            tc_fence_after();
            if (elect_one()) {
                // 16 keys an instruction: two groups of eight 128-byte rows of the values; 32 columns hold 32 keys' high parts, then their low parts
                const uint32_t v_lo = v_lo0 + s * (F::V_BYTES >> 4), p_at = tmem + b * AP_BN, o_at = tmem + F::O_COL + i % OUTS * VD;
#pragma unroll
                for (int k = 0; k < AP_BN / 16; k++) ap_umma_ts(o_at, p_at + 32 * (k / 2) + 8 * (k % 2), v_lo + k * (2048 >> 4), idesc, i >= OUTS || k != 0);
#pragma unroll
                for (int k = 0; k < AP_BN / 16; k++) ap_umma_ts(o_at, p_at + 32 * (k / 2) + 16 + 8 * (k % 2), v_lo + k * (2048 >> 4), idesc, 1);
                umma_commit(&pv_done[b]);
                umma_commit(&v_empty[s]);
            }
            __syncwarp();
            if (++b == BUFS) { b = 0; use++; }
        }
    } else {
        // ---- softmax: a thread a query row ---------------------------------------------------------------------------------------------------------------
        const int g = warp >> 2, quarter = warp & 3, r = threadIdx.x & (AP_BM - 1);
        const bool valid = r < rows;
        const int my_pos = min(pos0 + r, last_pos);      // (rows beyond the tile's own do as its last one does and are not written: no step is masked for them)
        const int my_lo = (window > 0 && my_pos - window + 1 > 0) ? my_pos - window + 1 : 0;
        const float scale_log2 = scale * 1.4426950408889634f;
        const uint32_t lanes = tmem + ((uint32_t)(quarter * 32) << 16), my_o = lanes + F::O_COL;
        // the first keys of the steps that every row of the warp counts whole: plain_from .. plain_to
        const int row0 = quarter * 32, plain_to = min(pos0 + row0, last_pos) - (AP_BN - 1), plain_from = window > 0 ? min(pos0 + row0 + 31, last_pos) - window + 1 : 0;
        float m = -INFINITY, l = 0.0f;              // the row's reference maximum (log2 units) and its sum against it
        // A failed wait ends the walk; the warp then only keeps its appointments, so that nobody waits for it without a limit.
        int i = g, b = g, use = 0;                  // step, its buffer i mod BUFS, i / BUFS
        bool lost = false;
        for (; i < n_it; i += GROUPS) {
            const int key0 = (kt0 + i) * AP_BN;
            const uint32_t my_s = lanes + b * AP_BN;
            if (!got(&s_full[b], use, 15)) break;
            tc_fence_after();
            // The loops below go over 32 scores at a time and are not unrolled, and the scores are read from tensor memory twice (first for their maximum): what
            // a thread needs are few registers.
            //
            // Raw scores: the maximum commutes with the (positive) scale; masked keys become -inf only in steps that touch the diagonal or the window's edge.
            if (key0 > plain_to || key0 < plain_from) {
#pragma unroll 1
                for (int c = 0; c < AP_BN; c += 32) {
                    const int lo_j = my_lo - key0 - c, hi_j = my_pos - key0 - c;      // of these keys the row counts lo_j .. hi_j
                    uint32_t sr[32];
                    tmem_ld32(my_s + c, sr);
                    tmem_loaded(sr);
#pragma unroll
                    for (int j = 0; j < 32; j++)
                        if (j < lo_j || j > hi_j) sr[j] = 0xff800000u;
                    tmem_st32(my_s + c, sr);
                }
                tmem_wait_st();
            }
            float mx;
            {
                uint32_t s0[32], s1[32];
                tmem_ld32_nowait(my_s, s0);
                tmem_ld32_nowait(my_s + 32, s1);
                tmem_wait_ld();
                tmem_loaded(s0);
                tmem_loaded(s1);
                mx = fmaxf(ap_largest32(s0), ap_largest32(s1)) * scale_log2;
            }
            // The group before has settled its step's reference maximum: a row's thread there has left it for the row's thread here, in one word with the step's
            // number.  (A barrier's arrival and wait a step, in the place of this word, were a chain of 1,000 cycles a step through all groups.)
            float had = mx;                         // (O is written, not added to, by the first product)
            if (i > 0 && !ap_settled(&settled[r], i - 1, had, wc.cycles)) {
                give_up(wc.error, &failed, 23);
                lost = true;
            }
            if (__any_sync(0xffffffffu, lost)) break;
            const bool raise = mx > had + RAISE;    // also the first counted key after none (had = -inf)
            const float now = raise ? mx : had;
            ap_settle(&settled[r], i, now);         // (what comes of it for O is done before this step's probabilities are told, and the next step's product follows theirs)
            if (__any_sync(0xffffffffu, raise)) {
                // scale this warp's rows of O to the new maxima; every earlier product must have landed
                if (!got(&pv_done[b == 0 ? BUFS - 1 : b - 1], b == 0 ? use - 1 : use, 17)) break;
                tc_fence_after();
                const float alpha = raise ? ap_ex2(had - mx) : 1.0f;
#pragma unroll 1
                for (int c = 0; c < OUTS * VD; c += 16) {       // (an output that no product has been added to yet is written whole by its first)
                    uint32_t orr[16];
                    tmem_ld16(my_o + c, orr);
#pragma unroll
                    for (int j = 0; j < 16; j++) orr[j] = __float_as_uint(__uint_as_float(orr[j]) * alpha);
                    ap_tmem_st16(my_o + c, orr);
                }
                tmem_wait_st();
                tc_fence_before();
            }
            if (now != m) {                         // the sum so far, against the new maximum (there is none yet while m = -inf)
                l *= ap_ex2(m - now);
                m = now;
            }
            const float m_use = m == -INFINITY ? 0.0f : m;
            const uint64_t scale2 = ap_two(scale_log2, scale_log2), shift2 = ap_two(-m_use, -m_use), minus = ap_two(-1.0f, -1.0f);
            uint64_t sum2 = ap_two(0.0f, 0.0f);
#pragma unroll 1
            for (int c = 0; c < AP_BN; c += 32) {
                uint32_t sr[32], hi[16], lo[16];
                tmem_ld32(my_s + c, sr);
                tmem_loaded(sr);
#pragma unroll
                for (int j = 0; j < 32; j += 2) {
                    float x0, x1, p0, p1, r0, r1;
                    ap_split2(ap_fma2(ap_two(__uint_as_float(sr[j]), __uint_as_float(sr[j + 1])), scale2, shift2), x0, x1);
                    const uint64_t p = ap_two(ap_ex2(x0), ap_ex2(x1));
                    sum2 = ap_add2(sum2, p);
                    ap_split2(p, p0, p1);
                    const uint32_t hp = ap_pack(p0, p1);
                    ap_split2(ap_fma2(ap_two(__uint_as_float(hp << 16), __uint_as_float(hp & 0xffff0000u)), minus, p), r0, r1);
                    hi[j / 2] = hp;
                    lo[j / 2] = ap_pack(r0, r1);
                }
                ap_tmem_st16(my_s + c, hi);         // 32 columns of scores become 16 of high and 16 of low parts
                ap_tmem_st16(my_s + c + 16, lo);
            }
            float sum0, sum1;
            ap_split2(sum2, sum0, sum1);
            l += sum0 + sum1;
            // the values' rows beyond the last position (pages not loaded, slots not yet written): never counted, but 0 * garbage must not be NaN
            if (kt0 + i == kt1 && (last_pos & (AP_BN - 1)) != AP_BN - 1) {
                if (!got(&v_full[i % STAGES], i / STAGES, 22)) break;       // the values have landed
                const int z0 = (last_pos & (AP_BN - 1)) + 1;
                uint8_t* vs = smem + F::V_OFF + (i % STAGES) * F::V_BYTES;
                for (int idx = r; idx < (AP_BN - z0) * 8; idx += AP_BM)
                    for (int p = 0; p < F::VP; p++) *reinterpret_cast<uint4*>(vs + p * F::PANEL + (z0 + idx / 8) * 128 + (idx & 7) * 16) = make_uint4(0, 0, 0, 0);
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");       // the zeros are for the tensor core
            }
            tmem_wait_st();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_plain(&p_full[b]);
            b += GROUPS;
            if (b >= BUFS) { b -= BUFS; use++; }
        }
        bool ok = i >= n_it;
        __syncwarp();
        for (; i < n_it; i += GROUPS)
            if (lane == 0) mbar_arrive_plain(&p_full[i % BUFS]);
        // the end: every group is through, its sums against the last maxima are added; a group takes its share of the columns
        asm volatile("bar.sync 1, %0;" ::"n"(SOFT * 32) : "memory");
        ok = ok && got(&pv_done[(n_it - 1) % BUFS], (n_it - 1) / BUFS, 18);
        const float last = __uint_as_float((uint32_t)settled[r]);
        if (last != m) l *= ap_ex2(m - last);       // (a group without a step has l = 0 and m = -inf)
        m = last;
        l_row[g][r] = l;
        asm volatile("bar.sync 1, %0;" ::"n"(SOFT * 32) : "memory");
        l = l_row[0][r];
#pragma unroll
        for (int j = 1; j < GROUPS; j++) l += l_row[j][r];
        tc_fence_after();
        const size_t first = ((size_t)tile * nh + h) * sc.parts, slot = first + part;
        const int c = g * OUT;
        __nv_bfloat16* dst = out + (size_t)(tok0 + r) * out_ld + (size_t)h * VD + c;
        auto write = [&](int d0, const float* a, float inv) {            // 16 columns
#pragma unroll
            for (int d = 0; d < 16; d += 8) {
                uint4 v;
                v.x = ap_pack(a[d] * inv, a[d + 1] * inv);
                v.y = ap_pack(a[d + 2] * inv, a[d + 3] * inv);
                v.z = ap_pack(a[d + 4] * inv, a[d + 5] * inv);
                v.w = ap_pack(a[d + 6] * inv, a[d + 7] * inv);
                *reinterpret_cast<uint4*>(dst + d0 + d) = v;
            }
        };
        if (ok) {
            float inv = valid ? 1.0f / l : 0.0f;
            if (gate && valid) inv = gated(inv, gate, gate_ld, tok0 + r, h);
#pragma unroll 1
            for (int d0 = 0; d0 < OUT; d0 += 16) {
                uint32_t o[16];
                float acc[16];
                __syncwarp();
                tmem_ld16(my_o + c + d0, o);
#pragma unroll
                for (int d = 0; d < 16; d++) acc[d] = __uint_as_float(o[d]);
#pragma unroll
                for (int u = 1; u < OUTS; u++) {
                    if (u >= n_it) break;
                    tmem_ld16(my_o + u * VD + c + d0, o);
#pragma unroll
                    for (int d = 0; d < 16; d++) acc[d] += __uint_as_float(o[d]);
                }
                if (valid && n_parts == 1) write(d0, acc, inv);
                if (valid && n_parts > 1) {
                    // this part's unnormalised output, reference maximum and sum; a row without a counted key in this part (its keys all lie in earlier
                    // parts) leaves maximum -inf and nothing else
                    float* po = sc.part_o + (slot * AP_BM + r) * VD + c + d0;
#pragma unroll
                    for (int d = 0; d < 16; d += 4) *reinterpret_cast<float4*>(po + d) = make_float4(acc[d], acc[d + 1], acc[d + 2], acc[d + 3]);
                    if (c + d0 == 0) *reinterpret_cast<float2*>(sc.part_ml + (slot * AP_BM + r) * 2) = make_float2(m, l);
                }
            }
        }
        if (n_parts > 1) {
            // The softmax threads meet; thread 0's counting releases the block's partial and acquires the others'.  (A block whose wait ran out counts too,
            // so that the counter returns to zero; the error word says that the result is not valid.)
            asm volatile("bar.sync 1, %0;" ::"n"(SOFT * 32) : "memory");
            if (threadIdx.x == 0) {
                int* counter = sc.counters + (size_t)tile * nh + h;
                int old;
                asm volatile("atom.acq_rel.gpu.global.add.s32 %0, [%1], 1;" : "=r"(old) : "l"(counter) : "memory");
                is_last = old == n_parts - 1;
                if (is_last) *counter = 0;          // ready for the next launch
            }
            asm volatile("bar.sync 1, %0;" ::"n"(SOFT * 32) : "memory");
            if (is_last && valid) {
                // parts in part order: running maximum, weights 2^(part's maximum - maximum), sum, output
#pragma unroll 1
                for (int d0 = 0; d0 < OUT; d0 += 16) {
                    float mm = -INFINITY, ll = 0.0f, acc[16];
#pragma unroll
                    for (int d = 0; d < 16; d++) acc[d] = 0.0f;
#pragma unroll 1
                    for (int j = 0; j < n_parts; j++) {
                        const float2 pm = __ldcg(reinterpret_cast<const float2*>(sc.part_ml + ((first + j) * AP_BM + r) * 2));
                        if (pm.x == -INFINITY) continue;
                        const float cm = fmaxf(mm, pm.x);
                        const float keep = mm == -INFINITY ? 0.0f : ap_ex2(mm - cm), w = ap_ex2(pm.x - cm);
                        const float4* src = reinterpret_cast<const float4*>(sc.part_o + ((first + j) * AP_BM + r) * VD + c + d0);
                        ll = ll * keep + pm.y * w;
#pragma unroll
                        for (int d = 0; d < 16; d += 4) {
                            const float4 v = __ldcg(src + d / 4);
                            acc[d] = acc[d] * keep + v.x * w; acc[d + 1] = acc[d + 1] * keep + v.y * w;
                            acc[d + 2] = acc[d + 2] * keep + v.z * w; acc[d + 3] = acc[d + 3] * keep + v.w * w;
                        }
                        mm = cm;
                    }
                    write(d0, acc, 1.0f / ll);      // (no gate: the launches that have one do not cut their walks)
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == SOFT + 1) {
        if (failed) __nanosleep(200000);             // after a failed wait: let copies in flight land
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(F::TMEM) : "memory");
    }
}

// A [rows, cols] bfloat16 matrix with row stride ld (elements), read in boxes of box_rows x 64 columns, 128-byte swizzle.
static bool ap_make_map(CUtensorMap* map, const void* base, long long rows, int cols, long long ld, int box_rows) {
    EncodeTiledFn enc = encode_tiled();
    if (!enc) return false;
    cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
    cuuint32_t box[2] = {64u, (cuuint32_t)box_rows};
    cuuint32_t elem[2] = {1, 1};
    return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
               CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// The rows of `dim` values (keys or values) of every page: [pages][rows of a page][dim], pages page_elems elements apart, read in boxes of box_rows x 64 columns.
static bool ap_make_page_map(CUtensorMap* map, const void* base, int dim, int page_rows, long long pages, long long page_elems, int box_rows) {
    EncodeTiledFn enc = encode_tiled();
    if (!enc) return false;
    cuuint64_t dims[3] = {(cuuint64_t)dim, (cuuint64_t)page_rows, (cuuint64_t)pages};
    cuuint64_t strides[2] = {(cuuint64_t)dim * 2, (cuuint64_t)page_elems * 2};
    cuuint32_t box[3] = {64u, (cuuint32_t)box_rows, 1u};
    cuuint32_t elem[3] = {1, 1, 1};
    return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
               CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <typename F>
static int launch_ap(const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mv, const int32_t* block_tables, const int32_t* tiles, void* out, int nh, int nkv,
                     int page_size, int max_blocks, float scale, int window, int out_ld, const float* gate, int gate_ld, int* error, const ApScratch& sc,
                     cudaStream_t stream) {
    auto kern = attention_prefill_tcgen05_kernel<F>;
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)F::SMEM);
    if (e != cudaSuccess) return (int)e;
    // (an ordinary launch: started under programmatic dependent launch, with the kernel after it fetching its weights
    // meanwhile, a 2,048-token prompt at the 135M sizes took 2.90 instead of 2.72 ms)
    return launch_plain(kern, dim3(sc.n_tiles * sc.parts * nh), dim3(F::THREADS), F::SMEM, stream, mq, mk, mv, block_tables, tiles, (__nv_bfloat16*)out, nh, nkv, page_size,
                        max_blocks, scale, window, out_ld, gate, gate_ld, wait_ctl(error, WAIT_FAMILY_ATTENTION_PREFILL), sc);
}

}  // namespace vk

using namespace vk;

// Which form a launch for heads of 64 takes: 0 two groups and two blocks a multiprocessor, 1 four groups and one block, 2 (default) by the size of the launch, 3 one
// group and three blocks.
static int g_prefill_streams_mode = -1;
static int prefill_streams_mode() {
    if (g_prefill_streams_mode < 0) {
        const char* e = getenv("VITNA_ATT_STREAMS");
        g_prefill_streams_mode = e ? (atoi(e) == 3 ? 3 : atoi(e) ? 1 : 0) : 2;
    }
    return g_prefill_streams_mode;
}
// Returns the mode that was in force.
VK_API int vk_set_prefill_streams(int mode) {
    const int was = prefill_streams_mode();
    if (mode >= 0 && mode <= 3) g_prefill_streams_mode = mode;
    return was;
}

// How a launch for heads of 64 is worked out: the steps of a part, the parts that a tile can have, and the softmax groups of the form (1, 2 or 4).
struct ApPlan {
    int part_steps, parts, groups;
};
static ApPlan ap_plan(int n_tiles, int nh, int window, int grid_context) {
    // Walks are cut only when the launch has fewer blocks than three quarters of the multiprocessors (a portion of a few
    // hundred tokens far into a context): measured, a part costs about five key steps of set-up, meeting and adding
    // up, which a whole prompt's launch (a block or more a multiprocessor already) does not win back.
    // VITNA_ATT_PART=n (n >= 16) cuts every launch into parts of n steps, for measurements.
    static const int forced = [] { const char* e = getenv("VITNA_ATT_PART"); const int v = e ? atoi(e) : 0; return v >= AP_PART ? v : 0; }();
    const bool cut = forced || (long long)n_tiles * nh * 4 <= (long long)148 * 3;
    const int part_steps = forced ? forced : cut ? AP_PART : (1 << 24);      // never below AP_PART: the scratch is laid out for that
    // The steps of the longest walk that a tile can have.  Under a window its rows' keys lie within window + 126 positions of each other: without that bound a window's cut
    // launch had blocks for parts that no tile reaches, and real ones came to lie two on a multiprocessor (20 heads, 4 portions of 128 behind 3,000 tokens, window 256: 14.1 -> 17.0 us).
    const int steps = (grid_context - 1) / AP_BN + 1;
    const int walk = window > 0 ? (int)min((long long)steps, ((long long)window + AP_BM - 2) / AP_BN + 2) : steps;
    const int parts = cut ? (walk - 1) / part_steps + 1 : 1;
    // Which form.
    //   Two groups and two blocks a multiprocessor where there are blocks for it: 32 heads and 8,192 / 2,048 tokens (2,048 and 512 blocks) 442 / 47 us against 529 / 56 with
    //     four groups in one block; and for short walks in few blocks, which end before four groups have begun (a window of 64, 300 tokens of 9 heads 9.9 against 10.4).
    //   Four groups, and two outputs, where a block has a multiprocessor to itself, or two or three share one for a long walk: 9 heads and 2,048 tokens (144 blocks) 25.3
    //     against 27.3, 2,600 (189) 30.7 against 34.2, 4,096 (288) 49.1 against 53.3; 100 tokens 6,000 into a context (nine blocks, cut) 25.2 against 29.1.  From 297 to 369
    //     blocks two groups are 13 % the faster and their one output rounds 25 % more results to the wrong bfloat16: the two outputs' sums are worth that.
    //   One group and three blocks for many blocks of walks that have nothing to overlap inside a block: 32 heads and 32 portions of 16 tokens 20.9 us with the kernel
    //     before, 24.1 with two groups, 18.6 with one; three and four steps in more than 600 blocks 1.06 and 0.91 of that kernel's time.
    // VITNA_ATT_STREAMS=0 / 1 / 3 in the environment, or vk_set_prefill_streams, forces one (tests, measurements).
    const int mode = prefill_streams_mode();
    const long long blocks = (long long)n_tiles * parts * nh;
    const int groups = mode != 2 ? (mode == 3 ? 1 : mode == 1 ? 4 : 2) : walk <= 4 && blocks > 296 ? 1 : walk > 8 && blocks < 370 ? 4 : 2;
    return {part_steps, parts, groups};
}
// For tests: the groups of the form that such a launch takes, and 16 times the parts that a tile can have.
VK_API int vk_attention_prefill_plan(int n_tiles, int nh, int window, int grid_context) {
    const ApPlan p = ap_plan(n_tiles, nh, window, grid_context);
    return p.groups + 16 * p.parts;
}

// Bytes of scratch for launches of up to cap_tiles tiles whose contexts reach max_context positions: the parts' outputs,
// their maxima and sums, and the counters, in that order, each 256-byte aligned.
VK_API size_t vk_attention_prefill_tcgen05_scratch_bytes(int cap_tiles, int nh, int max_context) {
    const size_t parts = (size_t)((max_context - 1) / AP_BN) / AP_PART + 1;
    auto up = [](size_t b) { return (b + 255) / 256 * 256; };
    return up((size_t)cap_tiles * nh * parts * AP_BM * 64 * 4) + up((size_t)cap_tiles * nh * parts * AP_BM * 2 * 4) +
           up((size_t)cap_tiles * nh * 4);
}

// q [n_tokens, nh*hd] bfloat16; cache [pages][2][nkv][page_size][hd] bfloat16 (one layer); tiles [n_tiles][4] with up to 128
// rows a tile; out as q.  hd = 64; page_size a multiple of 8 that divides 64 or is a multiple of it.
// scratch: vk_attention_prefill_tcgen05_scratch_bytes(cap_tiles, nh, max_context) bytes whose counters part (the last) was
// zero before the first launch; cap_tiles and max_context fix its layout; grid_context (<= max_context) bounds every
// position + 1 of this launch and sizes the grid (a captured graph keeps it).
// error: a word the kernel sets (non-zero) if a bounded wait ran out.  VK_BAD_SHAPE for what this kernel does not take.
VK_API int vk_attention_prefill_tcgen05(const void* q, const void* cache, const int32_t* block_tables, const int32_t* tiles, void* out,
                                        int n_tokens, int n_tiles, int pages, int nh, int nkv, int hd, int page_size, int max_blocks,
                                        float scale, int window, void* scratch, int cap_tiles, int max_context, int grid_context,
                                        int* error, cudaStream_t stream) {
    if (n_tiles <= 0) return VK_OK;
    if (nh <= 0 || nkv <= 0 || nh % nkv != 0 || page_size <= 0 || max_blocks <= 0 || window < 0 || n_tokens <= 0 || pages <= 0 || !error ||
        !scratch || max_context <= 0 || grid_context <= 0 || grid_context > max_context)
        return VK_BAD_SHAPE;
    if (hd != 64 || page_size % 8 != 0 || (AP_BN % page_size != 0 && page_size % AP_BN != 0)) return VK_BAD_SHAPE;
    if (nh > 65535 || n_tiles > cap_tiles) return VK_TOO_LARGE;
    const long long cache_rows = (long long)pages * 2 * nkv * page_size;
    if (cache_rows >= (1ll << 31)) return VK_TOO_LARGE;
    if (((uintptr_t)q % 16) || ((uintptr_t)cache % 16) || ((uintptr_t)out % 16) || ((uintptr_t)scratch % 16)) return VK_BAD_ALIGNMENT;
    const int box_rows = page_size < AP_BN ? page_size : AP_BN;
    CUtensorMap mq;
    if (!ap_make_map(&mq, q, n_tokens, nh * hd, (long long)nh * hd, AP_BM)) return VK_BAD_SHAPE;
    const size_t max_parts = (size_t)((max_context - 1) / AP_BN) / AP_PART + 1;
    auto up = [](size_t b) { return (b + 255) / 256 * 256; };
    ApScratch sc;
    sc.part_o = (float*)scratch;
    sc.part_ml = (float*)((char*)scratch + up((size_t)cap_tiles * nh * max_parts * AP_BM * 64 * 4));
    sc.counters = (int*)((char*)sc.part_ml + up((size_t)cap_tiles * nh * max_parts * AP_BM * 2 * 4));
    const ApPlan plan = ap_plan(n_tiles, nh, window, grid_context);
    sc.part_steps = plan.part_steps;
    sc.parts = plan.parts;
    sc.n_tiles = n_tiles;
    if ((long long)n_tiles * sc.parts * nh > 0x7fffffffll) return VK_TOO_LARGE;
    CUtensorMap mk, mv;
    const long long page_elems = 2ll * nkv * page_size * hd;
    if (!ap_make_page_map(&mk, cache, hd, nkv * page_size, pages, page_elems, box_rows) ||
        !ap_make_page_map(&mv, (const __nv_bfloat16*)cache + (size_t)nkv * page_size * hd, hd, nkv * page_size, pages, page_elems, box_rows))
        return VK_BAD_SHAPE;
#define GO(...) \
    return launch_ap<ApForm<__VA_ARGS__>>(mq, mk, mv, block_tables, tiles, out, nh, nkv, page_size, max_blocks, scale, window, nh * hd, nullptr, 0, error, sc, stream)
    if (plan.groups == 4) GO(64, 64, 4, 5, 5, 1, 2);
    if (plan.groups == 1) GO(64, 64, 1, 1, 2, 3);
    GO(64, 64, 2, 3, 4, 2);
#undef GO
}

// The same for keys of hd and values of vd values, one of them 128 and the other 64 or 128 (a page holds its keys [nkv][page_size][hd], then its values
// [nkv][page_size][vd]); rows of out are out_ld elements apart; gate float32 [n_tokens][gate_ld] or null: head h of token t times sigmoid(gate[t][h]).  Walks are not
// cut and there is no scratch.  Up to 148 blocks have a multiprocessor each: four groups (97 to 193 KB of shared memory).  More than that share them: two groups and two
// blocks.  Four groups / two, of the time that the kernel before them took: 149 to 296 blocks, walks of 5 and 6 steps (windows of up to 256) 1.09 / 0.81 (64 x 128), 1.04 / 0.76
// (128 x 64), 1.07 / 0.82 (128 x 128), of 41 steps and more 0.68 / 0.72, 0.73 / 0.67, 0.64 / 0.67; above 600 blocks 1.20 / 0.81, - and 1.09 / 0.75, 0.83 / 0.73 and 0.64 / 0.63.  In up to
// 148 blocks walks of up to 6 steps are at 0.90 to 1.12 with four groups (0.92 to 1.15 with two), longer ones at 0.56 to 0.92 (0.64 to 1.09).
VK_API int vk_attention_prefill_tcgen05_dims(const void* q, const void* cache, const int32_t* block_tables, const int32_t* tiles, void* out, int n_tokens, int n_tiles,
                                             int pages, int nh, int nkv, int hd, int vd, int page_size, int max_blocks, float scale, int window, int out_ld,
                                             const float* gate, int gate_ld, int* error, cudaStream_t stream) {
    if (n_tiles <= 0) return VK_OK;
    if (nh <= 0 || nkv <= 0 || nh % nkv != 0 || page_size <= 0 || max_blocks <= 0 || window < 0 || n_tokens <= 0 || pages <= 0 || !error) return VK_BAD_SHAPE;
    if (page_size % 8 != 0 || (AP_BN % page_size != 0 && page_size % AP_BN != 0) || out_ld < nh * vd || out_ld % 8 != 0) return VK_BAD_SHAPE;
    if (nh > 65535 || (long long)n_tiles * nh > 0x7fffffffll || (long long)nkv * page_size >= (1ll << 31)) return VK_TOO_LARGE;
    if (((uintptr_t)q % 16) || ((uintptr_t)cache % 16) || ((uintptr_t)out % 16)) return VK_BAD_ALIGNMENT;
    CUtensorMap mq, mk, mv;
    const int box_rows = page_size < AP_BN ? page_size : AP_BN;
    const long long page_elems = (long long)nkv * page_size * (hd + vd);
    if (!ap_make_map(&mq, q, n_tokens, nh * hd, (long long)nh * hd, AP_BM) || !ap_make_page_map(&mk, cache, hd, nkv * page_size, pages, page_elems, box_rows) ||
        !ap_make_page_map(&mv, (const __nv_bfloat16*)cache + (size_t)nkv * page_size * hd, vd, nkv * page_size, pages, page_elems, box_rows))
        return VK_BAD_SHAPE;
    ApScratch sc = {};
    sc.parts = 1;
    sc.part_steps = 1 << 24;
    sc.n_tiles = n_tiles;
    const bool two = (long long)n_tiles * nh > 148;
#define GO(...) \
    return launch_ap<ApForm<__VA_ARGS__>>(mq, mk, mv, block_tables, tiles, out, nh, nkv, page_size, max_blocks, scale, window, out_ld, gate, gate_ld, error, sc, stream)
    if (hd == 128 && vd == 128) { if (two) GO(128, 128, 2, 2, 2, 2); GO(128, 128, 4, 5, 5, 1); }
    if (hd == 64 && vd == 128) { if (two) GO(64, 128, 2, 2, 3, 2); GO(64, 128, 4, 5, 5, 1); }
    if (hd == 128 && vd == 64) { if (two) GO(128, 64, 2, 3, 3, 2); GO(128, 64, 4, 5, 5, 1); }
#undef GO
    return VK_BAD_SHAPE;
}
