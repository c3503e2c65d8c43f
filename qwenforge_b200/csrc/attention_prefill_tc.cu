// Causal grouped-query flash attention for spans of new tokens over the paged cache on the fifth-generation tensor
// cores (tcgen05), bf16, head sizes 64 and 128. Same contract as the mma.sync kernel of attention_prefill.cu: the
// span's own keys are in the cache already, a query at position p sees keys max(0, p - window + 1) <= j <= p.
//
// A tile is 128 consecutive query tokens of one (sequence, query head). A block serves two tiles of one kv head that see
// the same keys: two query heads of the group on the same tokens, and where the heads run out the next 128 tokens. It
// walks the keys in blocks of two pages (128 keys), keys and values fetched once for both tiles by tiled copies (two
// stages each), and keeps four matrices in tensor memory: per tile the scores S [128 x 128] and the output O [128 x D].
//   warps 0-3, 4-7   a tile's rows, a thread each (lane = row): load the row of S, maximum, base-2 exponentials, sum without
//                    exchange between threads; the weights go back to tensor memory as bf16 over the scores, where the
//                    tensor cores read them as the left operand
//   warp 8           issues the products: O += P V of a tile as soon as its weights are written, then S = Q K^T of its next
//                    block when that product is done (the scores overwrite the weights it reads)
//   warp 9           issues the copies
// While one tile's products run, the other tile's rows are at their exponentials: a block of keys costs 16,384 of them a
// tile, 1,024 cycles of the SM's special-function units, and as many cycles of products at D = 128, so the two alternate.
// O stays in tensor memory. The exponentials of a row are taken against a reference maximum that is only moved when the
// true maximum has grown by more than 2^8 since (weights stay below 256, well inside bf16 and float32); only then does the
// warp rescale its rows of O (load, multiply, store), with no product on them in flight. Numerator and denominator
// carry the same reference, so the quotient at the end is unchanged.
// What bounds it: the chain scores -> exponentials -> product of a tile, of which two tiles overlap. (With one tile of 128
// rows and 64 keys a turn per block, two or three blocks per SM, weights through shared memory, a turn's hand-overs cost more
// than its work: 22% of the special-function rate, 32% of the tensor cores'.) Measured so and now, microseconds: one prompt of
// 8,192 tokens, 28 heads of 128: 856, 449 (1,072 TFLOP/s); 1,024 tokens behind 15,360, 16 heads of 128: 268, 144; one prompt of
// 4,096 tokens, 14 heads of 64: 89, 64. (At head size 64 many tiles are done first in the small blocks of
// attention_prefill_page.cuh: `launch` chooses.) Masked keys cost nothing behind the comparison (their score is
// -infinity), three-way maxima and two-way multiply-adds and additions take 640 instructions a row and turn to 400, and a warp
// arrives once for its rows: 642 -> 1,072 TFLOP/s together. (A quarter or half of the exponentials by a polynomial on the
// multiply-add pipe, and the exponentials of 16 to 64 weights laid out one after another, made no difference.)
// There is no block-wide barrier inside the loop: rows and issuers hand over through shared-memory barriers. Every wait on
// a barrier is bounded: a wait that runs out sets QF_ERR_COPY_TIMEOUT and ends the thread's loop, and the block still frees
// its tensor memory and returns. No copy uses cluster multicast.
// Few tiles of many pages leave SMs without a block. With SPLIT > 1 that many blocks (a cluster) share their tiles: each takes
// every SPLIT-th block of keys, and at the end each brings a slice of the output's columns together: the others pass their sums
// of that slice, and their rows' reference maxima and sums, through distributed shared memory (column by column, so that a
// warp's 32 rows make one 128-byte store).
#include <cooperative_groups.h>

#include "tcgen05.cuh"

// The largest of three: one instruction.
__device__ __forceinline__ float max3(float a, float b, float c) {
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

#define TA_BM 128              // rows of a tile
// (also of attention_prefill_page.cuh)
#define TA_BK 128              // keys of a turn: two pages

#include "attention_prefill_page.cuh"

template <int D, int SPLIT, int PER>
__global__ void __launch_bounds__(128 * PER + 64, 1)
prefill_tc_kernel(const __grid_constant__ CUtensorMap q_map, const __grid_constant__ CUtensorMap kv_map,
                  bf16* __restrict__ out, const int* __restrict__ cu_q, const int* __restrict__ tok_pos,
                  const int* __restrict__ slots, KvSite<bf16> site, int n_heads, int n_seqs, float scale_log2, int window,
                  int* err, const float* __restrict__ sinks, int planes) {
    constexpr int CB = D / 64;                    // blocks of 64 columns in a row of Q, K or V
    constexpr int Q_BLOCK = TA_BM * 128;          // bytes of one [128][64] block of Q
    constexpr int KV_BLOCK = TA_BK * 128;         // bytes of one [128][64] block of two pages' keys or values
    constexpr int PAGE_BYTES = QF_PAGE * 128;     // one page's part of it
    constexpr int Q_BYTES = CB * Q_BLOCK, KV_BYTES = CB * KV_BLOCK;
    constexpr uint32_t TMEM_COLS = 256 * PER, O_COL = 128 * PER;   // S (and P) of tile t in columns 128 t .., O behind them
    constexpr int PRODUCTS = 4 * PER, COPIES = 4 * PER + 1;         // the issuing warps
    extern __shared__ unsigned char smem_unaligned[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_unaligned) + 1023) & ~(uintptr_t)1023);
    unsigned char* q_s = smem;                          // [PER][CB][128][64]
    unsigned char* k_s = q_s + PER * Q_BYTES;             // [2][CB][128][64]
    unsigned char* v_s = k_s + 2 * KV_BYTES;            // [2][CB][128][64]
    // SPLIT > 1: what the cluster's other blocks send, over Q and the stages, which are free when all have left their loops (the
    // first barrier of the cluster below): [SPLIT][PER][DS][128] sums of this block's columns, [SPLIT][PER][2][128] references and sums
    constexpr int DS = D / SPLIT;                       // columns of the output that a block of the cluster brings together
    float* merge_s = reinterpret_cast<float*>(smem);
    float* merge_ml = merge_s + SPLIT * PER * DS * TA_BM;
    const int rank = (int)(blockIdx.x % SPLIT);
    __shared__ __align__(8) uint64_t bar_q, bar_k[2], bar_v[2], bar_k_free[2], bar_v_free[2], bar_s[2], bar_p[2], bar_pv[2], bar_end;
    __shared__ uint32_t tmem_base_s;

    // Which pair of tiles this block serves (PER 1: which single tile): those further down a prompt walk more keys, so they come first.
    const int unit = (int)(blockIdx.x / SPLIT), units = (int)(gridDim.x / SPLIT);
    const int per_pair = site.kv_heads * n_seqs, group = n_heads / site.kv_heads;
    const int pair = units / per_pair - 1 - unit / per_pair, kvh = (unit % per_pair) % site.kv_heads, seq = (unit % per_pair) / site.kv_heads;
    // Launched as a programmatic dependent: what a block works out and sets up before its first copy (its tiles, the barriers, its
    // tensor memory) runs under the tail of the kernel before, which wrote the queries and the new keys and values; they are
    // read, and the output written, only after the wait. The kernel after it may start when every block has its tensor memory (or has ended).
    const int q_begin = cu_q[seq], q_len = cu_q[seq + 1] - q_begin;
    const int tiles_here = (q_len + TA_BM - 1) / TA_BM * group;   // of this sequence and kv head; tile n: head n % group, rows n / group
    if (PER * pair >= tiles_here) return;
    const int slot = slots[seq];
    const int warp = threadIdx.x >> 5, t = PER == 2 && warp < 8 ? warp >> 2 : 0, row = threadIdx.x & 127;   // row threads: tile t, row `row`
    const int q_width = n_heads * D;
    int row0[2], head[2], n_rows[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const int tile = PER * pair + i;
        row0[i] = tile / group * TA_BM, head[i] = kvh * group + tile % group;
        n_rows[i] = i < PER && tile < tiles_here ? min(TA_BM, q_len - row0[i]) : 0;
    }
    const int my_row0 = t ? row0[1] : row0[0], my_head = t ? head[1] : head[0], my_rows = t ? n_rows[1] : n_rows[0];
    bf16* out_row = out + (size_t)(q_begin + my_row0 + row) * q_width + (size_t)my_head * D;
    if (slot < 0) {  // padding entry: defined output, no cache access
        grid_dependency_wait();
        if (warp < PRODUCTS && row < my_rows)
            for (int c = 0; c < D; c += 8) *reinterpret_cast<uint4*>(out_row + c) = make_uint4(0, 0, 0, 0);
        return;
    }
    // The first tile's rows are never behind the second's. Blocks of keys: two pages from page p_first on; this block takes
    // every SPLIT-th of them, tile i the first turns[i] of those.
    const int pos_first = tok_pos[q_begin + row0[0]];   // position of the first tile's first row; positions run on from there
    const int p_first = (window > 0 ? max(0, pos_first - window + 1) : 0) / QF_PAGE;
    int turns[2], p_lo[2], p_end[2];   // (p_lo, p_end: the pages that any row of the tile sees)
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const int pos = pos_first + row0[i] - row0[0], last = pos + n_rows[i] - 1;
        p_lo[i] = (window > 0 ? max(0, pos - window + 1) : 0) / QF_PAGE;
        p_end[i] = n_rows[i] > 0 ? last / QF_PAGE + 1 : 0;
        const int blocks = p_end[i] > p_first ? (p_end[i] - p_first + 1) / 2 : 0;
        turns[i] = blocks > rank ? (blocks - rank + SPLIT - 1) / SPLIT : 0;
    }
    const int all_turns = max(turns[0], turns[1]), p_last = max(p_end[0], p_end[1]) - 1;
    // What lies in a page that none of a tile's rows sees is not multiplied by their weights of zero (0 times infinity is not 0): the
    // second page behind the last, or behind the other tile's window. A second tile's first turn may have no page left.
    const bool first_empty = rank == 0 && p_lo[1] >= p_first + 2;

    if (threadIdx.x == 0) {
        mbar_init(&bar_q, 1);
        mbar_init(&bar_end, 1);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            mbar_init(&bar_k[i], 1);
            mbar_init(&bar_v[i], 1);
            mbar_init(&bar_k_free[i], 1);
            mbar_init(&bar_v_free[i], 1);
            mbar_init(&bar_s[i], 1);
            mbar_init(&bar_p[i], TA_BM / 32);
            mbar_init(&bar_pv[i], 1);
        }
    }
    if (warp == PRODUCTS) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&tmem_base_s)), "r"(TMEM_COLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    grid_launch_dependents();
    grid_dependency_wait();
    const uint32_t tmem = tmem_base_s;
    bool timed_out = false;
    float m_ref = QF_NEG_BIG, l_run = 0.f;  // row threads: the reference maximum of the exponentials, and their sum
    // A warp waits as one: the loads and stores of tensor memory and the choice of the issuing lane are collective, so
    // the lanes of a warp must leave their loop together if a wait runs out.
    auto wait_all = [&](uint64_t* bar, uint32_t parity) { return __all_sync(0xffffffffu, mbar_wait(bar, parity)) != 0; };

    if (warp == COPIES) {
        // ---- the copies. All lanes run the loop (uniform values); one lane issues.
        const bool leader = elect_one();
        const int* table_row = site.table + (long long)slot * site.table_stride;
        if (all_turns > 0 && leader) {
            mbar_expect_tx(&bar_q, (n_rows[1] > 0 ? 2 : 1) * Q_BYTES);
#pragma unroll
            for (int i = 0; i < 2; ++i)
                if (n_rows[i] > 0)
#pragma unroll
                    for (int cb = 0; cb < CB; ++cb)
                        tma_load_2d(q_s + i * Q_BYTES + cb * Q_BLOCK, &q_map, head[i] * D + cb * 64, q_begin + row0[i], &bar_q);
        }
        __syncwarp();
        int keys = 0, values = 0;   // turns whose copies have been asked for
        for (int j = 0; j < all_turns; ++j) {
            const int stage = j & 1, first = p_first + 2 * (rank + j * SPLIT);
            const uint32_t freed = ((j >> 1) + 1) & 1;   // the turn before last has been read
            int page[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                page[h] = table_row[min(first + h, p_last)];   // (beyond the last page: masked keys, values that nothing reads)
                if (page[h] < 0) {  // a page the sequence does not hold: reported; some held memory is read instead
                    if (leader) atomicOr(err, QF_ERR_NO_PAGE);
                    page[h] = 0;
                }
            }
            if (j >= 2 && !wait_all(&bar_k_free[stage], freed)) {
                timed_out = true;
                break;
            }
            // row of the cache seen as one matrix [pages * planes * kv_heads * 64][D]; with one plane per page the values
            // are the keys themselves (the same rows fetched into the values' stage)
            ++keys;
            if (leader) {
                mbar_expect_tx(&bar_k[stage], KV_BYTES);
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int cb = 0; cb < CB; ++cb)
                        tma_load_2d(k_s + stage * KV_BYTES + cb * KV_BLOCK + h * PAGE_BYTES, &kv_map, cb * 64,
                                    (int)(((long long)page[h] * planes * site.kv_heads + kvh) * QF_PAGE), &bar_k[stage]);
            }
            __syncwarp();
            if (j >= 2 && !wait_all(&bar_v_free[stage], freed)) {
                timed_out = true;
                break;
            }
            ++values;
            if (leader) {
                mbar_expect_tx(&bar_v[stage], KV_BYTES);
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int cb = 0; cb < CB; ++cb)
                        tma_load_2d(v_s + stage * KV_BYTES + cb * KV_BLOCK + h * PAGE_BYTES, &kv_map, cb * 64,
                                    (int)((((long long)page[h] * planes + planes - 1) * site.kv_heads + kvh) * QF_PAGE), &bar_v[stage]);
            }
            __syncwarp();
        }
        // The block ends, also after a wait that ran out, only when nothing is on its way to its shared memory (long arrived otherwise).
        if (all_turns > 0) timed_out |= !wait_all(&bar_q, 0);
        for (int j = max(keys - 2, 0); j < keys; ++j) timed_out |= !wait_all(&bar_k[j & 1], (j >> 1) & 1);
        for (int j = max(values - 2, 0); j < values; ++j) timed_out |= !wait_all(&bar_v[j & 1], (j >> 1) & 1);
    } else if (warp == PRODUCTS) {
        // ---- the products
        const bool leader = elect_one();
        // descriptors: an address field counts 16 bytes, so 16 columns of a K-major row (32 bytes) are 2 units
        const uint64_t desc_q = smem_desc_sw128(q_s), desc_k = smem_desc_sw128(k_s), desc_v = smem_desc_mn_sw128(v_s, KV_BLOCK);
        constexpr uint32_t idesc_s = umma_idesc_bf16(TA_BM, TA_BK, false), idesc_pv = umma_idesc_bf16(TA_BM, D, true);
        // S of tile i, turn j; the last tile that reads a turn's keys hands their stage back
        auto issue_s = [&](int i, int j) {
            if (!wait_all(&bar_k[j & 1], (j >> 1) & 1)) return false;
            tc_fence_after();
            if (leader) {
                const uint64_t dq = desc_q + (uint64_t)(i * (Q_BYTES >> 4)), dk = desc_k + (uint64_t)((j & 1) * (KV_BYTES >> 4));
#pragma unroll
                for (int ks = 0; ks < D / 16; ++ks)
                    umma_bf16(tmem + 128 * i, dq + (uint64_t)((ks / 4) * (Q_BLOCK >> 4) + 2 * (ks % 4)),
                              dk + (uint64_t)((ks / 4) * (KV_BLOCK >> 4) + 2 * (ks % 4)), idesc_s, ks > 0 ? 1u : 0u);
                umma_commit(&bar_s[i]);
                if (i == 1 || j >= turns[1]) umma_commit(&bar_k_free[j & 1]);
            }
            __syncwarp();
            return true;
        };
        if (all_turns > 0) timed_out = !wait_all(&bar_q, 0);
        for (int i = 0; i < 2 && !timed_out; ++i)
            if (turns[i] > 0) timed_out = !issue_s(i, 0);
        for (int j = 0; j < all_turns && !timed_out; ++j) {
            for (int i = 0; i < 2 && !timed_out; ++i) {
                if (j >= turns[i]) continue;
                if (!wait_all(&bar_v[j & 1], (j >> 1) & 1) || !wait_all(&bar_p[i], j & 1)) {   // every row has written its weights
                    timed_out = true;
                    break;
                }
                tc_fence_after();
                if (leader) {   // values [128 keys][D] as they lie (MN-major), 16 keys are two groups of 8 rows (2048 bytes)
                    const uint64_t dv = desc_v + (uint64_t)((j & 1) * (KV_BYTES >> 4));
                    const int first = p_first + 2 * (rank + j * SPLIT);
                    const int k0 = first >= p_lo[i] ? 0 : first + 1 >= p_lo[i] ? 4 : 8, k1 = first + 1 < p_end[i] ? 8 : 4;
#pragma unroll
                    for (int kk = 0; kk < TA_BK / 16; ++kk)
                        if (kk >= k0 && kk < k1)
                            umma_bf16_tmem_a(tmem + O_COL + 128 * i, tmem + 128 * i + 8 * kk, dv + (uint64_t)(kk * (2048 >> 4)), idesc_pv,
                                             (j > 0 || kk > k0) ? 1u : 0u);
                    umma_commit(&bar_pv[i]);
                    if (i == 1 || j >= turns[1]) umma_commit(&bar_v_free[j & 1]);
                }
                __syncwarp();
                if (j + 1 < turns[i] && (!wait_all(&bar_pv[i], j & 1) || !issue_s(i, j + 1))) timed_out = true;
            }
        }
        if (leader) umma_commit(&bar_end);   // nor while a product of its is at work
        __syncwarp();
        timed_out |= !wait_all(&bar_end, 0);
    } else {
        // ---- the row threads
        const int my_turns = t ? turns[1] : turns[0];
        const int pos0 = pos_first + my_row0 - row0[0], row_pos = pos0 + row, row_lo = window > 0 ? max(0, row_pos - window + 1) : 0;
        const uint32_t lanes = tmem + ((uint32_t)((warp & 3) * 32) << 16), s_at = lanes + 128 * t, o_at = lanes + O_COL + 128 * t;
        const float folded = scale_log2 > 0.f ? scale_log2 : 1.f;
        for (int j = 0; j < my_turns; ++j) {
            if (!wait_all(&bar_s[t], j & 1)) {   // (the product of the turn before is done too: S was issued after it)
                timed_out = true;
                break;
            }
            tc_fence_after();
            float s[TA_BK];
            tmem_load_row_128(s_at, s);
            if (!(scale_log2 > 0.f)) {   // below, the scale is folded into the exponent, behind the maximum and the mask: above zero only
#pragma unroll
                for (int i = 0; i < TA_BK; ++i) s[i] *= scale_log2;
            }
            const int key0 = (p_first + 2 * (rank + j * SPLIT)) * QF_PAGE;
            // a block of keys that every row of the tile sees whole needs no mask
            const bool full = key0 + TA_BK - 1 <= pos0 && key0 >= (window > 0 ? max(0, pos0 + TA_BM - 1 - window + 1) : 0);
            if (!full) {   // a key that the row does not see gets the weight 2^-inf = 0
#pragma unroll
                for (int i = 0; i < TA_BK; ++i) s[i] = (key0 + i <= row_pos && key0 + i >= row_lo) ? s[i] : -INFINITY;
            }
            float mx[4];  // four chains instead of one: the comparisons do not wait for each other
#pragma unroll
            for (int i = 0; i < 4; ++i) mx[i] = s[i];
#pragma unroll
            for (int i = 4; i < TA_BK - 4; i += 8)
#pragma unroll
                for (int c = 0; c < 4; ++c) mx[c] = max3(mx[c], s[i + c], s[i + 4 + c]);
#pragma unroll
            for (int c = 0; c < 4; ++c) mx[c] = fmaxf(mx[c], s[TA_BK - 4 + c]);
            // (the scores stay unscaled; the scale is folded into the exponent)
            const float m_true = fmaxf(m_ref, fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * folded);
            float f_o = 1.0f;
            bool moved = false;
            if (j == 0) {
                m_ref = m_true;  // nothing to rescale yet: the first products overwrite O
                if (t && first_empty) {   // (no products in this turn: O begins as zeros)
                    uint32_t zeros[16];
#pragma unroll
                    for (int i = 0; i < 16; ++i) zeros[i] = 0u;
#pragma unroll 1
                    for (int c0 = 0; c0 < D; c0 += 16) tmem_store_16(o_at + c0, zeros);
                }
            } else if (m_true - m_ref > 8.0f) {
                moved = true;
                f_o = fast_exp2(m_ref - m_true);
                m_ref = m_true;
                l_run *= f_o;
            }
            if (__any_sync(0xffffffffu, moved)) {  // the warp's 32 rows of O are loaded and stored together
#pragma unroll 1
                for (int c0 = 0; c0 < D; c0 += 16) {
                    uint32_t raw[16];
                    tmem_load_16(o_at + c0, raw);
#pragma unroll
                    for (int i = 0; i < 16; ++i) raw[i] = __float_as_uint(__uint_as_float(raw[i]) * f_o);
                    tmem_store_16(o_at + c0, raw);
                }
            }
            // two neighbouring weights an instruction where the pipes allow it: s * scale - reference, and the sums
            const float2 by = make_float2(folded, folded), less = make_float2(-m_ref, -m_ref);
            float2 part[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll
            for (int h = 0; h < 2; ++h) {   // half of the weights at a time: the first are stored while the others are formed
                uint32_t packed[32];
#pragma unroll
                for (int i = 0; i < 64; i += 2) {
                    float2 p = __ffma2_rn(make_float2(s[64 * h + i], s[64 * h + i + 1]), by, less);
                    p.x = fast_exp2(p.x), p.y = fast_exp2(p.y);
                    part[(i >> 1) & 1] = __fadd2_rn(part[(i >> 1) & 1], p);
                    packed[i / 2] = pack_bf16(p.x, p.y);
                }
                tmem_store_32(s_at + 32 * h, packed);
            }
            l_run += (part[0].x + part[0].y) + (part[1].x + part[1].y);
            tmem_store_wait();
            tc_fence_before();
            __syncwarp();
            if ((threadIdx.x & 31) == 0) mbar_arrive(&bar_p[t]);
        }
        if (!timed_out && my_turns > 0 && !wait_all(&bar_pv[t], (my_turns - 1) & 1)) timed_out = true;
        tc_fence_after();
        if (SPLIT == 1 && !timed_out && my_turns > 0) {  // the loads are collective: every lane of the warp takes part, rows beyond the span store nothing
            float den = l_run, keep = 1.f;
            if (sinks) {  // a sink's term joins the sum of weights once, in base-2 units like the scores, on a common maximum
                const float s2 = sinks[my_head] * 1.4426950408889634f, m_new = fmaxf(m_ref, s2);
                keep = exp2f(m_ref - m_new);
                den = l_run * keep + exp2f(s2 - m_new);
            }
            const float inv = den > 0.f ? keep / den : 0.f;
#pragma unroll
            for (int c0 = 0; c0 < D; c0 += 32) {
                uint32_t raw[32];
                tmem_load_32(o_at + c0, raw);
                if (row < my_rows) {
#pragma unroll
                    for (int c = 0; c < 32; c += 8) {
                        float v[8];
#pragma unroll
                        for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(raw[c + i]) * inv;
                        *reinterpret_cast<uint4*>(out_row + c0 + c) =
                            make_uint4(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]), pack_bf16(v[4], v[5]), pack_bf16(v[6], v[7]));
                    }
                }
            }
        }
    }
    if (SPLIT > 1) {
        const int my_turns = t ? turns[1] : turns[0];
        const bool have = my_turns > 0 && !timed_out;
        const uint32_t o_at = tmem + ((uint32_t)((warp & 3) * 32) << 16) + O_COL + 128 * t;
        cooperative_groups::this_cluster().sync();  // every thread of all blocks: all have left their loops, their stages are free
        if (warp < PRODUCTS && my_rows > 0) {
            // every block brings a slice of the columns together: this block's sums of every other slice go to its block, its rows'
            // reference maxima and sums of weights to all
#pragma unroll
            for (int to = 0; to < SPLIT; ++to) {
                float* ml = cooperative_groups::this_cluster().map_shared_rank(merge_ml, to) + (rank * PER + t) * 2 * TA_BM + row;
                ml[0] = have ? m_ref : QF_NEG_BIG;
                ml[TA_BM] = have ? l_run : 0.f;
                if (to == rank) continue;
                float* sums = cooperative_groups::this_cluster().map_shared_rank(merge_s, to) + (size_t)(rank * PER + t) * DS * TA_BM + row;
#pragma unroll 1
                for (int c0 = 0; c0 < DS; c0 += 8) {
                    uint32_t raw[8];
                    if (have) tmem_load_8(o_at + to * DS + c0, raw);
#pragma unroll
                    for (int i = 0; i < 8; ++i) sums[(c0 + i) * TA_BM] = have ? __uint_as_float(raw[i]) : 0.f;
                }
            }
        }
        cooperative_groups::this_cluster().sync();  // the other blocks' parts have arrived
        if (warp < PRODUCTS && my_rows > 0) {
            // every part carries a reference maximum of its own; the common one is the largest
            float m_all = QF_NEG_BIG, l_all = 0.f, keep = 1.f, by[SPLIT];
#pragma unroll
            for (int r = 0; r < SPLIT; ++r) m_all = fmaxf(m_all, by[r] = merge_ml[(r * PER + t) * 2 * TA_BM + row]);
#pragma unroll
            for (int r = 0; r < SPLIT; ++r) {
                by[r] = fast_exp2(by[r] - m_all);
                l_all = fmaf(merge_ml[((r * PER + t) * 2 + 1) * TA_BM + row], by[r], l_all);
            }
            if (sinks) {  // a sink's term joins the sum of weights once, in base-2 units like the scores, on a common maximum
                const float s2 = sinks[my_head] * 1.4426950408889634f, m_new = fmaxf(m_all, s2);
                keep = exp2f(m_all - m_new);
                l_all = l_all * keep + exp2f(s2 - m_new);
            }
            const float inv = l_all > 0.f ? keep / l_all : 0.f;
#pragma unroll 1
            for (int c0 = 0; c0 < DS; c0 += 8) {
                uint32_t raw[8];
                if (have) tmem_load_8(o_at + rank * DS + c0, raw);
                float v[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    v[i] = 0.f;
#pragma unroll
                    for (int r = 0; r < SPLIT; ++r) {
                        const float part = r == rank ? (have ? __uint_as_float(raw[i]) : 0.f) : merge_s[((size_t)(r * PER + t) * DS + c0 + i) * TA_BM + row];
                        v[i] = fmaf(part, by[r], v[i]);
                    }
                    v[i] *= inv;
                }
                if (row < my_rows)
                    *reinterpret_cast<uint4*>(out_row + rank * DS + c0) =
                        make_uint4(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]), pack_bf16(v[4], v[5]), pack_bf16(v[6], v[7]));
            }
        }
    }
    if (timed_out) atomicOr(err, QF_ERR_COPY_TIMEOUT);
    tc_fence_before();
    __syncthreads();
    if (warp == PRODUCTS)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32  %0, %1;" ::"r"(tmem), "r"(TMEM_COLS));
}

template <int D, int SPLIT, int PER>
static int launch_variant(const CUtensorMap& q_map, const CUtensorMap& kv_map, void* out, const int* cu_q, const int* tok_pos,
                          const int* slots, KvSite<bf16> site, int n_heads, int n_seqs, long long tiles, float scale,
                          int window, int* err, const float* sinks, int planes, cudaStream_t stream) {
    // One block per SM, also where two would find room, and no other kernel's that takes tensor memory: a block with two tiles holds
    // all of its SM's, and the blocks of clusters that wait for one another must not wait for tensor memory as well.
    constexpr size_t stages = (size_t)(D / 64) * (PER * TA_BM + 4 * TA_BK) * 128 + 1024, alone = QF_TMEM_SMEM_ALONE;
    constexpr size_t merge = (size_t)PER * (D + 2 * SPLIT) * TA_BM * sizeof(float) + 1024;
    constexpr size_t smem = stages > merge ? (stages > alone ? stages : alone) : (merge > alone ? merge : alone);
    static_assert(qf_tmem_fits(256 * PER, smem) && smem <= 227 * 1024, "the rule of tcgen05.cuh");
    auto kernel = prefill_tc_kernel<D, SPLIT, PER>;
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
    const long long blocks = (tiles + PER - 1) / PER * site.kv_heads * n_seqs * SPLIT;
    if (blocks > 0x7fffffffll) return (int)cudaErrorInvalidValue;
    cudaLaunchConfig_t config = {};
    config.gridDim = dim3((unsigned)blocks);
    config.blockDim = dim3(128 * PER + 64);
    config.dynamicSmemBytes = smem;
    config.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = SPLIT;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    config.attrs = attr;
    config.numAttrs = SPLIT > 1 ? 2 : 1;
    return (int)cudaLaunchKernelEx(&config, kernel, q_map, kv_map, (bf16*)out, cu_q, tok_pos, slots, site, n_heads, n_seqs,
                                   scale * 1.4426950408889634f, window, err, sinks, planes);
}

template <int D>
static int launch(const void* q, void* out, const int* cu_q, const int* tok_pos, const int* slots, void* base,
                  const int* table, long long page_elems, int table_stride, int kv_heads, int n_heads, int n_seqs,
                  int n_tokens, int max_q_len, int max_kv_len, float scale, int window, int* err, const float* sinks,
                  int shared_values, cudaStream_t stream) {
    // the cache pages must be what the map takes them for: [planes][kv_heads][64][D] without gaps
    const int planes = shared_values ? 1 : 2;
    if (page_elems != (long long)planes * kv_heads * QF_PAGE * D) return (int)cudaErrorInvalidValue;
    KvSite<bf16> site{(bf16*)base, table, page_elems, table_stride, kv_heads, D};
    CUtensorMap q_map = {}, kv_map = {};
    const long long q_width = (long long)n_heads * D;
    if (!qf_make_map_bf16(&q_map, q, n_tokens, q_width, q_width, TA_BM)) return (int)cudaErrorNotSupported;
    // The cache of this entry as one matrix of rows of D elements. The map is given more rows than any cache has
    // (its extent only bounds what a copy may address; copies address rows of held pages only).
    if (!qf_make_map_bf16(&kv_map, base, 1ll << 31, D, D, QF_PAGE)) return (int)cudaErrorNotSupported;
    const int q_tiles = (max_q_len + TA_BM - 1) / TA_BM;
    const long long tiles = (long long)q_tiles * (n_heads / kv_heads);   // of the longest sequence and a kv head
    // How many tiles a block takes and how many blocks share them: the choice that is done first by this estimate, in
    // microseconds as measured (prompts and portions, 14 to 28 heads, inside a graph): a turn takes 1.75 with one tile and 2.05
    // with two at D = 128, 1.5 and 1.85 at D = 64; a block's start and end take 3 to 6.5 with one tile and 5 to 13 with two, the more
    // the more blocks a cluster has; clusters of four and of eight do not find room on every SM. Tiles x blocks 1 x 1, 2 x 1, 2 x 2
    // and 2 x 8, chosen first: one prompt of 4,096 tokens, 14 heads of 64: 91, [62], 73, 211; of 1,024: 15.4, 19, [14], 45; 256 tokens
    // behind 8,000: 99, 115, 63, [25]; 64 behind 8,000, 16 heads of 128: 112, 127, 71, [31]; four prompts of 183 to 275: [7.2], 9.1, 10, 53.
    const int span = window > 0 && window + TA_BM < max_kv_len ? window + TA_BM : max_kv_len;
    const float longest = (float)((span + TA_BK - 1) / TA_BK), mean = longest > q_tiles ? longest - 0.5f * q_tiles : 0.5f * longest + 0.5f;
    // Tiles that hold rows, of an average sequence and query head (the grid also has blocks for the rows that shorter sequences lack, which
    // end at once): the longest sequence, and the others as long as what is left.
    const float rest = n_seqs > 1 ? fmaxf((float)(n_tokens - max_q_len) / (float)(n_seqs - 1), 1.f) : 0.f;
    const float live = (q_tiles + (n_seqs - 1) * fminf((float)q_tiles, ceilf(rest / TA_BM))) / (float)n_seqs;
    const int sms = qf_sm_count() > 0 ? qf_sm_count() : 1;
    const float turn[2] = {D <= 64 ? 1.5f : 1.75f, D <= 64 ? 1.85f : 2.05f}, ends[2][4] = {{3.f, 5.f, 5.5f, 6.5f}, {5.f, 6.5f, 9.f, 13.f}};
    const int room[4] = {sms, sms, sms - sms / 8, sms * 77 / 100 > 0 ? sms * 77 / 100 : 1};
    // Blocks of one tile and of two: the tiles of a sequence and kv head go in pairs, of which an odd count leaves half a block.
    const int group = n_heads / kv_heads;
    const float pairs = n_seqs == 1 ? ceilf(live * group / 2) : fmaxf(live * group / 2 + (group & 1 ? 0.25f : 0.f), (float)((group + 1) / 2));
    const float count[2] = {live * n_heads * n_seqs, pairs * kv_heads * n_seqs};
    int per = 2, split = 1;
    float least = -1.f;
    for (int p = 2; p >= 1; --p)
        for (int n = 0; n < 4; ++n) {
            const long long blocks = (long long)ceilf(count[p - 1] - 0.01f) << n;
            const float alone = ceilf(longest / (1 << n)) * turn[p - 1] + ends[p - 1][n];
            // (of several sequences the count is an estimate itself: a twentieth more than a round is taken for one)
            const long long rounds = n_seqs > 1 && blocks * 20 <= room[n] * 21ll ? 1 : (blocks + room[n] - 1) / room[n];
            const float all = (float)rounds * (mean / (1 << n) * turn[p - 1] + ends[p - 1][n]);
            const float time = alone > all ? alone : all;
            if (least < 0.f || time < least) least = time, per = p, split = 1 << n;
        }
    if (D == 64) {   // (in favour of the small blocks by what the estimates are uncertain of, less where every chain is alike)
        bool two;
        if ((q_tiles > 1 ? 0.85f : 0.95f) * pages_time(live, n_heads, n_seqs, n_tokens, span, q_tiles, sms, two) <= least)
            return two ? launch_pages<true>(q_map, kv_map, out, cu_q, tok_pos, slots, site, n_heads, n_seqs, max_q_len, scale, window, err, sinks, planes, stream)
                       : launch_pages<false>(q_map, kv_map, out, cu_q, tok_pos, slots, site, n_heads, n_seqs, max_q_len, scale, window, err, sinks, planes, stream);
    }
#define QF_TC_LAUNCH(SPLIT, PER) \
    launch_variant<D, SPLIT, PER>(q_map, kv_map, out, cu_q, tok_pos, slots, site, n_heads, n_seqs, tiles, scale, window, err, sinks, planes, stream)
    if (per == 1) return split == 1 ? QF_TC_LAUNCH(1, 1) : split == 2 ? QF_TC_LAUNCH(2, 1) : split == 4 ? QF_TC_LAUNCH(4, 1) : QF_TC_LAUNCH(8, 1);
    return split == 1 ? QF_TC_LAUNCH(1, 2) : split == 2 ? QF_TC_LAUNCH(2, 2) : split == 4 ? QF_TC_LAUNCH(4, 2) : QF_TC_LAUNCH(8, 2);
#undef QF_TC_LAUNCH
}

// The arguments of qf_attention_prefill (with `max_kv_len`, the bound that steers the sharing of a tile) and the number
// of rows of q (n_tokens). cudaErrorInvalidValue for a head
// size other than 64 or 128, or for cache pages with gaps (the caller then uses another kernel).
// `sinks` (float32 per query head, or null) and `shared_values` (pages of one plane whose rows are keys and values both) as
// in the other attention kernels.
QF_EXPORT int qf_attention_prefill_tc_ex(const void* q, void* out, const int* cu_q, const int* tok_pos, const int* slots,
                                         void* base, const int* table, long long page_elems, int table_stride, int kv_heads,
                                         int head_dim, int n_heads, int n_seqs, int n_tokens, int max_q_len, int max_kv_len,
                                         float scale, int window, int* err, const float* sinks, int shared_values,
                                         cudaStream_t stream) {
    if (n_seqs <= 0 || max_q_len <= 0 || n_tokens <= 0) return 0;
    if (kv_heads <= 0 || n_heads % kv_heads) return (int)cudaErrorInvalidValue;
    if (head_dim == 64)
        return launch<64>(q, out, cu_q, tok_pos, slots, base, table, page_elems, table_stride, kv_heads, n_heads, n_seqs,
                          n_tokens, max_q_len, max_kv_len, scale, window, err, sinks, shared_values, stream);
    if (head_dim == 128)
        return launch<128>(q, out, cu_q, tok_pos, slots, base, table, page_elems, table_stride, kv_heads, n_heads, n_seqs,
                           n_tokens, max_q_len, max_kv_len, scale, window, err, sinks, shared_values, stream);
    return (int)cudaErrorInvalidValue;
}

QF_EXPORT int qf_attention_prefill_tc(const void* q, void* out, const int* cu_q, const int* tok_pos, const int* slots,
                                      void* base, const int* table, long long page_elems, int table_stride, int kv_heads,
                                      int head_dim, int n_heads, int n_seqs, int n_tokens, int max_q_len, int max_kv_len,
                                      float scale, int window, int* err, cudaStream_t stream) {
    return qf_attention_prefill_tc_ex(q, out, cu_q, tok_pos, slots, base, table, page_elems, table_stride, kv_heads, head_dim,
                                      n_heads, n_seqs, n_tokens, max_q_len, max_kv_len, scale, window, err, nullptr, 0, stream);
}
