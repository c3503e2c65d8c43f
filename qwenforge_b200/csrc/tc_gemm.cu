// Matrix products for many token rows on the fifth-generation tensor cores (tcgen05), bf16 in, float32
// accumulation in tensor memory:   C[M][N] = A[M][K] * W[N][K]^T
// with the feed-forward's gate fused in:  EPI_SWIGLU writes silu(gate) * up for W = [gate rows | up rows].
//
// One block computes one 128 x 128 or 128 x 256 tile of C. Operand tiles of 128 rows x 64 columns (128 bytes per row) are
// brought into shared memory by the tensor memory accelerator (2-D tiled copies with the 128-byte swizzle that
// the tensor cores read) through a ring of stages. Thread 0 of warp 0 issues the copies, thread 0 of warp 1 issues
// the tcgen05.mma instructions (four of K = 16 per stage) whose accumulator is 128 lanes x 128 or 256 columns of
// tensor memory; `tcgen05.commit` hands a stage back when its products have been read, and signals the epilogue at the
// end. All four warps then read their 32 accumulator lanes with tcgen05.ld, apply the epilogue and store.
// Two blocks fit an SM, so one block's epilogue overlaps the other's products. Every wait on a barrier is bounded;
// a wait that runs out sets QF_ERR_COPY_TIMEOUT, and the block still frees its tensor memory and returns.
// Copies use no cluster multicast; every block loads its own tiles.
#include "tcgen05.cuh"

enum { TC_PLAIN = 0, TC_SWIGLU = 1, TC_QKV = 2 };

// What the TC_QKV epilogue needs beside the product: W = [q heads | k heads | v heads] of head_dim rows each; the sums get
// the bias, q and k heads are rotated by the token's angles (a table [tokens][head_dim / 2] of (cos, sin) made once per
// step), q goes to q_out [tokens][n_heads * head_dim], k and v to the token's place in its sequence's cache page.
struct TcQkvArgs {
    const bf16* bias;        // [(n_heads + 2 kv_heads) * head_dim] or null
    const float2* angles;    // [tokens][head_dim / 2] (cos, sin), or null: no rotation
    const int* tok_pos;
    const int* tok_seq;
    const int* slots;
    bf16* q_out;
    bf16* kv_base;
    const int* table;
    long long page_elems;
    int table_stride, n_heads, kv_heads, head_dim, write_cache;
    const float* inv_freq;   // (the pairs' form) [head_dim / 2] frequencies, or null: no rotation
};

// One head (or half of one) of the TC_QKV epilogue for this thread's token row: P = D / 2 rotation pairs, W of them per
// turn from tensor memory columns `col` (first halves) and `col + P` (second halves).
template <int W>
__device__ __forceinline__ void qkv_head_turn(uint32_t lane_addr, int col, int P, const float* bias_s, const float2* angle_row,
                                              int first_pair, bool rotate, bf16* dst, bool store) {
    uint32_t lo[W], hi[W];
    if constexpr (W == 32) {
        tmem_load_32(lane_addr + col, lo);
        tmem_load_32(lane_addr + col + P, hi);
    } else {
        tmem_load_16(lane_addr + col, lo);
        tmem_load_16(lane_addr + col + P, hi);
    }
    if (!store) return;
    uint32_t o1[W / 2], o2[W / 2];
#pragma unroll
    for (int j = 0; j < W; j += 2) {
        float y1[2], y2[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const float x1 = __uint_as_float(lo[j + e]) + bias_s[col + j + e], x2 = __uint_as_float(hi[j + e]) + bias_s[col + P + j + e];
            if (rotate) {
                const float2 a = angle_row[first_pair + j + e];  // (cos, sin)
                y1[e] = x1 * a.x - x2 * a.y;
                y2[e] = x2 * a.x + x1 * a.y;
            } else {
                y1[e] = x1;
                y2[e] = x2;
            }
        }
        o1[j / 2] = pack_bf16(y1[0], y1[1]);
        o2[j / 2] = pack_bf16(y2[0], y2[1]);
    }
#pragma unroll
    for (int j = 0; j < W / 2; j += 4) {
        *reinterpret_cast<uint4*>(dst + first_pair + 2 * j) = make_uint4(o1[j], o1[j + 1], o1[j + 2], o1[j + 3]);
        *reinterpret_cast<uint4*>(dst + P + first_pair + 2 * j) = make_uint4(o2[j], o2[j + 1], o2[j + 2], o2[j + 3]);
    }
}

// Grouped products (the experts of a mixture-of-experts feed-forward): the rows of A are sorted by group and cut into tiles
// of 128 rows by a plan on the device (csrc/moe.cu). Tile i belongs to group tile_group[i], starts at row tile_row0[i] (any
// row: a tiled copy's row coordinate has no alignment rule) and ends where the group's rows end; what the tile holds beyond
// that end are the next group's rows, which are multiplied and not stored. Group g's weights are rows g * w_rows .. of W.
// The grid has a block row for every tile that any routing can have; those beyond n_tiles[0] end at once. `row_scale`
// (float32 per row, or null) multiplies both halves of the TC_SWIGLU epilogue's sums before the gate: a weight on the
// expert's input moved behind its first product. tile_group == null: an ordinary product.
struct TcGroups {
    const int* tile_group;
    const int* tile_row0;
    const int* offsets;
    const int* n_tiles;
    const float* row_scale;
    int w_rows;
    // gate_limit > 0: the TC_SWIGLU epilogue's gate is the clamped one, g * sigmoid(gate_alpha * g) * (u + 1) with
    // g = min(gate, limit), u = clamp(up, -limit, limit), instead of silu(gate) * up
    float gate_limit;
    float gate_alpha;
};

#define TC_BM 128
#define TC_BK 64
#define TC_THREADS 128
// tile width BN: 128 (three stages of 32 KB, two blocks per SM) or 256 (four stages of 48 KB, one block per SM)
template <int BN> struct TcGeometry {
    static constexpr int stages = BN == 128 ? 3 : 4;
    static constexpr int stage_bytes = (TC_BM + BN) * TC_BK * 2;
    static constexpr size_t smem = (size_t)stages * stage_bytes + 1024;
    static_assert(qf_tmem_fits(BN, smem), "the rule of tcgen05.cuh");
};

// Instruction descriptor: float32 accumulator, bf16 A and B, both K-major, N = BN, M = 128.
template <int BN> __device__ __forceinline__ constexpr uint32_t tc_idesc() {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(TC_BM >> 4) << 24);
}

template <int EPI, int BN>
__global__ void __launch_bounds__(TC_THREADS)
tc_gemm_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, bf16* __restrict__ out,
               int M, int n_out, int K, int inter, int ldo, const TcQkvArgs qa, int* err, const TcGroups gr) {
    if (gr.tile_group && (int)blockIdx.y >= gr.n_tiles[0]) return;   // the whole block, before it holds anything
    extern __shared__ unsigned char smem_unaligned[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_unaligned) + 1023) & ~(uintptr_t)1023);
    constexpr int TC_STAGES = TcGeometry<BN>::stages, TC_STAGE_BYTES = TcGeometry<BN>::stage_bytes;
    constexpr int HALF = BN / 2;  // TC_SWIGLU: gate columns [0, HALF), up columns [HALF, BN)
    __shared__ __align__(8) uint64_t full_bar[TC_STAGES], empty_bar[TC_STAGES], acc_bar;
    __shared__ uint32_t tmem_base_s;
    __shared__ float bias_s[EPI == TC_QKV ? BN : 1];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tile_n = blockIdx.x, tile_m = blockIdx.y;
    const int n_k = (K + TC_BK - 1) / TC_BK;
    const int group = gr.tile_group ? gr.tile_group[blockIdx.y] : 0;
    const int row0 = gr.tile_group ? gr.tile_row0[blockIdx.y] : tile_m * TC_BM;   // first row of the tile
    const int row_end = gr.tile_group ? min(gr.offsets[group + 1], M) : M;       // rows from here on are not this tile's
    const int w_row0 = gr.tile_group ? group * gr.w_rows : 0;                     // first weight row of the tile's group
    // TC_QKV: where this thread's token row stands and where its key and value go (element offset in the cache, -1: nowhere)
    long long kv_at = -1;
    auto find_row = [&]() {
        const int row = tile_m * TC_BM + warp * 32 + lane;
        if (row < M && qa.write_cache) {
            const int slot = qa.slots[qa.tok_seq[row]], pos = qa.tok_pos[row];
            if (slot >= 0) {
                const int page = qa.table[(long long)slot * qa.table_stride + pos / QF_PAGE];
                if (page < 0) atomicOr(err, QF_ERR_NO_PAGE);
                else kv_at = (long long)page * qa.page_elems + (long long)(pos % QF_PAGE) * qa.head_dim;
            }
        }
    };

    if (threadIdx.x == 0) {
        for (int s = 0; s < TC_STAGES; ++s) {
            mbar_init(&full_bar[s], 1);
            mbar_init(&empty_bar[s], 1);
        }
        mbar_init(&acc_bar, 1);
    }
    if (warp == 0) {  // one warp allocates the accumulator: 128 columns of tensor memory
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&tmem_base_s)), "r"(BN));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_acc = tmem_base_s;
    bool timed_out = false;

    if (warp == 0 && lane == 0) {
        // ---- producer: fill the ring with operand tiles
        for (int kb = 0; kb < n_k && !timed_out; ++kb) {
            const int s = kb % TC_STAGES;
            if (kb >= TC_STAGES && !mbar_wait(&empty_bar[s], ((kb / TC_STAGES) - 1) & 1)) {
                timed_out = true;
                break;
            }
            unsigned char* a_s = smem + (size_t)s * TC_STAGE_BYTES;
            unsigned char* b_s = a_s + TC_BM * TC_BK * 2;
            mbar_expect_tx(&full_bar[s], TC_STAGE_BYTES);
            tma_load_2d(a_s, &map_a, kb * TC_BK, row0, &full_bar[s]);
#pragma unroll
            for (int box = 0; box < BN / 64; ++box) {  // boxes of 64 weight rows
                int w_row = tile_n * BN + 64 * box;
                if (EPI == TC_SWIGLU)  // HALF gate rows, then the HALF matching up rows
                    w_row = 64 * box < HALF ? tile_n * HALF + 64 * box : inter + tile_n * HALF + (64 * box - HALF);
                tma_load_2d(b_s + (size_t)box * 64 * TC_BK * 2, &map_b, kb * TC_BK, w_row0 + w_row, &full_bar[s]);
            }
        }
    } else if (warp == 1 && lane == 0) {
        // ---- one thread issues the products
        for (int kb = 0; kb < n_k && !timed_out; ++kb) {
            const int s = kb % TC_STAGES;
            if (!mbar_wait(&full_bar[s], (kb / TC_STAGES) & 1)) {
                timed_out = true;
                break;
            }
            tc_fence_after();
            const unsigned char* a_s = smem + (size_t)s * TC_STAGE_BYTES;
            const unsigned char* b_s = a_s + TC_BM * TC_BK * 2;
            const uint64_t da = smem_desc_sw128(a_s), db = smem_desc_sw128(b_s);
#pragma unroll
            for (int k4 = 0; k4 < TC_BK / 16; ++k4)  // 16 columns = 32 bytes = 2 units of the address field
                umma_bf16(tmem_acc, da + 2 * k4, db + 2 * k4, tc_idesc<BN>(), (kb > 0 || k4 > 0) ? 1u : 0u);
            umma_commit(&empty_bar[s]);  // arrives when these products have finished reading the stage
        }
        umma_commit(&acc_bar);           // arrives when every product has finished
    } else if (EPI == TC_QKV) {
        // the other threads use the time of the products: the tile's bias values and their rows' places in the cache
        for (int i = threadIdx.x - (threadIdx.x > 32 ? 2 : 1); i < BN; i += TC_THREADS - 2) {
            const int col = tile_n * BN + i;
            bias_s[i] = (qa.bias && col < n_out) ? __bfloat162float(qa.bias[col]) : 0.f;
        }
        find_row();
    }
    if (EPI == TC_QKV && lane == 0 && warp < 2) find_row();  // the two issuing threads' own rows
    if (timed_out) atomicOr(err, QF_ERR_COPY_TIMEOUT);
    __syncwarp();

    // ---- epilogue: warp w owns accumulator lanes (= tile rows) 32 w .. 32 w + 31
    if (!mbar_wait(&acc_bar, 0) && lane == 0) atomicOr(err, QF_ERR_COPY_TIMEOUT);
    tc_fence_after();
    const int row = row0 + warp * 32 + lane;
    const uint32_t lane_base = tmem_acc + ((uint32_t)(warp * 32) << 16);
    if (EPI == TC_QKV) {
        __syncthreads();  // the tile's bias values are in shared memory
        const int D = qa.head_dim, P = D / 2, total_heads = qa.n_heads + 2 * qa.kv_heads;
        const float2* angle_row = qa.angles ? qa.angles + (size_t)row * P : nullptr;
        for (int h = 0; h < BN / D; ++h) {   // the heads of this tile (the launch made sure that heads do not straddle tiles)
            const int head = tile_n * (BN / D) + h;
            if (head >= total_heads) break;
            const bool is_q = head < qa.n_heads, rotate = angle_row != nullptr && head < qa.n_heads + qa.kv_heads;
            bf16* dst = nullptr;
            if (row < M) {
                if (is_q) dst = qa.q_out + ((size_t)row * qa.n_heads + head) * D;
                else if (kv_at >= 0) dst = qa.kv_base + kv_at + (long long)(head - qa.n_heads) * QF_PAGE * D;  // keys, then values
            }
            // the loads from tensor memory are the whole warp's: every lane walks the turns, rows without a place store nothing
            if (P >= 32) {
                for (int first = 0; first < P; first += 32)
                    qkv_head_turn<32>(lane_base, h * D + first, P, bias_s, angle_row, first, rotate, dst, dst != nullptr);
            } else {
                qkv_head_turn<16>(lane_base, h * D, P, bias_s, angle_row, 0, rotate, dst, dst != nullptr);
            }
        }
    } else if (EPI == TC_SWIGLU) {
#pragma unroll
        for (int c0 = 0; c0 < HALF; c0 += 32) {
            uint32_t g[32], u[32];
            tmem_load_32(lane_base + c0, g);
            tmem_load_32(lane_base + HALF + c0, u);
            const int col = tile_n * HALF + c0;
            if (row < row_end && col < n_out) {
                const float rs = gr.row_scale ? gr.row_scale[row] : 1.0f;
                uint32_t packed[16];
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    float g0 = rs * __uint_as_float(g[2 * j]), g1 = rs * __uint_as_float(g[2 * j + 1]);
                    float u0 = rs * __uint_as_float(u[2 * j]), u1 = rs * __uint_as_float(u[2 * j + 1]);
                    float a = 1.0f;
                    if (gr.gate_limit > 0.f) {
                        const float lim = gr.gate_limit;
                        g0 = fminf(g0, lim), g1 = fminf(g1, lim);
                        u0 = fminf(fmaxf(u0, -lim), lim) + 1.0f, u1 = fminf(fmaxf(u1, -lim), lim) + 1.0f;
                        a = gr.gate_alpha;
                    }
                    packed[j] = pack_bf16(g0 / (1.0f + expf(-a * g0)) * u0, g1 / (1.0f + expf(-a * g1)) * u1);
                }
                bf16* dst = out + (size_t)row * ldo + col;
                if (col + 32 <= n_out) {
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        *reinterpret_cast<uint4*>(dst + 8 * j) = make_uint4(packed[4 * j], packed[4 * j + 1], packed[4 * j + 2], packed[4 * j + 3]);
                } else {
                    for (int j = 0; j < n_out - col; ++j) dst[j] = reinterpret_cast<const bf16*>(packed)[j];
                }
            }
        }
    } else {
#pragma unroll
        for (int c0 = 0; c0 < BN; c0 += 32) {
            uint32_t v[32];
            tmem_load_32(lane_base + c0, v);
            const int col = tile_n * BN + c0;
            if (row < row_end && col < n_out) {
                uint32_t packed[16];
#pragma unroll
                for (int j = 0; j < 16; ++j) packed[j] = pack_bf16(__uint_as_float(v[2 * j]), __uint_as_float(v[2 * j + 1]));
                bf16* dst = out + (size_t)row * ldo + col;
                if (col + 32 <= n_out) {
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        *reinterpret_cast<uint4*>(dst + 8 * j) = make_uint4(packed[4 * j], packed[4 * j + 1], packed[4 * j + 2], packed[4 * j + 3]);
                } else {
                    for (int j = 0; j < n_out - col; ++j) dst[j] = reinterpret_cast<const bf16*>(packed)[j];
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32  %0, %1;" ::"r"(tmem_acc), "r"(BN));
}

// ------------------------------------------------------------------------------------------------------------------
// The persistent form, for products of many tiles: pairs of SMs walk tiles of 256 x BN (tile index = pair, pair + pairs, ...;
// neighbouring pairs work on the same weight rows, which the L2 then serves). A pair is a cluster of two blocks, each of
// which brings 128 rows of A and BN / 2 rows of W per stage; one thread of its first block issues the products of both
// (tcgen05.mma, cta_group::2: 256 x BN x 16), which read the two blocks' shared memory, and each block's tensor memory gets
// the sums of its own 128 rows. The ring of stages runs on across tiles, and the accumulator is double: while the tensor
// cores fill one half of tensor memory with a tile's sums, eight epilogue warps read the other half, so a tile's epilogue and
// the start of the next tile's copies hide under products. Warp 0 issues copies, warp 1 of the first block products, warps 2
// to 9 own the epilogue: warp w reads accumulator lanes 32 (w % 4) .. + 31 (the lanes a warp may read are fixed by its number)
// and one half of the tile's columns. The launch is a programmatic dependent one: barriers and tensor memory are set up under
// the tail of the kernel before (a 905-token prompt of 24 layers: 1,548 -> 1,512 microseconds).
// What bounds it: at large K the tensor cores (7358 x 22016 x 2048: 407 microseconds, 1,631 TFLOP/s; one block a tile of 128 x 256,
// which reads 1.5 times the bytes from the L2 per product, took 476); at K = 896 the tiles' last round and what the
// ring takes to fill and the sums to drain (2048 x 9728 x 896 with the gate: 27 microseconds, 36 on single blocks).
// (The first tile's weights asked for before the wait for the kernel ahead: 1,528 instead of 1,512. Not kept.)
#define TP_THREADS 320
#define TP_EPI_WARPS 8
#define TP_PATCH_BYTES (32 * 128)
template <int BN> struct PairGeometry {   // BN 256 or 192: six stages; 128: eight; 64: nine
    static constexpr int stage_bytes = (TC_BM + BN / 2) * TC_BK * 2;
    static constexpr int stages = BN >= 192 ? 6 : BN == 128 ? 8 : 9;
    static constexpr size_t smem = (size_t)stages * stage_bytes + TP_EPI_WARPS * TP_PATCH_BYTES + 1024;
    static_assert(qf_tmem_fits(512, smem) && smem + 512 <= 227 * 1024, "the rule of tcgen05.cuh; what an SM gives a block");
};

// A warp's patch of results on its way out: 32 rows of 128 bytes, their 16-byte pieces permuted so that a row per lane is written and a
// row per eight lanes read without conflicts. (A row per lane stored straight to memory touches 32 lines an instruction, 1
// microsecond for 64 columns of a tile: 2048 x 9728 x 896 with the gate took 31 microseconds so, 27 by way of patches; 905 rows 18.9 and 16.8.)
__device__ __forceinline__ uint4* patch_at(unsigned char* patch, int row, int piece) {
    return reinterpret_cast<uint4*>(patch + row * 128 + ((piece ^ (row & 7)) << 4));
}

__device__ __forceinline__ float fast_silu(float x) { return __fdividef(x, 1.0f + __expf(-x)); }

// Tile t of the persistent walk. The pairs of the grid work on neighbouring t at any time, so the order decides what
// the L2 holds: tiles go by groups of `group_n` column tiles (their weight rows together fit in a quarter of the L2),
// and inside a group the column runs fastest, so that the pairs at work share a few row tiles of A and the group's
// weights, A streams through once per group, and the weights are read once. (With the row tile running fastest over
// the whole matrix, A was read again for every column tile once it outgrew the L2: 838 instead of 330 milliseconds
// for a 32,768-token step at Qwen2.5-7B sizes.)
__device__ __forceinline__ void tile_of(int t, int m_tiles, int n_tiles, int group_n, int& tile_m, int& tile_n) {
    const int per_group = group_n * m_tiles, g = t / per_group, first = g * group_n;
    const int width = min(group_n, n_tiles - first), local = t - g * per_group;
    tile_m = local / width;
    tile_n = first + local % width;
}

// The two epilogue warps of a quadrant of rows wait for each other.
__device__ __forceinline__ void quadrant_sync(int quad) { asm volatile("bar.sync %0, 64;" ::"r"(1 + quad) : "memory"); }

// 16 neighbouring rotation pairs of a head in this thread's row of the accumulator (first halves from column `lo` of its lane, second
// halves from `hi`), with the bias of both, rotated by cs = (cos, sin) where `rotate`, as 16-byte pieces of the row. The sums are rounded
// to bfloat16 first, as those of a product that is stored are: from the same sums come the queries, keys and values of such a product with
// the rotation kernel behind it, bit for bit (the library's product may add K in another order and so give other sums).
__device__ __forceinline__ void rotated_pairs(uint32_t lo, uint32_t hi, const bf16* bias_lo, const bf16* bias_hi, const float2* cs,
                                              bool rotate, uint4 (&out_lo)[2], uint4 (&out_hi)[2]) {
    uint32_t x[16], y[16];
    tmem_load_two(lo, hi, x, y);
#pragma unroll
    for (int j0 = 0; j0 < 16; j0 += 8) {
        uint32_t b1[4] = {0, 0, 0, 0}, b2[4] = {0, 0, 0, 0}, o1[4], o2[4];
        if (bias_lo) {
            const uint4 u = __ldg(reinterpret_cast<const uint4*>(bias_lo + j0)), v = __ldg(reinterpret_cast<const uint4*>(bias_hi + j0));
            b1[0] = u.x, b1[1] = u.y, b1[2] = u.z, b1[3] = u.w;
            b2[0] = v.x, b2[1] = v.y, b2[2] = v.z, b2[3] = v.w;
        }
#pragma unroll
        for (int j = 0; j < 8; j += 2) {
            float z1[2], z2[2];
            const uint32_t p1 = pack_bf16(__uint_as_float(x[j0 + j]), __uint_as_float(x[j0 + j + 1]));
            const uint32_t p2 = pack_bf16(__uint_as_float(y[j0 + j]), __uint_as_float(y[j0 + j + 1]));
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const float x1 = __uint_as_float(e ? p1 & 0xffff0000u : p1 << 16) + __uint_as_float(e ? b1[j / 2] & 0xffff0000u : b1[j / 2] << 16);
                const float x2 = __uint_as_float(e ? p2 & 0xffff0000u : p2 << 16) + __uint_as_float(e ? b2[j / 2] & 0xffff0000u : b2[j / 2] << 16);
                const float2 a = cs[j0 + j + e];
                z1[e] = rotate ? x1 * a.x - x2 * a.y : x1;
                z2[e] = rotate ? x2 * a.x + x1 * a.y : x2;
            }
            o1[j / 2] = pack_bf16(z1[0], z1[1]);
            o2[j / 2] = pack_bf16(z2[0], z2[1]);
        }
        out_lo[j0 / 8] = make_uint4(o1[0], o1[1], o1[2], o1[3]);
        out_hi[j0 / 8] = make_uint4(o2[0], o2[1], o2[2], o2[3]);
    }
}

// TC_PLAIN: the columns of W from n_out on, n_tail of them, are not rounded: their float32 sums go to tail [M][n_tail]. What a recurrent
// mixer's gates are made of rides on its projections' product so, where it was a launch of its own (7 microseconds).
struct TcTail {
    float* tail;
    int n_tail;
};

// P: rotation pairs of a head (TC_QKV; whole heads per tile)
template <int EPI, int BN, int P = 0>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(TP_THREADS, 1)
tc_gemm_pair_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                    bf16* __restrict__ out, int M, int n_out, int K, int inter, int ldo, int m_tiles, int n_tiles, int group_n,
                    int* err, const TcQkvArgs qa, const TcTail tail) {
    extern __shared__ unsigned char smem_unaligned[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_unaligned) + 1023) & ~(uintptr_t)1023);
    constexpr int STAGES = PairGeometry<BN>::stages, STAGE_BYTES = PairGeometry<BN>::stage_bytes;
    constexpr int HALF = BN / 2;      // the columns whose weight rows a block brings; TC_SWIGLU: gate columns [0, HALF), up columns [HALF, BN)
    __shared__ __align__(8) uint64_t full_bar[STAGES], empty_bar[STAGES], acc_full[2], acc_empty[2];
    __shared__ uint32_t tmem_base_s;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cluster_rank();
    const int pair = (int)blockIdx.x >> 1, pairs = (int)gridDim.x >> 1;
    const int n_k = (K + TC_BK - 1) / TC_BK, total = m_tiles * n_tiles;

    if (threadIdx.x == 32) {
        tma_prefetch_map(&map_a);
        tma_prefetch_map(&map_b);
    }
    // Both blocks' copies of a stage arrive at the first block's full_bar (one arrival, which announces both blocks' bytes); a
    // stage's and a tile's end are told to both blocks' empty_bar and acc_full; all sixteen epilogue warps arrive at the
    // first block's acc_empty.
    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(&full_bar[s], 1);
            mbar_init(&empty_bar[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&acc_full[b], 1);
            mbar_init(&acc_empty[b], 2 * TP_EPI_WARPS);
        }
    }
    if (warp == 0) {  // both accumulators: all 512 columns of either block's tensor memory
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&tmem_base_s)), "r"(512));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::);
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync();                   // the other block's barriers and tensor memory are there too
    tc_fence_after();
    const uint32_t tmem = tmem_base_s;
    bool timed_out = false;
    grid_launch_dependents();         // (this kernel has its tensor memory)

    if (warp == 0) {
        // ---- copies: all lanes run the loops, one issues
        const bool leader = elect_one();
        const uint32_t full0 = cluster_addr(full_bar, 0);
        int s = 0, issued = 0;
        uint32_t turn = 0;            // of the ring: its parity is that of the stage's copies in hand
        grid_dependency_wait();
        for (int t = pair; t < total && !timed_out; t += pairs) {
            int tile_m, tile_n;
            tile_of(t, m_tiles, n_tiles, group_n, tile_m, tile_n);
            const int a_row = (2 * tile_m + (int)rank) * TC_BM;
            // the first block brings the tile's first half of weight rows (TC_SWIGLU: the gate rows), the second the other (the up rows)
            const int w_row = EPI == TC_SWIGLU ? (int)rank * inter + tile_n * HALF : tile_n * BN + (int)rank * HALF;
            for (int kb = 0; kb < n_k; ++kb) {
                if (!__all_sync(0xffffffffu, mbar_wait(&empty_bar[s], (turn & 1) ^ 1))) {   // (true at once in the first turn)
                    timed_out = true;
                    break;
                }
                if (leader) {
                    unsigned char* a_s = smem + (size_t)s * STAGE_BYTES;
                    if (rank == 0) mbar_expect_tx(&full_bar[s], 2 * STAGE_BYTES);
                    tma_load_2d_pair(a_s, &map_a, kb * TC_BK, a_row, full0 + 8 * s);
                    tma_load_2d_pair(a_s + TC_BM * TC_BK * 2, &map_b, kb * TC_BK, w_row, full0 + 8 * s);
                }
                __syncwarp();
                if (issued < STAGES) ++issued;
                if (++s == STAGES) s = 0, ++turn;
            }
        }
        // what is on its way into either block has arrived before they end (as far as a bounded wait can say): the last stages'
        // releases, or after a wait that ran out the copies
        for (; issued > 0; --issued) {
            if (--s < 0) s = STAGES - 1, --turn;
            if (!timed_out) mbar_wait(&empty_bar[s], turn & 1);
            else if (rank == 0) mbar_wait(&full_bar[s], turn & 1);
        }
    } else if (warp == 1 && rank == 0) {
        // ---- products of both blocks
        const bool leader = elect_one();
        int s = 0, i = 0;
        uint32_t turn = 0;
        for (int t = pair; t < total && !timed_out; t += pairs, ++i) {
            const int buf = i & 1;
            if (!__all_sync(0xffffffffu, mbar_wait(&acc_empty[buf], ((i >> 1) & 1) ^ 1))) {  // both epilogues have read this half
                timed_out = true;
                break;
            }
            tc_fence_after();
            const uint32_t acc = tmem + (uint32_t)(buf * 256);
            for (int kb = 0; kb < n_k; ++kb) {
                if (!__all_sync(0xffffffffu, mbar_wait(&full_bar[s], turn & 1))) {
                    timed_out = true;
                    break;
                }
                tc_fence_after();
                if (leader) {
                    const unsigned char* a_s = smem + (size_t)s * STAGE_BYTES;
                    const uint64_t da = smem_desc_sw128(a_s), db = smem_desc_sw128(a_s + TC_BM * TC_BK * 2);
#pragma unroll
                    for (int k4 = 0; k4 < TC_BK / 16; ++k4)
                        umma_bf16_pair(acc, da + 2 * k4, db + 2 * k4, umma_idesc_bf16(2 * TC_BM, BN, false), (kb > 0 || k4 > 0) ? 1u : 0u);
                    umma_commit_pair(&empty_bar[s]);
                }
                __syncwarp();
                if (++s == STAGES) s = 0, ++turn;
            }
            if (timed_out) break;
            if (leader) umma_commit_pair(&acc_full[buf]);  // arrives when the tile's products have finished
            __syncwarp();
        }
    } else if (warp >= 2) {
        // ---- epilogue
        const int quad = warp & 3, half = (warp - 2) >> 2;
        unsigned char* patches = smem + (size_t)STAGES * STAGE_BYTES;
        unsigned char* patch = patches + (warp - 2) * TP_PATCH_BYTES;   // this warp's own (TC_QKV: shared by a quadrant's two warps, below)
        int i = 0;
        if (EPI == TC_QKV) grid_dependency_wait();   // (positions, slots and page tables)
        for (int t = pair; t < total; t += pairs, ++i) {
            const int buf = i & 1;
            int tile_m, tile_n;
            tile_of(t, m_tiles, n_tiles, group_n, tile_m, tile_n);
            const int row0 = (2 * tile_m + (int)rank) * TC_BM + quad * 32, row = row0 + lane;   // the warp's first row, this thread's
            const uint32_t lane_base = tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)(buf * 256);
            auto sums_there = [&]() {
                const bool there = __all_sync(0xffffffffu, mbar_wait(&acc_full[buf], (i >> 1) & 1));
                tc_fence_after();
                return there;
            };
            auto sums_read = [&]() {     // the warp has read its part of the half
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive_cluster(cluster_addr(&acc_empty[buf], 0));
            };
            if constexpr (EPI == TC_QKV) {
                constexpr int D = 2 * P, Q = P / 2;   // this thread makes pairs [half * Q, half * Q + Q) of every head in its row
                // under the tile's products: the row's angles and its place in the cache
                const int pos = row < M ? qa.tok_pos[row] : 0;
                long long kv_at = -1;                 // element offset in the cache, -1: nowhere
                if (row < M && qa.write_cache) {
                    const int slot = qa.slots[qa.tok_seq[row]];
                    if (slot >= 0) {
                        const int page = qa.table[(long long)slot * qa.table_stride + pos / QF_PAGE];
                        if (page < 0) atomicOr(err, QF_ERR_NO_PAGE);
                        else kv_at = (long long)page * qa.page_elems + (long long)(pos % QF_PAGE) * D;
                    }
                }
                float2 cs[Q];
#pragma unroll
                for (int j = 0; j < Q; ++j) {
                    cs[j] = make_float2(1.f, 0.f);
                    if (qa.inv_freq) sincosf((float)pos * __ldg(qa.inv_freq + half * Q + j), &cs[j].y, &cs[j].x);
                }
                // A head goes out by way of the quadrant's two patches: 128 bytes a row in one (D = 64), first halves in one and
                // second halves in the other (D = 128). Each warp then stores half of the quadrant's rows, eight lanes a row.
                unsigned char* shared = patches + quad * 2 * TP_PATCH_BYTES;
                long long out_at[4];
                int out_row[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const int r = (half * 4 + u) * 4 + (lane >> 3);
                    out_row[u] = row0 + r, out_at[u] = __shfl_sync(0xffffffffu, kv_at, r);
                }
                // after a wait that ran out a warp still passes all barriers below, where its quadrant's other warp may wait for it
                if (!timed_out && !sums_there()) timed_out = true;
#pragma unroll 1
                for (int h = 0; h < BN / D; ++h) {
                    const int head = tile_n * (BN / D) + h;
                    if (head >= qa.n_heads + 2 * qa.kv_heads) break;
                    unsigned char* at = D == 64 ? shared + (h & 1) * TP_PATCH_BYTES : shared;
                    const bool rotate = qa.inv_freq != nullptr && head < qa.n_heads + qa.kv_heads;
#pragma unroll
                    for (int j0 = 0; j0 < Q; j0 += 16) {   // 16 pairs a turn
                        const uint32_t lo = lane_base + h * D + half * Q + j0;
                        const bf16* bias = qa.bias ? qa.bias + head * D + half * Q + j0 : nullptr;
                        uint4 first[2], second[2];
                        rotated_pairs(lo, lo + P, bias, bias + P, cs + j0, rotate, first, second);
#pragma unroll
                        for (int j = 0; j < 2; ++j) {
                            *patch_at(at, lane, half * (Q / 8) + j0 / 8 + j) = first[j];
                            if (D == 64) *patch_at(at, lane, 4 + half * (Q / 8) + j0 / 8 + j) = second[j];
                            else *patch_at(at + TP_PATCH_BYTES, lane, half * (Q / 8) + j0 / 8 + j) = second[j];
                        }
                    }
                    quadrant_sync(quad);
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        if (out_row[u] >= M || timed_out) continue;
                        bf16* dst = nullptr;
                        if (head < qa.n_heads) dst = qa.q_out + ((size_t)out_row[u] * qa.n_heads + head) * D;
                        else if (out_at[u] >= 0) dst = qa.kv_base + out_at[u] + (long long)(head - qa.n_heads) * QF_PAGE * D;   // keys, then values
                        if (!dst) continue;
                        const int r = (half * 4 + u) * 4 + (lane >> 3);
#pragma unroll
                        for (int part = 0; part < D / 64; ++part)
                            *reinterpret_cast<uint4*>(dst + part * 64 + (lane & 7) * 8) = *patch_at(at + part * TP_PATCH_BYTES, r, lane & 7);
                    }
                    if (D == 128) quadrant_sync(quad);   // (D = 64: the next head goes by the other patch, and the one after by a barrier more)
                }
                if (D == 64) quadrant_sync(quad);
                if (!timed_out) sums_read();
            } else {
                if (!sums_there()) {
                    timed_out = true;
                    break;
                }
                // this warp's columns of results, up to 64 at a time
                constexpr int OWN = EPI == TC_SWIGLU ? HALF / 2 : HALF;
                const int col0 = (EPI == TC_SWIGLU ? tile_n * HALF : tile_n * BN) + half * OWN;
#pragma unroll
                for (int c = 0; c < OWN; c += 64) {
                    constexpr int W = OWN % 32 == 0 ? 32 : 16;   // columns a turn
                    const int n_cols = OWN - c < 64 ? OWN - c : 64;
#pragma unroll
                    for (int e = 0; e < n_cols; e += W) {
                        uint32_t packed[W / 2];
                        if constexpr (EPI == TC_SWIGLU) {
                            uint32_t g[W], u[W];
                            tmem_load_two(lane_base + half * OWN + c + e, lane_base + HALF + half * OWN + c + e, g, u);
#pragma unroll
                            for (int j = 0; j < W / 2; ++j)
                                packed[j] = pack_bf16(fast_silu(__uint_as_float(g[2 * j])) * __uint_as_float(u[2 * j]),
                                                      fast_silu(__uint_as_float(g[2 * j + 1])) * __uint_as_float(u[2 * j + 1]));
                        } else {
                            uint32_t v[W];
                            if constexpr (W == 32) tmem_load_32(lane_base + half * OWN + c + e, v);
                            else tmem_load_16(lane_base + half * OWN + c + e, v);
                            const int beyond = col0 + c + e - n_out;   // of the turn's first column
                            if (tail.n_tail > 0 && beyond > -W && beyond < tail.n_tail && row0 + lane < M) {
                                float* dst = tail.tail + (size_t)(row0 + lane) * tail.n_tail + beyond;
#pragma unroll
                                for (int j = 0; j < W; ++j)
                                    if (beyond + j >= 0 && beyond + j < tail.n_tail) dst[j] = __uint_as_float(v[j]);
                            }
#pragma unroll
                            for (int j = 0; j < W / 2; ++j) packed[j] = pack_bf16(__uint_as_float(v[2 * j]), __uint_as_float(v[2 * j + 1]));
                        }
#pragma unroll
                        for (int j = 0; j < W / 8; ++j)
                            *patch_at(patch, lane, e / 8 + j) = make_uint4(packed[4 * j], packed[4 * j + 1], packed[4 * j + 2], packed[4 * j + 3]);
                    }
                    if (c + 64 >= OWN) sums_read();
                    else __syncwarp();
                    const int pieces = n_cols / 8;
#pragma unroll
                    for (int u = 0; u < pieces; ++u) {
                        const int r = (u * 32 + lane) / pieces, piece = (u * 32 + lane) % pieces, col = col0 + c + 8 * piece;
                        if (row0 + r >= M || col >= n_out) continue;
                        bf16* dst = out + (size_t)(row0 + r) * ldo + col;
                        const uint4* src = patch_at(patch, r, piece);
                        if (EPI != TC_PLAIN || col + 8 <= n_out) {   // (TC_SWIGLU: n_out is a multiple of eight)
                            *reinterpret_cast<uint4*>(dst) = *src;
                        } else {                                    // a ragged last piece: what lies behind the row's columns is not this product's
                            for (int j = 0; j < n_out - col; ++j) dst[j] = reinterpret_cast<const bf16*>(src)[j];
                        }
                    }
                    __syncwarp();
                }
            }
        }
    }
    if (timed_out && lane == 0) atomicOr(err, QF_ERR_COPY_TIMEOUT);
    tc_fence_before();
    __syncthreads();
    cluster_sync();                   // nothing of the other block's reaches into this one any more
    tc_fence_after();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32  %0, %1;" ::"r"(tmem), "r"(512));
}

template <int EPI, int BN, int P = 0>
static int launch_pair(const CUtensorMap& map_a, const void* w, int w_rows, int ldw, void* out, int m, int n_out, int k, int inter,
                       int ldo, int* err, cudaStream_t stream, const TcQkvArgs& qa = TcQkvArgs{}, const TcTail& tail = TcTail{}) {
    constexpr size_t smem = PairGeometry<BN>::smem;
    CUtensorMap map_b;                // boxes of a block's half of a tile's weight rows
    if (!qf_make_map_bf16(&map_b, w, w_rows, k, ldw, BN / 2)) return (int)cudaErrorNotSupported;
    cudaError_t e = cudaFuncSetAttribute(tc_gemm_pair_kernel<EPI, BN, P>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
    const int tile_cols = EPI == TC_SWIGLU ? BN / 2 : BN;
    const int m_tiles = (m + 2 * TC_BM - 1) / (2 * TC_BM), n_tiles = (n_out + tail.n_tail + tile_cols - 1) / tile_cols;
    const int total = m_tiles * n_tiles, pairs = qf_sm_count() / 2;
    // column tiles whose weight rows together take about 32 MB, a quarter of the L2; 4 at least
    long long group_n = (32ll << 20) / ((long long)BN * k * 2);
    group_n = group_n < 4 ? 4 : group_n;
    group_n = group_n > n_tiles ? n_tiles : group_n;
    return (int)launch_pdl(tc_gemm_pair_kernel<EPI, BN, P>, dim3(2 * (total < pairs ? total : pairs)), dim3(TP_THREADS), smem, stream,
                           map_a, map_b, (bf16*)out, m, n_out, k, inter, ldo, m_tiles, n_tiles, (int)group_n, err, qa, tail);
}

// Tiles of 256 columns, or of 192 where the wide ones' last round would leave many pairs idle: a round of the narrow ones takes
// 0.8 of a wide one's time (measured 0.75 at K = 896, 0.81 at 2,048; with the results stored straight to memory, 905 x 9728 x 896: 204
// narrow tiles in three rounds of 74 pairs 18.9 microseconds, 152 wide ones in three rounds 21.4; 1024 x 22016 x 2048: seven rounds
// 67.7, five 65.0). Tiles of 128 columns were never the fastest (23.5 and 86.4).
static int pair_columns(int epilogue, int m, int n_out) {
    const long long pairs = qf_sm_count() / 2 > 0 ? qf_sm_count() / 2 : 1, m_tiles = (m + 255) / 256;
    auto rounds = [&](int columns) {
        const int cols = epilogue == TC_SWIGLU ? columns / 2 : columns;
        return (m_tiles * ((n_out + cols - 1) / cols) + pairs - 1) / pairs;
    };
    return 4 * rounds(192) < 5 * rounds(256) ? 192 : 256;
}

template <int EPI>
static int launch_persistent(const CUtensorMap& map_a, const void* w, int w_rows, int ldw, void* out, int m, int n_out, int k, int inter,
                             int ldo, int* err, cudaStream_t stream) {
    return pair_columns(EPI, m, n_out) == 192 ? launch_pair<EPI, 192>(map_a, w, w_rows, ldw, out, m, n_out, k, inter, ldo, err, stream)
                                              : launch_pair<EPI, 256>(map_a, w, w_rows, ldw, out, m, n_out, k, inter, ldo, err, stream);
}

template <int EPI, int BN>
static int launch_tc(const CUtensorMap& map_a, const CUtensorMap& map_b, void* out, int m, int n_out, int k, int inter, int ldo,
                     int* err, dim3 grid, cudaStream_t stream) {
    const size_t smem = TcGeometry<BN>::smem;
    cudaError_t e = cudaFuncSetAttribute(tc_gemm_kernel<EPI, BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
    tc_gemm_kernel<EPI, BN><<<grid, TC_THREADS, smem, stream>>>(map_a, map_b, (bf16*)out, m, n_out, k, inter, ldo, TcQkvArgs{}, err,
                                                                TcGroups{});
    return (int)cudaGetLastError();
}

template <int EPI>
static int launch_tc_grouped(const CUtensorMap& map_a, const CUtensorMap& map_b, void* out, int m, int n_out, int k, int inter, int ldo,
                             int* err, dim3 grid, const TcGroups& groups, cudaStream_t stream) {
    const size_t smem = TcGeometry<128>::smem;
    cudaError_t e = cudaFuncSetAttribute(tc_gemm_kernel<EPI, 128>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
    tc_gemm_kernel<EPI, 128><<<grid, TC_THREADS, smem, stream>>>(map_a, map_b, (bf16*)out, m, n_out, k, inter, ldo, TcQkvArgs{}, err, groups);
    return (int)cudaGetLastError();
}

// The grouped form (see TcGroups): a [m][lda] rows sorted by group, w [n_groups * n][ldw] the groups' weights one after the
// other (n rows each; TC_SWIGLU: n = 2 * inter, a group's gate rows then its up rows), out [m][ldo] with n columns
// (TC_SWIGLU: inter). The plan's tiles have 128 rows; max_tiles bounds their number. The conditions of qf_tc_gemm hold.
// gate_limit > 0 (TC_SWIGLU only): the clamped gate of TcGroups instead of the SwiGLU.
QF_EXPORT int qf_tc_gemm_grouped_gated(int epilogue, const void* a, int lda, const void* w, int ldw, int n_groups, void* out, int ldo,
                                       int m, int n, int k, const int* tile_group, const int* tile_row0, const int* offsets,
                                       const int* n_tiles, int max_tiles, const float* row_scale, float gate_limit, float gate_alpha,
                                       int* err, cudaStream_t stream) {
    if (m <= 0 || n <= 0 || n_groups <= 0) return 0;
    if (k <= 0 || k % 8 || lda % 8 || ldw % 8 || ldo % 8 || !tile_group || max_tiles <= 0 || max_tiles > 65535) return (int)cudaErrorInvalidValue;
    if (((uintptr_t)a | (uintptr_t)w | (uintptr_t)out) % 16) return (int)cudaErrorInvalidValue;
    CUtensorMap map_a, map_b;
    if (!qf_make_map_bf16(&map_a, a, m, k, lda, TC_BM) || !qf_make_map_bf16(&map_b, w, (long long)n_groups * n, k, ldw, 64))
        return (int)cudaErrorNotSupported;
    TcGroups groups{tile_group, tile_row0, offsets, n_tiles, row_scale, n, gate_limit, gate_alpha};
    if (gate_limit > 0.f && epilogue != TC_SWIGLU) return (int)cudaErrorInvalidValue;
    if (epilogue == TC_SWIGLU) {
        if (n % 2 || (n / 2) % 8) return (int)cudaErrorInvalidValue;
        const int inter = n / 2;
        return launch_tc_grouped<TC_SWIGLU>(map_a, map_b, out, m, inter, k, inter, ldo, err, dim3((inter + 63) / 64, max_tiles), groups, stream);
    }
    if (epilogue != TC_PLAIN || row_scale) return (int)cudaErrorInvalidValue;
    return launch_tc_grouped<TC_PLAIN>(map_a, map_b, out, m, n, k, 0, ldo, err, dim3((n + 127) / 128, max_tiles), groups, stream);
}

QF_EXPORT int qf_tc_gemm_grouped(int epilogue, const void* a, int lda, const void* w, int ldw, int n_groups, void* out, int ldo,
                                 int m, int n, int k, const int* tile_group, const int* tile_row0, const int* offsets,
                                 const int* n_tiles, int max_tiles, const float* row_scale, int* err, cudaStream_t stream) {
    return qf_tc_gemm_grouped_gated(epilogue, a, lda, w, ldw, n_groups, out, ldo, m, n, k, tile_group, tile_row0, offsets, n_tiles,
                                    max_tiles, row_scale, 0.f, 0.f, err, stream);
}

static int g_persistent = 1;
// A measuring aid: 0 sends every product to the one-tile-per-block kernel.
QF_EXPORT void qf_tc_gemm_set_persistent(int on) { g_persistent = on; }

// Whether a product of these sizes has tiles for every SM and so runs in the persistent kernel (n as in qf_tc_gemm), and the
// columns of its tiles there.
QF_EXPORT int qf_tc_gemm_pair_columns(int epilogue, int m, int n) { return pair_columns(epilogue, m, epilogue == TC_SWIGLU ? n / 2 : n); }
QF_EXPORT int qf_tc_gemm_is_persistent(int epilogue, int m, int n) {
    if (!g_persistent || m <= 0 || n <= 0) return 0;
    const long long m_tiles = (m + TC_BM - 1) / TC_BM;
    const long long n_tiles = epilogue == TC_SWIGLU ? (n / 2 + 127) / 128 : (n + 255) / 256;
    return m_tiles * n_tiles >= qf_sm_count();
}

// a [m][lda], w [n][ldw] (for TC_SWIGLU: n = 2 * inter, gate rows then up rows), out [m][ldo] with n columns
// (TC_SWIGLU: inter columns). Needs k, lda, ldw, ldo multiples of 8 and 16-byte aligned bases; for TC_SWIGLU
// inter a multiple of 8. Returns cudaErrorInvalidValue for what it does not take, cudaErrorNotSupported when
// the driver has no tensor-map encoder.
QF_EXPORT int qf_tc_gemm(int epilogue, const void* a, int lda, const void* w, int ldw, void* out, int ldo, int m, int n, int k,
                         int* err, cudaStream_t stream) {
    if (m <= 0 || n <= 0) return 0;
    if (k <= 0 || k % 8 || lda % 8 || ldw % 8 || ldo % 8) return (int)cudaErrorInvalidValue;
    if (((uintptr_t)a | (uintptr_t)w | (uintptr_t)out) % 16) return (int)cudaErrorInvalidValue;
    if (epilogue != TC_PLAIN && (epilogue != TC_SWIGLU || n % 2 || (n / 2) % 8)) return (int)cudaErrorInvalidValue;
    CUtensorMap map_a, map_b;         // (a launch on pairs makes the weights' map itself, with its own boxes)
    if (!qf_make_map_bf16(&map_a, a, m, k, lda, TC_BM)) return (int)cudaErrorNotSupported;
    // wide tiles when there are enough of them to fill the SMs; narrow ones otherwise
    const int inter = n / 2, m_tiles = (m + TC_BM - 1) / TC_BM;
    const bool wide = (long long)m_tiles * (epilogue == TC_SWIGLU ? (inter + 127) / 128 : (n + 255) / 256) >= qf_sm_count();
    if (wide && g_persistent)
        return epilogue == TC_SWIGLU ? launch_persistent<TC_SWIGLU>(map_a, w, n, ldw, out, m, inter, k, inter, ldo, err, stream)
                                     : launch_persistent<TC_PLAIN>(map_a, w, n, ldw, out, m, n, k, 0, ldo, err, stream);
    if (!qf_make_map_bf16(&map_b, w, n, k, ldw, 64)) return (int)cudaErrorNotSupported;
    if (epilogue == TC_SWIGLU)
        return wide ? launch_tc<TC_SWIGLU, 256>(map_a, map_b, out, m, inter, k, inter, ldo, err, dim3((inter + 127) / 128, m_tiles), stream)
                    : launch_tc<TC_SWIGLU, 128>(map_a, map_b, out, m, inter, k, inter, ldo, err, dim3((inter + 63) / 64, m_tiles), stream);
    return wide ? launch_tc<TC_PLAIN, 256>(map_a, map_b, out, m, n, k, 0, ldo, err, dim3((n + 255) / 256, m_tiles), stream)
                : launch_tc<TC_PLAIN, 128>(map_a, map_b, out, m, n, k, 0, ldo, err, dim3((n + 127) / 128, m_tiles), stream);
}


// The QKV product with bias, rotation and cache write in its epilogue (see TcQkvArgs): a [m][lda] against
// w [(n_heads + 2 kv_heads) * head_dim][ldw]. Head sizes 32, 64 and 128 (whole heads per tile of 128 columns); k, lda, ldw
// multiples of 8, 16-byte aligned bases, and rows of q_out and cache pages that keep 16-byte alignment. Returns
// cudaErrorInvalidValue for what it does not take, cudaErrorNotSupported when the driver has no tensor-map encoder.
QF_EXPORT int qf_tc_gemm_qkv(const void* a, int lda, const void* w, int ldw, int m, int k, const TcQkvArgs* args, int* err,
                             cudaStream_t stream) {
    const TcQkvArgs& q = *args;
    const int d = q.head_dim, n = (q.n_heads + 2 * q.kv_heads) * d;
    if (m <= 0 || n <= 0) return 0;
    if (d != 32 && d != 64 && d != 128) return (int)cudaErrorInvalidValue;
    if (k <= 0 || k % 8 || lda % 8 || ldw % 8 || q.page_elems % 8) return (int)cudaErrorInvalidValue;
    if (((uintptr_t)a | (uintptr_t)w | (uintptr_t)q.q_out | (uintptr_t)q.kv_base) % 16) return (int)cudaErrorInvalidValue;
    CUtensorMap map_a, map_b;
    if (!qf_make_map_bf16(&map_a, a, m, k, lda, TC_BM) || !qf_make_map_bf16(&map_b, w, n, k, ldw, 64)) return (int)cudaErrorNotSupported;
    const size_t smem = TcGeometry<128>::smem;
    cudaError_t e = cudaFuncSetAttribute(tc_gemm_kernel<TC_QKV, 128>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
    dim3 grid((n + 127) / 128, (m + TC_BM - 1) / TC_BM);
    tc_gemm_kernel<TC_QKV, 128><<<grid, TC_THREADS, smem, stream>>>(map_a, map_b, nullptr, m, n, k, 0, 0, q, err, TcGroups{});
    return (int)cudaGetLastError();
}

// Columns of the tiles of the pairs' QKV product (whole heads), and whether its tiles keep the pairs at work. A round of tiles of 192,
// 128 and 64 columns takes 0.85, 0.75 and 0.66 of the time of one of 256 (905 x 1152 x 896: 9.4, 8.6, 8.5 and 11.1 microseconds, a round each;
// 8192 x 1152 x 896: 24.1 in three rounds, 27.1 in four, 40.6 in eight, 27.2 in three).
static int qkv_columns(int m, int n, int d, float* busy) {
    const long long pairs = qf_sm_count() / 2 > 0 ? qf_sm_count() / 2 : 1, m_tiles = (m + 255) / 256;
    const struct { int columns; float round; } forms[] = {{256, 1.f}, {192, 0.85f}, {128, 0.75f}, {64, 0.66f}};
    int best = 0;
    float least = 0.f;
    for (const auto& f : forms) {
        if (f.columns % d) continue;
        const long long tiles = m_tiles * ((n + f.columns - 1) / f.columns), rounds = (tiles + pairs - 1) / pairs;
        if (best == 0 || f.round * (float)rounds < least) {
            best = f.columns, least = f.round * (float)rounds;
            *busy = (float)tiles / (float)(rounds * pairs);
        }
    }
    return best;
}

// Whether qf_tc_gemm_qkv_pairs is the faster way for these sizes, against the library's product and the rotation kernel behind it: beyond 512
// rows where its tiles keep three quarters of the pairs at work (7358 x 2560 x 2048: 56 microseconds against 70; 1536 x 2560 x 2048 19.2
// and 22.0, 60 of 74 pairs; 2048 x 2560 x 2048, 80 of 148, 28.7 and 26.4; 1536 x 4608 x 3584, 108 of 148, 47.8 and 44.5; 256 x 4608 x 3584
// 20.7 and 18.4), and for heads of 64 with weights of up to 4 MB and K up to 1,280 columns and to the product's own always (1152 x 896: 7.5
// against 8.0 for 64 rows, 8.8 and 10.1 for 900). A narrow tile's time is its copies of A, K by K, while the library cuts a long K
// among blocks, so tiles of 64 columns are the faster way up to K = 1,536 and of 128 up to 3,072. With the norm kernel ahead, this
// way / the other: 64 x 512 x 4096 18.8 / 12.4, 64 x 512 x 1024 9.4 / 8.9, 300 x 1024 x 2048 12.6 / 11.2, 2048 x 512 x 3072 19.9 / 17.3 and
// 1300 x 1280 x 4096 24.1 / 22.5; within the lines 900 x 1024 x 1536 12.5 / 12.5, 700 x 2560 x 2048 15.4 / 17.6, 4096 x 512 x 3072 28.2 / 30.5.
QF_EXPORT int qf_tc_gemm_qkv_pairs_pays(int m, int n, int k, int head_dim) {
    if (m <= 0 || n <= 0 || (head_dim != 64 && head_dim != 128)) return 0;
    if (head_dim == 64 && (long long)n * k * 2 <= (4ll << 20) && k <= 1280 && k <= n) return 1;
    float busy = 0.f;
    const int columns = qkv_columns(m, n, head_dim, &busy);
    return m > 512 && busy >= 0.75f && (columns > 128 || k <= 24 * columns);
}

// The same on pairs of SMs, with the angles worked out in the epilogue (args->inv_freq; args->angles is not read): head sizes 64 and 128.
QF_EXPORT int qf_tc_gemm_qkv_pairs(const void* a, int lda, const void* w, int ldw, int m, int k, const TcQkvArgs* args, int* err,
                                   cudaStream_t stream) {
    const TcQkvArgs& q = *args;
    const int d = q.head_dim, n = (q.n_heads + 2 * q.kv_heads) * d;
    if (m <= 0 || n <= 0) return 0;
    if (d != 64 && d != 128) return (int)cudaErrorInvalidValue;
    if (k <= 0 || k % 8 || lda % 8 || ldw % 8 || q.page_elems % 8) return (int)cudaErrorInvalidValue;
    if (((uintptr_t)a | (uintptr_t)w | (uintptr_t)q.q_out | (uintptr_t)q.kv_base | (uintptr_t)q.bias) % 16) return (int)cudaErrorInvalidValue;
    CUtensorMap map_a;
    if (!qf_make_map_bf16(&map_a, a, m, k, lda, TC_BM)) return (int)cudaErrorNotSupported;
#define QF_QKV(BN, P) launch_pair<TC_QKV, BN, P>(map_a, w, n, ldw, nullptr, m, n, k, 0, 0, err, stream, q)
    float busy;
    const int columns = qkv_columns(m, n, d, &busy);
    if (d == 128) return columns == 256 ? QF_QKV(256, 64) : QF_QKV(128, 64);
    return columns == 256 ? QF_QKV(256, 32) : columns == 192 ? QF_QKV(192, 32) : columns == 128 ? QF_QKV(128, 32) : QF_QKV(64, 32);
#undef QF_QKV
}

// a [m][lda] against w [n + n_tail][ldw]: the first n columns to out [m][ldo] in bfloat16, the others in float32 to tail [m][n_tail]. The
// conditions of qf_tc_gemm, and n a multiple of 8.
QF_EXPORT int qf_tc_gemm_tail(const void* a, int lda, const void* w, int ldw, void* out, int ldo, float* tail, int m, int n, int n_tail, int k,
                              int* err, cudaStream_t stream) {
    if (m <= 0) return 0;
    if (n <= 0 || n_tail <= 0 || n % 8 || k <= 0 || k % 8 || lda % 8 || ldw % 8 || ldo % 8) return (int)cudaErrorInvalidValue;
    if (((uintptr_t)a | (uintptr_t)w | (uintptr_t)out) % 16) return (int)cudaErrorInvalidValue;
    CUtensorMap map_a;
    if (!qf_make_map_bf16(&map_a, a, m, k, lda, TC_BM)) return (int)cudaErrorNotSupported;
    const TcTail t{tail, n_tail};
    return pair_columns(TC_PLAIN, m, n + n_tail) == 192 ? launch_pair<TC_PLAIN, 192>(map_a, w, n + n_tail, ldw, out, m, n, k, 0, ldo, err, stream, TcQkvArgs{}, t)
                                                        : launch_pair<TC_PLAIN, 256>(map_a, w, n + n_tail, ldw, out, m, n, k, 0, ldo, err, stream, TcQkvArgs{}, t);
}
