// The recurrence of a matrix state per head with one decay per token and head, written out over chunks of tokens:
//
//   S <- decay_t S + take_t k_t v_t^T,  n <- decay_t n + take_t k_t,   y_t = S^T q_t,  nq_t = n . q_t
//
// (`outer_state_scan_kernel` of recurrent.cu walks the same recurrence token by token.) With i, j tokens of a chunk and
// W_ij = take_j decay_(j+1) .. decay_i, the chunk's outputs are
//   y_i = (decay_0 .. decay_i) S0^T q_i + sum_{j <= i} W_ij (q_i . k_j) v_j
// and its state afterwards is  (decay_0 .. decay_last) S0 + sum_j W_(last)j k_j v_j^T.  Three launches: (1) `parts`: every
// chunk's own sum; (2) `chain`: the states before every chunk; (3) `outputs`.
// What bounds it: the scan is a chain of one update per token (0.12 microseconds each, whatever the width of the GPU); here
// the chain is one step per 128 tokens and everything else is products. Measured on one prompt of 2,048 tokens, 7 heads of
// 64 x 128: 200 -> 29 microseconds; 32 heads of 128 x 128: 427 -> 97.
// (One block walking a sequence's chunks with its tile of S in registers moves fewer bytes than parts and chain, and took
// 46 and 105 microseconds where these take 16 and 71: a link of that chain is a chunk's products, 3 microseconds.)
// 128 tokens per chunk: with 64 the records (32 heads x 64 KB a chunk) are twice the bytes, with 256 the products inside
// a chunk outgrow the others.
//
// Precision. q, k and v are bfloat16 numbers, so q . k is a bfloat16 product with float32 sums as it stands. Everything that
// is float32 in the recurrence stays so: a float32 operand (S, the weighted scores, the weighted values) is cut into three
// bfloat16 numbers whose sum is that operand exactly (eight bits of the significand each), one product for each. The
// sums over tokens and rows are float32 additions of what the tensor cores make of 16 at a time (MmaFirst): errors against 64 bits,
// outputs / states, 2,048 tokens of 7 heads of 64 x 128 with an mLSTM's gates 9.2e-8 / 6.3e-8, token by token 1.20e-7 / 8.2e-8
// (sums left to the tensor cores: 4.4e-7 / 9.0e-8). The weights are products of decays, never quotients or differences of
// logarithms: a chunk is cut into eighths of 16 tokens, and W_ij is (decays from the start of i's eighth to i) x (decays of the
// whole eighths between) x (decays behind j to the end of j's eighth), each factor at most as large as the decays make it, so
// nothing overflows or cancels.
#include "chunks.cuh"

#define SC_CHUNK 128
#define SC_SUB 16
#define SC_VT 64              // columns of v of a block, both kernels
#define SC_OUT_THREADS 256    // of a block of outputs: a warp per eighth

struct ChunkArgs {
    const bf16 *q, *k, *v;
    int q_stride, k_stride, v_stride;
    const float *decay, *take;      // [T][heads]; or, with rate_log, decay holds the pre-activations (rows gate_stride apart) of
    const float *dt_bias, *rate_log;  // dt = softplus(pre + dt_bias), decay = exp(-exp(rate_log) dt), take = dt
    int gate_stride;
    const int *cu_q, *slots;
    float* state;
    long long slot_stride, s_offset, n_offset;   // n_offset < 0: no vector n
    int n_heads, n_groups, vdim;
    float q_scale;
    float *records, *n_records, *whole;   // [record][heads][vdim][D], [record][heads][D], [record][heads]
    float *y, *nq;
    Portion portion;
};

// A token's decay and take (the arithmetic of `decay_gates_kernel` in recurrent.cu where they come as pre-activations: a launch
// less, 4 microseconds of the device's time and 7 of the host's).
__device__ __forceinline__ float2 gates_of(const ChunkArgs& a, int token, int head) {
    const float x = a.decay[(size_t)token * a.gate_stride + head];
    if (!a.rate_log) return make_float2(x, a.take[(size_t)token * a.gate_stride + head]);
    const float z = x + a.dt_bias[head], dt = fmaxf(z, 0.f) + log1pf(expf(-fabsf(z)));
    return make_float2(expf(-expf(a.rate_log[head]) * dt), dt);
}

// ------------------------------------------------------------------------------------------------------------------
// (1) A chunk's own part of the state after it, sum_j W_(last)j k_j v_j^T, for 64 columns of v (16 per warp) and all rows of S.
// The products are S^T += (weighted v)^T k: rows of v, columns of k, so that a warp weights and cuts its own 16 columns of v
// and nobody else's (about 400 instructions, against 3 D / 8 x 8 products). The fifth warp, where it is launched, makes the
// part of n beside them (blocks of the first 64 columns only).
template <int D>
__global__ void __launch_bounds__(160)
chunk_parts_kernel(const ChunkArgs a) {
    grid_chain_entry();
    extern __shared__ __align__(128) unsigned char sc_smem[];
    unsigned char* k_s = sc_smem;                              // [128][D]
    unsigned char* v_s = sc_smem + SC_CHUNK * D * 2;           // [128][64]
    __shared__ __align__(16) float weight_s[SC_CHUNK];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, chunk = a.portion.chunk0 + (int)blockIdx.x, seq = blockIdx.z;
    const int v_tiles = a.vdim / SC_VT, head = blockIdx.y / v_tiles, v0 = (blockIdx.y % v_tiles) * SC_VT;
    const int t0 = a.cu_q[seq] + chunk * SC_CHUNK, n_here = min(SC_CHUNK, a.cu_q[seq + 1] - t0);
    if (n_here <= 0) return;
    const int group = head / (a.n_heads / a.n_groups);
    fetch_tile<SC_CHUNK, SC_VT>(v_s, a.v + (size_t)t0 * a.v_stride + head * a.vdim + v0, a.v_stride, n_here, threadIdx.x, blockDim.x);
    fetch_tile<SC_CHUNK, D>(k_s, a.k + (size_t)t0 * a.k_stride + group * D, a.k_stride, n_here, threadIdx.x, blockDim.x);
    cp_async_commit();
    const long long record = record_of<SC_CHUNK>(a.portion, a.cu_q, seq, chunk) * a.n_heads + head;
    if (warp == 0) {
        // What a token adds counts at the chunk's end: its take and the decays behind it. Four neighbouring tokens per lane,
        // the products over the lanes above by shuffles.
        float dec[4], w[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const float2 gate = 4 * lane + e < n_here ? gates_of(a, t0 + 4 * lane + e, head) : make_float2(1.f, 0.f);
            dec[e] = gate.x, w[e] = gate.y;
        }
        Running inclusive{dec[0], 0.f};
#pragma unroll
        for (int e = 1; e < 4; ++e) inclusive.times(dec[e]);
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const Running above{__shfl_down_sync(0xffffffffu, inclusive.value, o), __shfl_down_sync(0xffffffffu, inclusive.rest, o)};
            if (lane + o < 32) inclusive.times(above);
        }
        Running behind{__shfl_down_sync(0xffffffffu, inclusive.value, 1), __shfl_down_sync(0xffffffffu, inclusive.rest, 1)};
        if (lane == 31) behind = Running{1.f, 0.f};
#pragma unroll
        for (int e = 3; e >= 0; --e) {
            w[e] = behind.of(w[e]);
            behind.times(dec[e]);
        }
        *reinterpret_cast<float4*>(weight_s + 4 * lane) = make_float4(w[0], w[1], w[2], w[3]);
        if (lane == 0 && v0 == 0) a.whole[record] = inclusive.value + inclusive.rest;
    }
    cp_async_wait<0>();
    __syncthreads();
    if (warp == 4) {
        if (v0 != 0) return;
#pragma unroll
        for (int u = 0; u < D / 32; ++u) {
            const int d = lane + 32 * u;
            float sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 8
            for (int j = 0; j < SC_CHUNK; ++j)
                sum[j & 3] = fmaf(weight_s[j], __bfloat162float(*reinterpret_cast<const bf16*>(k_s + tile_at<D>(j, d >> 3) + (d & 7) * 2)), sum[j & 3]);
            a.n_records[record * D + d] = (sum[0] + sum[1]) + (sum[2] + sum[3]);
        }
        return;
    }
    const int g = lane >> 2, t2 = (lane & 3) * 2;
    float acc[D / 8][4];
#pragma unroll
    for (int nt = 0; nt < D / 8; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[nt][e] = 0.f;
#pragma unroll 2
    for (int kk = 0; kk < SC_CHUNK / 16; ++kk) {
        // (v^T): rows of v's 16 columns, columns of 16 tokens
        uint32_t raw[4], hi[4], mid[4], lo[4];
        ldmatrix_x4_trans(raw, v_s + tile_at<SC_VT>(kk * 16 + (lane & 7) + ((lane >> 4) << 3), warp * 2 + ((lane >> 3) & 1)));
        const float2 w0 = *reinterpret_cast<const float2*>(weight_s + kk * 16 + t2);
        const float2 w1 = *reinterpret_cast<const float2*>(weight_s + kk * 16 + 8 + t2);
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const float2 w = r < 2 ? w0 : w1;
            const Thirds x = thirds(lower_bf16(raw[r]) * w.x, upper_bf16(raw[r]) * w.y);
            hi[r] = x.hi, mid[r] = x.mid, lo[r] = x.lo;
        }
#pragma unroll
        for (int n2 = 0; n2 < D / 16; n2 += 2) {   // eight sums in turn: no product waits for the one before it
            uint32_t b[2][4];
            float sum[4][4], low[4][4];
#pragma unroll
            for (int np = 0; np < 2; ++np) ldmatrix_x4_trans(b[np], k_s + tile_at<D>(kk * 16 + (lane & 15), (n2 + np) * 2 + (lane >> 4)));
            auto part = [&](auto mma, float (&to)[4][4], const uint32_t (&x)[4]) {
#pragma unroll
                for (int np = 0; np < 2; ++np) {
                    mma(to[2 * np], x, b[np][0], b[np][1]);
                    mma(to[2 * np + 1], x, b[np][2], b[np][3]);
                }
            };
            part(MmaFirst{}, low, lo);
            part(MmaFirst{}, sum, hi);
            part(MmaNext{}, low, mid);
            add_sums(sum, low);
            add_sums(acc + 2 * n2, sum);
        }
    }
    float* rec = a.records + record * D * a.vdim + (size_t)(v0 + warp * 16 + g) * D + t2;
#pragma unroll
    for (int nt = 0; nt < D / 8; ++nt) {
        *reinterpret_cast<float2*>(rec + nt * 8) = make_float2(acc[nt][0], acc[nt][1]);
        *reinterpret_cast<float2*>(rec + 8 * D + nt * 8) = make_float2(acc[nt][2], acc[nt][3]);
    }
}

// ------------------------------------------------------------------------------------------------------------------
// (2) The states before every chunk, in the place of the chunks' own parts, and the one after the last in the sequence's state: a
// thread takes four neighbouring rows of S in one column of v and walks the chunks with eight records' loads on their way (a
// link of the chain is one multiply-add; the records come from L2). A warp's 32 threads are 8 columns x 16 rows: whole
// sectors of the records and, transposed, of the state. The last block of a head takes n.
template <int D>
__global__ void __launch_bounds__(256)
chunk_chain_kernel(const ChunkArgs a) {
    grid_chain_entry();
    constexpr int AHEAD = 8;
    const int lane = threadIdx.x & 31, head = blockIdx.y, seq = blockIdx.z;
    const int len = a.cu_q[seq + 1] - a.cu_q[seq], slot = a.slots[seq];
    const int chunk0 = a.portion.chunk0, left = (len + SC_CHUNK - 1) / SC_CHUNK - chunk0;
    const int n_chunks = a.portion.each > 0 ? min(left, a.portion.each) : left;
    if (n_chunks <= 0) return;
    const long long first = record_of<SC_CHUNK>(a.portion, a.cu_q, seq, chunk0) * a.n_heads + head;
    // the sequence's state, or what stands for it between portions (zeros before the first)
    const bool held = slot >= 0;
    float* kept = held ? a.state + slot * a.slot_stride : a.portion.carry ? a.portion.carry + (long long)seq * a.n_heads * D * (a.vdim + 1) : nullptr;
    const long long s_offset = held ? a.s_offset : 0, n_offset = held ? a.n_offset : (long long)a.n_heads * D * a.vdim;
    const bool fresh = !kept || (!held && chunk0 == 0);
    const float* whole = a.whole + first;
    const int item = (int)blockIdx.x * 8 + (threadIdx.x >> 5);   // (8 columns of v, 16 rows of S)
    const int items = a.vdim / 8 * (D / 16);
    if (item >= items) {
        if (item != items || a.n_offset < 0) return;   // one warp of the grid carries n
        float* n_kept = kept ? kept + n_offset + (long long)head * D : nullptr;
        for (int d = lane; d < D; d += 32) {
            float n = fresh ? 0.f : n_kept[d];
            for (int c = 0; c < n_chunks; ++c) {
                float* at = a.n_records + (first + (long long)c * a.n_heads) * D + d;
                const float part = *at;
                *at = n;
                n = fmaf(n, whole[(long long)c * a.n_heads], part);
            }
            if (n_kept) n_kept[d] = n;
        }
        return;
    }
    const int col = item / (D / 16) * 8 + (lane >> 2), row = item % (D / 16) * 16 + (lane & 3) * 4;
    const long long pitch = (long long)a.n_heads * D * a.vdim;
    float* at = a.records + first * D * a.vdim + (size_t)col * D + row;
    float* s_kept = kept ? kept + s_offset + ((long long)head * D + row) * a.vdim + col : nullptr;
    float s[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) s[e] = fresh ? 0.f : s_kept[(size_t)e * a.vdim];
    float4 part[AHEAD];
    float w[AHEAD];
#pragma unroll
    for (int u = 0; u < AHEAD; ++u)
        if (u < n_chunks) {
            part[u] = *reinterpret_cast<const float4*>(at + u * pitch);
            w[u] = whole[(long long)u * a.n_heads];
        }
    for (int c0 = 0; c0 < n_chunks; c0 += AHEAD, at += AHEAD * pitch) {
#pragma unroll
        for (int u = 0; u < AHEAD; ++u)
            if (c0 + u < n_chunks) {
                const float4 mine = part[u];
                const float all = w[u];
                if (c0 + u + AHEAD < n_chunks) {
                    part[u] = *reinterpret_cast<const float4*>(at + (u + AHEAD) * pitch);
                    w[u] = whole[(long long)(c0 + u + AHEAD) * a.n_heads];
                }
                *reinterpret_cast<float4*>(at + u * pitch) = make_float4(s[0], s[1], s[2], s[3]);
                s[0] = fmaf(s[0], all, mine.x), s[1] = fmaf(s[1], all, mine.y);
                s[2] = fmaf(s[2], all, mine.z), s[3] = fmaf(s[3], all, mine.w);
            }
    }
    if (s_kept) {
#pragma unroll
        for (int e = 0; e < 4; ++e) s_kept[(size_t)e * a.vdim] = s[e];
    }
}

// ------------------------------------------------------------------------------------------------------------------
// (3) Outputs of one chunk, one head, 64 columns of v. Eight warps, one for each of the chunk's eighths (16 tokens each), dealt so that
// the two that share a scheduler have the same part of the triangle between them. (Four warps of two eighths each load every
// fragment of a key, a value or the state once for both, and leave an SM eight warps, which waited for their own instructions: 34
// chunks of 32 heads of 128 x 128 in 132 microseconds, 124 so.) First S0^T q on the record's three parts, scaled by the decays up to the row; then, 16 earlier tokens at a time, scores, weights,
// and the products with v added on top. Queries move to registers before the keys arrive in the same place, so that two
// blocks fit an SM.
template <int D>
__global__ void __launch_bounds__(SC_OUT_THREADS, 2)
chunk_outputs_kernel(const ChunkArgs a) {
    grid_chain_entry();
    extern __shared__ __align__(128) unsigned char sc_smem[];
    constexpr int QK_BYTES = SC_CHUNK * D * 2, V_BYTES = SC_CHUNK * SC_VT * 2, S_PART = SC_VT * D * 2, SUBS = SC_CHUNK / SC_SUB;
    unsigned char* qk_s = sc_smem;                 // [128][D]: the queries, then the keys
    unsigned char* v_s = qk_s + QK_BYTES;          // [128][64]
    unsigned char* s_s = v_s + V_BYTES;            // [3][64][D]: the state before the chunk, transposed, in three parts
    __shared__ __align__(16) float decay_s[SC_CHUNK], upto_s[SC_CHUNK], behind_s[SC_CHUNK], n_s[D];
    __shared__ float inner_s[SUBS][SC_SUB][SC_SUB + 1];   // W of one eighth: row, column
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, chunk = a.portion.chunk0 + (int)blockIdx.x, seq = blockIdx.z;
    const int v_tiles = a.vdim / SC_VT, head = blockIdx.y / v_tiles, v0 = (blockIdx.y % v_tiles) * SC_VT;
    const int t0 = a.cu_q[seq] + chunk * SC_CHUNK, n_here = min(SC_CHUNK, a.cu_q[seq + 1] - t0);
    if (n_here <= 0) return;
    const int group = head / (a.n_heads / a.n_groups);
    const bool with_n = a.n_offset >= 0 && v0 == 0;
    const long long record = record_of<SC_CHUNK>(a.portion, a.cu_q, seq, chunk) * a.n_heads + head;

    fetch_tile<SC_CHUNK, D>(qk_s, a.q + (size_t)t0 * a.q_stride + group * D, a.q_stride, n_here, threadIdx.x, SC_OUT_THREADS);
    cp_async_commit();
    fetch_tile<SC_CHUNK, SC_VT>(v_s, a.v + (size_t)t0 * a.v_stride + head * a.vdim + v0, a.v_stride, n_here, threadIdx.x, SC_OUT_THREADS);
    cp_async_commit();
    const float2 gate = threadIdx.x < n_here ? gates_of(a, t0 + threadIdx.x, head) : make_float2(1.f, 0.f);   // this thread's token
    const float my_take = gate.y;
    if (threadIdx.x < SC_CHUNK) decay_s[threadIdx.x] = gate.x;
    if (with_n && threadIdx.x < D) n_s[threadIdx.x] = a.n_records[record * D + threadIdx.x];
    const float* rec = a.records + record * D * a.vdim + (size_t)v0 * D;
#pragma unroll
    for (int half = 0; half < 2; ++half) {
        constexpr int EACH = SC_VT * D / 4 / SC_OUT_THREADS / 2;
        float4 held[EACH];
#pragma unroll
        for (int u = 0; u < EACH; ++u) held[u] = *reinterpret_cast<const float4*>(rec + 4 * (threadIdx.x + SC_OUT_THREADS * (half * EACH + u)));
#pragma unroll
        for (int u = 0; u < EACH; ++u) {
            const int i = 4 * (threadIdx.x + SC_OUT_THREADS * (half * EACH + u)), row = i / D, col = i % D;
            const Thirds x = thirds(held[u].x, held[u].y), z = thirds(held[u].z, held[u].w);
            unsigned char* at = s_s + tile_at<D>(row, col >> 3) + (col & 7) * 2;
            *reinterpret_cast<uint2*>(at) = make_uint2(x.hi, z.hi);
            *reinterpret_cast<uint2*>(at + S_PART) = make_uint2(x.mid, z.mid);
            *reinterpret_cast<uint2*>(at + 2 * S_PART) = make_uint2(x.lo, z.lo);
        }
    }
    cp_async_wait<1>();
    __syncthreads();

    const int tile = warp < 4 ? warp : 11 - warp;     // this warp's eighth
    const int g = lane >> 2, t2 = (lane & 3) * 2;
    uint32_t q_frag[D / 16][4];
#pragma unroll
    for (int kd = 0; kd < D / 16; ++kd) ldmatrix_x4(q_frag[kd], qk_s + tile_at<D>(tile * 16 + (lane & 15), kd * 2 + (lane >> 4)));
    if (threadIdx.x < SC_CHUNK) {   // the weights' factors: a thread takes a token
        const int sub = threadIdx.x / SC_SUB, p = threadIdx.x % SC_SUB;
        float dec[SC_SUB], upto = 1.f, w = my_take;
#pragma unroll
        for (int l = 0; l < SC_SUB; l += 4) *reinterpret_cast<float4*>(dec + l) = *reinterpret_cast<const float4*>(decay_s + sub * SC_SUB + l);
#pragma unroll
        for (int l = 0; l < SC_SUB; ++l) {
            if (l <= p) upto *= dec[l];
            else w *= dec[l];
            if (l >= p) inner_s[sub][l][p] = w;
        }
        upto_s[threadIdx.x] = upto;
        behind_s[threadIdx.x] = w;     // (row 15 of the eighth: every decay behind the token)
    }
    cp_async_wait<0>();
    __syncthreads();                   // the queries are in registers, v has arrived
    fetch_tile<SC_CHUNK, D>(qk_s, a.k + (size_t)t0 * a.k_stride + group * D, a.k_stride, n_here, threadIdx.x, SC_OUT_THREADS);
    cp_async_commit();
    // A row of v that is not finite must not reach the tokens before it through a weight of zero: looked for here, kept apart below.
    int odd = 0;
#pragma unroll
    for (int i = 0; i < V_BYTES / 16 / SC_OUT_THREADS; ++i) {
        const uint4 x = *reinterpret_cast<const uint4*>(v_s + 16 * (threadIdx.x + SC_OUT_THREADS * i));
        const uint32_t parts[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) odd |= (parts[e] & 0x7f80u) == 0x7f80u || (parts[e] & 0x7f800000u) == 0x7f800000u;
    }

    // ---- what the state before the chunk says
    float acc[SC_VT / 8][4];
#pragma unroll
    for (int nt = 0; nt < SC_VT / 8; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[nt][e] = 0.f;
    float n_sum[2] = {0.f, 0.f};   // n . q of rows g and g + 8 (this thread's part), then the scores' sums as well
#pragma unroll
    for (int kd = 0; kd < D / 16; ++kd) {
#pragma unroll
        for (int vp = 0; vp < SC_VT / 16; vp += 2) {   // four sums in turn
            float sum[4][4];
#pragma unroll
            for (int part = 2; part >= 0; --part)
#pragma unroll
                for (int p = 0; p < 2; ++p) {
                    uint32_t b[4];
                    ldmatrix_x4(b, s_s + part * S_PART + tile_at<D>((vp + p) * 16 + (lane & 7) + ((lane >> 4) << 3), kd * 2 + ((lane >> 3) & 1)));
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        if (part == 2) MmaFirst{}(sum[2 * p + h], q_frag[kd], b[2 * h], b[2 * h + 1]);
                        else MmaNext{}(sum[2 * p + h], q_frag[kd], b[2 * h], b[2 * h + 1]);
                    }
                }
            add_sums(acc + 2 * vp, sum);
        }
        if (with_n) {
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const float* n_at = n_s + kd * 16 + (r >> 1) * 8 + t2;
                n_sum[r & 1] = fmaf(lower_bf16(q_frag[kd][r]), n_at[0], n_sum[r & 1]);
                n_sum[r & 1] = fmaf(upper_bf16(q_frag[kd][r]), n_at[1], n_sum[r & 1]);
            }
        }
    }
    cp_async_wait<0>();
    const bool not_finite = __syncthreads_or(odd) != 0;   // (and the keys have arrived)
    float f[2];                        // the decays from the eighth in hand up to rows g and g + 8, and the scale of q
    {
        f[0] = upto_s[tile * 16 + g] * a.q_scale, f[1] = upto_s[tile * 16 + g + 8] * a.q_scale;
        float before = 1.f;            // the decays of the whole eighths before this one
        for (int c = 0; c < tile; ++c) before *= upto_s[c * 16 + 15];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const float all = f[r] * before;
#pragma unroll
            for (int nt = 0; nt < SC_VT / 8; ++nt) acc[nt][2 * r] *= all, acc[nt][2 * r + 1] *= all;
            n_sum[r] *= all;
        }
    }

    // ---- what the chunk's own tokens say, from the eighth's own tokens back to the chunk's first
#pragma unroll 1
    for (int c = tile; c >= 0; --c) {
        float s[2][4];
#pragma unroll
        for (int kd = 0; kd < D / 16; ++kd) {
            uint32_t b[4];
            ldmatrix_x4(b, qk_s + tile_at<D>(c * 16 + (lane & 7) + ((lane >> 4) << 3), kd * 2 + ((lane >> 3) & 1)));
            float sum[2][4];
            MmaFirst{}(sum[0], q_frag[kd], b[0], b[1]);
            MmaFirst{}(sum[1], q_frag[kd], b[2], b[3]);
            if (kd > 0) add_sums(s, sum);
            else
#pragma unroll
                for (int e = 0; e < 4; ++e) s[0][e] = sum[0][e], s[1][e] = sum[1][e];
        }
        if (c == tile) {
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int row = g + (e >> 1) * 8, col = h * 8 + t2 + (e & 1);
                    s[h][e] = col <= row ? s[h][e] * a.q_scale * inner_s[c][row][col] : 0.f;
                }
        } else {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const float2 w = *reinterpret_cast<const float2*>(behind_s + c * 16 + h * 8 + t2);
                s[h][0] *= f[0] * w.x, s[h][1] *= f[0] * w.y;
                s[h][2] *= f[1] * w.x, s[h][3] *= f[1] * w.y;
            }
            const float all = upto_s[c * 16 + 15];
            f[0] *= all, f[1] *= all;
        }
        n_sum[0] += (s[0][0] + s[0][1]) + (s[1][0] + s[1][1]);
        n_sum[1] += (s[0][2] + s[0][3]) + (s[1][2] + s[1][3]);
        if (c == tile && not_finite) {   // token by token, so that what lies behind a row is left out and not multiplied by zero
#pragma unroll 1
            for (int j = 0; j < SC_SUB; ++j) {
                const int from = (lane & ~3) | ((j & 7) >> 1);
                const float w0 = __shfl_sync(0xffffffffu, j < 8 ? (j & 1 ? s[0][1] : s[0][0]) : (j & 1 ? s[1][1] : s[1][0]), from);
                const float w1 = __shfl_sync(0xffffffffu, j < 8 ? (j & 1 ? s[0][3] : s[0][2]) : (j & 1 ? s[1][3] : s[1][2]), from);
#pragma unroll
                for (int nt = 0; nt < SC_VT / 8; ++nt) {
                    const uint32_t x = *reinterpret_cast<const uint32_t*>(v_s + tile_at<SC_VT>(c * 16 + j, nt) + t2 * 2);
                    if (j <= g) acc[nt][0] = fmaf(w0, lower_bf16(x), acc[nt][0]), acc[nt][1] = fmaf(w0, upper_bf16(x), acc[nt][1]);
                    if (j <= g + 8) acc[nt][2] = fmaf(w1, lower_bf16(x), acc[nt][2]), acc[nt][3] = fmaf(w1, upper_bf16(x), acc[nt][3]);
                }
            }
            continue;
        }
        uint32_t hi[4], mid[4], lo[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const Thirds x = thirds(s[r >> 1][(r & 1) * 2], s[r >> 1][(r & 1) * 2 + 1]);
            hi[r] = x.hi, mid[r] = x.mid, lo[r] = x.lo;
        }
#pragma unroll
        for (int v2 = 0; v2 < SC_VT / 16; v2 += 2) {
            uint32_t b[2][4];
#pragma unroll
            for (int p = 0; p < 2; ++p) ldmatrix_x4_trans(b[p], v_s + tile_at<SC_VT>(c * 16 + (lane & 15), (v2 + p) * 2 + (lane >> 4)));
            float sum[4][4];
            auto part = [&](auto mma, const uint32_t (&x)[4]) {
#pragma unroll
                for (int p = 0; p < 2; ++p) {
                    mma(sum[2 * p], x, b[p][0], b[p][1]);
                    mma(sum[2 * p + 1], x, b[p][2], b[p][3]);
                }
            };
            part(MmaFirst{}, lo);
            part(MmaNext{}, mid);
            part(MmaNext{}, hi);
            add_sums(acc + 2 * v2, sum);
        }
    }

    const int width = a.n_heads * a.vdim, row = tile * 16 + g;
    float* y0 = a.y + (size_t)(t0 + row) * width + head * a.vdim + v0 + t2;
#pragma unroll
    for (int nt = 0; nt < SC_VT / 8; ++nt) {
        if (row < n_here) *reinterpret_cast<float2*>(y0 + nt * 8) = make_float2(acc[nt][0], acc[nt][1]);
        if (row + 8 < n_here) *reinterpret_cast<float2*>(y0 + 8 * (size_t)width + nt * 8) = make_float2(acc[nt][2], acc[nt][3]);
    }
    if (with_n) {
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            float sum = n_sum[r];
            sum += __shfl_xor_sync(0xffffffffu, sum, 1);
            sum += __shfl_xor_sync(0xffffffffu, sum, 2);
            if ((lane & 3) == 0 && row + 8 * r < n_here) a.nq[(size_t)(t0 + row + 8 * r) * a.n_heads + head] = sum;
        }
    }
}

template <int D>
static int launch_chunks(ChunkArgs a, int n_seqs, int max_q_len, cudaStream_t stream) {
    constexpr size_t parts_smem = (size_t)SC_CHUNK * D * 2 + SC_CHUNK * SC_VT * 2, outputs_smem = parts_smem + 3 * (size_t)SC_VT * D * 2;
    cudaError_t e = cudaFuncSetAttribute(chunk_parts_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)parts_smem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(chunk_outputs_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)outputs_smem);
    const int items = a.vdim / 8 * (D / 16) + (a.n_offset >= 0 ? 1 : 0), chunks = (max_q_len + SC_CHUNK - 1) / SC_CHUNK;
    const int each = a.portion.each > 0 ? min(a.portion.each, chunks) : chunks;
    for (int chunk0 = 0; chunk0 < chunks && e == cudaSuccess; chunk0 += each) {
        a.portion.chunk0 = chunk0;
        const dim3 grid(min(each, chunks - chunk0), a.vdim / SC_VT * a.n_heads, n_seqs);
        e = launch_pdl(chunk_parts_kernel<D>, grid, dim3(a.n_offset >= 0 ? 160 : 128), parts_smem, stream, a);
        if (e == cudaSuccess) e = launch_pdl(chunk_chain_kernel<D>, dim3((items + 7) / 8, a.n_heads, n_seqs), dim3(256), 0, stream, a);
        if (e == cudaSuccess) e = launch_pdl(chunk_outputs_kernel<D>, grid, dim3(SC_OUT_THREADS), outputs_smem, stream, a);
    }
    return (int)e;
}

// q, k: bfloat16 [T][groups * dim], v: bfloat16 [T][heads * vdim], rows strided in whole eights and 16-byte aligned; decay, take:
// float32 [T][heads] (rate_log null), or decay the pre-activations of both, rows gate_stride apart; y: float32 [T][heads * vdim]; nq: float32 [T][heads] or null (then n_offset < 0). scratch: float32
// [n_records][heads][dim * vdim + dim + 1], 16-byte aligned; n_records = n_tokens / 128 + n_seqs with each == 0, else n_seqs * each, and
// the call goes through `each` chunks of every sequence at a time, with [n_seqs][heads][dim * vdim + dim] floats behind the scratch
// for what passes from one portion to the next. max_q_len: the most tokens any sequence brings.
QF_EXPORT int qf_state_chunks(const void* q, int q_stride, const void* k, int k_stride, const void* v, int v_stride, const float* decay,
                              const float* take, const float* dt_bias, const float* rate_log, int gate_stride, const int* cu_q,
                              const int* slots, int n_seqs, int max_q_len, float* state,
                              long long slot_stride, long long s_offset, long long n_offset, int n_heads, int n_groups, int dim,
                              int vdim, float q_scale, float* scratch, long long n_records, int each, float* y, float* nq,
                              cudaStream_t stream) {
    if (n_seqs <= 0 || max_q_len <= 0) return 0;
    if ((dim != 64 && dim != 128) || vdim <= 0 || vdim % SC_VT || (!take && !rate_log) || ((q_stride | k_stride | v_stride) & 7) ||
        (((uintptr_t)q | (uintptr_t)k | (uintptr_t)v) & 15) || n_groups <= 0 || n_heads <= 0 || n_heads % n_groups || n_seqs > 65535 ||
        (long long)n_heads * (vdim / SC_VT) > 65535 || (n_offset >= 0 && !nq) || ((uintptr_t)scratch & 15))
        return (int)cudaErrorInvalidValue;
    if (each < 0 || (each > 0 && n_records < (long long)n_seqs * each)) return (int)cudaErrorInvalidValue;
    float *n_parts = scratch + n_records * n_heads * dim * vdim, *whole = n_parts + n_records * n_heads * dim;
    const ChunkArgs a{(const bf16*)q, (const bf16*)k, (const bf16*)v, q_stride, k_stride, v_stride, decay, take, dt_bias, rate_log, gate_stride, cu_q, slots, state,
                      slot_stride, s_offset, n_offset, n_heads, n_groups, vdim, q_scale, scratch, n_parts, whole, y, nq,
                      Portion{0, each, each > 0 ? whole + n_records * n_heads : nullptr}};
    return dim == 64 ? launch_chunks<64>(a, n_seqs, max_q_len, stream) : launch_chunks<128>(a, n_seqs, max_q_len, stream);
}
