// The recurrence of a matrix state per head with a decay per token and ROW of the state, written out over chunks of tokens:
//
//   S <- diag(w_t) S + k_t v_t^T,   y_t = S^T q_t  after the token's update,  or, with a bonus u,
//   y_t = (S + diag(u) k_t v_t^T)^T q_t  before it                                                  64 rows per head
//
// (`outer_state_scan_kernel` of recurrent.cu, modes 1 and 2, walks it token by token.) In a chunk of 64 tokens with the state S0
// before it, and W(j, i) the product over the tokens behind j up to i (with a bonus: up to i - 1) of the decays of a row,
//   y_i = sum_d q_id W(-1, i)_d S0_d + sum_{j < i} (sum_d q_id W(j, i)_d k_jd) v_j + (sum_d q_id (u_d) k_id) v_i
//   S_after = W(-1, last) S0 + sum_j (W(j, last) k_j) v_j^T
// in three launches: (1) `parts`: every chunk's own sum, and the decays from their pre-activations; (2) `chain`: the states before
// every chunk; (3) `outputs`.
// A weight belongs to a pair of tokens AND a row, so it goes into the operands: a chunk is cut into quarters of 16 tokens; between
// quarters W(j, i) is (decays of i's quarter up to i) x (decays of the whole quarters between) x (decays behind j in its quarter),
// put on q, q and k; within a quarter the products run along with j. Each factor is a product of decays, at most 1: nothing overflows
// or is divided. Every float32 operand of a product on the tensor cores is the exact sum of three bfloat16 numbers; of
// the nine products of two of them the six largest are taken (what is left out is below 2^-24 of the product, of either sign).
// What bounds it: the scan is a chain of one update per token (0.18 microseconds each); here the chain is one step per 64 tokens, the
// rest products and the quarters' own pairs. Measured, 2,048 tokens, 16 heads of 64 x 128: 283 -> 70
// microseconds; 7 heads: 262 -> 56.
#include "chunks.cuh"

#define RC_CHUNK 64
#define RC_D 64
#define RC_SUB 16
#define RC_VT 64              // columns of v of an output block
#define RC_LD (RC_D + 4)      // floats between staged float32 rows
#define RC_LH (RC_D + 8)      // bfloat16 numbers between staged rows of q and k
#define RC_PLANE (RC_CHUNK * RC_D * 2)

struct RowChunkArgs {
    const bf16 *q, *k, *v;
    int q_stride, k_stride, v_stride;
    const float *decay, *decay_bias, *bonus;   // decay [T][heads * 64]: the decays (kind 0) or their pre-activations
    int kind;                                  // 1: exp(-exp(z + b)), 2: sigmoid(z + b)^inv_tau
    float inv_tau;
    const int *cu_q, *slots;
    float* state;
    long long slot_stride, s_offset;
    int n_heads, vdim;
    float q_scale;
    float *records, *whole, *made;   // [record][heads][vdim][64], [record][heads][64], [T][heads * 64] (kind 0: not written)
    float* y;
    Portion portion;
    int v_each;      // tiles of 64 columns of v that a block of outputs takes, one after the other
};

__device__ __forceinline__ float row_log_sigmoid(float x) { return fminf(x, 0.f) - log1pf(expf(-fabsf(x))); }

// ------------------------------------------------------------------------------------------------------------------
// (1) A chunk of one head, all columns of v: sum_j (W(j, last) k_j) v_j^T as S^T += v^T (weighted k), 16 columns of v a warp and turn. A
// thread keeps its half column of decays in registers, all asked for at once: loaded, formed and stored one by one they were 32
// round trips (3,079 tokens of 16 heads of 64 x 128: 44 microseconds, 30 so).
__global__ void __launch_bounds__(128)
row_parts_kernel(const RowChunkArgs a) {
    grid_chain_entry();
    extern __shared__ __align__(128) unsigned char rc_smem[];
    unsigned char* kw_s = rc_smem;                                        // [3][64][64] the weighted keys' parts
    bf16* k_s = reinterpret_cast<bf16*>(kw_s + 3 * RC_PLANE);             // [64][RC_LH]
    unsigned char* v_s = reinterpret_cast<unsigned char*>(k_s + RC_CHUNK * RC_LH);   // [vdim / 64][64][64]
    __shared__ Running total_s[2][RC_D];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, head = blockIdx.y, seq = blockIdx.z;
    const int chunk = a.portion.chunk0 + (int)blockIdx.x, t0 = a.cu_q[seq] + chunk * RC_CHUNK, n_here = min(RC_CHUNK, a.cu_q[seq + 1] - t0);
    if (n_here <= 0) return;
    const long long record = record_of<RC_CHUNK>(a.portion, a.cu_q, seq, chunk) * a.n_heads + head;
    for (int i = threadIdx.x; i < RC_CHUNK * (RC_D / 8); i += 128) {
        const int row = i / 8, c = (i % 8) * 8;
        const bf16* src = a.k + (size_t)t0 * a.k_stride + head * RC_D + c;
        cp_async_16(k_s + row * RC_LH + c, row < n_here ? src + (size_t)row * a.k_stride : src, row < n_here);
    }
    for (int vt = 0; vt < a.vdim / RC_VT; ++vt)
        fetch_tile<RC_CHUNK, RC_VT>(v_s + vt * RC_CHUNK * RC_VT * 2, a.v + (size_t)t0 * a.v_stride + head * a.vdim + vt * RC_VT, a.v_stride,
                                    n_here, threadIdx.x, 128);
    cp_async_commit();
    const int d = threadIdx.x & 63, half = threadIdx.x >> 6;
    const size_t width = (size_t)a.n_heads * RC_D;
    float w[RC_CHUNK / 2];   // the decays of this thread's row of the state in half of the tokens
    {
        const float* src = a.decay + (size_t)t0 * width + head * RC_D + d;
#pragma unroll
        for (int i = 0; i < RC_CHUNK / 2; ++i) w[i] = src[min(half * (RC_CHUNK / 2) + i, n_here - 1) * width];   // all on their way at once
        if (a.kind != 0) {
            const float b = a.decay_bias[head * RC_D + d];
            float* made = a.made + (size_t)t0 * width + head * RC_D + d;
#pragma unroll
            for (int i = 0; i < RC_CHUNK / 2; ++i) {
                const float z = w[i] + b;
                w[i] = a.kind == 1 ? expf(-expf(z)) : expf(row_log_sigmoid(z) * a.inv_tau);
                if (half * (RC_CHUNK / 2) + i < n_here) made[(half * (RC_CHUNK / 2) + i) * width] = w[i];
            }
        }
        Running total{1.f, 0.f};
#pragma unroll
        for (int i = 0; i < RC_CHUNK / 2; ++i) {
            if (half * (RC_CHUNK / 2) + i >= n_here) w[i] = 1.f;
            total.times(w[i]);
        }
        total_s[half][d] = total;
    }
    cp_async_wait<0>();
    __syncthreads();
    Running behind{1.f, 0.f};
    if (half == 0) {
        Running all = total_s[0][d];
        behind = total_s[1][d];
        all.times(behind);
        a.whole[record * RC_D + d] = all.value + all.rest;
    }
#pragma unroll
    for (int i = RC_CHUNK / 2 - 1; i >= 0; --i) {
        const int row = half * (RC_CHUNK / 2) + i;
        const Thirds x = thirds(behind.of(__bfloat162float(k_s[row * RC_LH + d])), 0.f);
        unsigned char* at = kw_s + tile_at<RC_D>(row, d >> 3) + (d & 7) * 2;
        *reinterpret_cast<unsigned short*>(at) = (unsigned short)x.hi;
        *reinterpret_cast<unsigned short*>(at + RC_PLANE) = (unsigned short)x.mid;
        *reinterpret_cast<unsigned short*>(at + 2 * RC_PLANE) = (unsigned short)x.lo;
        behind.times(w[i]);
    }
    __syncthreads();
    const int g = lane >> 2, t2 = (lane & 3) * 2;
    for (int v0 = warp * 16; v0 < a.vdim; v0 += 64) {
        const unsigned char* vt = v_s + (v0 / RC_VT) * RC_CHUNK * RC_VT * 2;
        const int piece = (v0 % RC_VT) / 8;
        float acc[RC_D / 8][4], low[RC_D / 8][4];   // (low: the products of the lesser parts)
#pragma unroll
        for (int nt = 0; nt < RC_D / 8; ++nt)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[nt][e] = low[nt][e] = 0.f;
#pragma unroll
        for (int kk = 0; kk < RC_CHUNK / 16; ++kk) {
            uint32_t x[4];
            ldmatrix_x4_trans(x, vt + tile_at<RC_VT>(kk * 16 + (lane & 7) + ((lane >> 4) << 3), piece + ((lane >> 3) & 1)));
            float sum[RC_D / 8][4];
            auto part = [&](auto mma, float (&to)[RC_D / 8][4], int which) {
#pragma unroll
                for (int np = 0; np < RC_D / 16; ++np) {
                    uint32_t b[4];
                    ldmatrix_x4_trans(b, kw_s + which * RC_PLANE + tile_at<RC_D>(kk * 16 + (lane & 15), np * 2 + (lane >> 4)));
                    mma(to[2 * np], x, b[0], b[1]);
                    mma(to[2 * np + 1], x, b[2], b[3]);
                }
            };
            part(MmaNext{}, low, 2);
            part(MmaNext{}, low, 1);
            part(MmaFirst{}, sum, 0);
            add_sums(acc, sum);
        }
        add_sums(acc, low);
        float* rec = a.records + record * RC_D * a.vdim + (size_t)(v0 + g) * RC_D + t2;
#pragma unroll
        for (int nt = 0; nt < RC_D / 8; ++nt) {
            *reinterpret_cast<float2*>(rec + nt * 8) = make_float2(acc[nt][0], acc[nt][1]);
            *reinterpret_cast<float2*>(rec + 8 * RC_D + nt * 8) = make_float2(acc[nt][2], acc[nt][3]);
        }
    }
}

// ------------------------------------------------------------------------------------------------------------------
// (2) The states before every chunk, in the place of the chunks' own parts, and the one after the last in the sequence's state: a
// thread takes four neighbouring rows of S in one column of v, eight records' loads on their way. A warp's 32 threads are 8 columns
// x 16 rows: whole sectors of the records and, transposed, of the state.
__global__ void __launch_bounds__(256)
row_chain_kernel(const RowChunkArgs a) {
    grid_chain_entry();
    constexpr int AHEAD = 8;
    const int lane = threadIdx.x & 31, head = blockIdx.y, seq = blockIdx.z;
    const int len = a.cu_q[seq + 1] - a.cu_q[seq], slot = a.slots[seq], chunk0 = a.portion.chunk0, left = (len + RC_CHUNK - 1) / RC_CHUNK - chunk0;
    const int n_chunks = a.portion.each > 0 ? min(left, a.portion.each) : left;
    const int item = (int)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (n_chunks <= 0 || item >= a.vdim / 8 * (RC_D / 16)) return;
    const long long first = record_of<RC_CHUNK>(a.portion, a.cu_q, seq, chunk0) * a.n_heads + head, pitch = (long long)a.n_heads * RC_D * a.vdim;
    const int col = item / (RC_D / 16) * 8 + (lane >> 2), row = item % (RC_D / 16) * 16 + (lane & 3) * 4;
    const float* whole = a.whole + first * RC_D + row;
    float* at = a.records + first * RC_D * a.vdim + (size_t)col * RC_D + row;
    // the sequence's state, or what stands for it between portions (zeros before the first)
    float* base = slot >= 0 ? a.state + slot * a.slot_stride + a.s_offset : a.portion.carry ? a.portion.carry + (long long)seq * a.n_heads * RC_D * a.vdim : nullptr;
    float* kept = base ? base + ((long long)head * RC_D + row) * a.vdim + col : nullptr;
    const bool fresh = !kept || (slot < 0 && chunk0 == 0);
    float s[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) s[e] = fresh ? 0.f : kept[(size_t)e * a.vdim];
    float4 part[AHEAD], w[AHEAD];
#pragma unroll
    for (int u = 0; u < AHEAD; ++u)
        if (u < n_chunks) {
            part[u] = *reinterpret_cast<const float4*>(at + u * pitch);
            w[u] = *reinterpret_cast<const float4*>(whole + (long long)u * a.n_heads * RC_D);
        }
    for (int c0 = 0; c0 < n_chunks; c0 += AHEAD, at += AHEAD * pitch) {
#pragma unroll
        for (int u = 0; u < AHEAD; ++u)
            if (c0 + u < n_chunks) {
                const float4 mine = part[u], all = w[u];
                if (c0 + u + AHEAD < n_chunks) {
                    part[u] = *reinterpret_cast<const float4*>(at + (u + AHEAD) * pitch);
                    w[u] = *reinterpret_cast<const float4*>(whole + (long long)(c0 + u + AHEAD) * a.n_heads * RC_D);
                }
                *reinterpret_cast<float4*>(at + u * pitch) = make_float4(s[0], s[1], s[2], s[3]);
                s[0] = fmaf(s[0], all.x, mine.x), s[1] = fmaf(s[1], all.y, mine.y);
                s[2] = fmaf(s[2], all.z, mine.z), s[3] = fmaf(s[3], all.w, mine.w);
            }
    }
    if (kept) {
#pragma unroll
        for (int e = 0; e < 4; ++e) kept[(size_t)e * a.vdim] = s[e];
    }
}

// ------------------------------------------------------------------------------------------------------------------
// (3) Outputs of one chunk, one head, 64 columns of v; a warp takes a quarter of the tokens.
template <bool BONUS>
__global__ void __launch_bounds__(128, 2)
row_outputs_kernel(const RowChunkArgs a) {
    grid_chain_entry();
    extern __shared__ __align__(128) unsigned char rc_smem[];
    unsigned char* kh_s = rc_smem;                                              // [3][64][64] keys times the decays behind them in their quarter
    float* qh_s = reinterpret_cast<float*>(kh_s + 3 * RC_PLANE);                // [64][RC_LD] queries times the decays of their quarter up to them
    bf16* k_s = reinterpret_cast<bf16*>(qh_s + RC_CHUNK * RC_LD);               // [64][RC_LH]
    unsigned char* v_all = reinterpret_cast<unsigned char*>(k_s + RC_CHUNK * RC_LH);   // [v_each][64][64]
    float* w_s = reinterpret_cast<float*>(v_all + a.v_each * (RC_CHUNK * RC_VT * 2));   // [64][RC_LD]
    bf16* q_s = reinterpret_cast<bf16*>(w_s + RC_CHUNK * RC_LD);                // [64][RC_LH]
    unsigned char* s_s = reinterpret_cast<unsigned char*>(w_s);                 // [3][64 v][64] the state's parts, over w_s and q_s
    static_assert(3 * RC_VT * RC_D * 2 <= RC_CHUNK * RC_LD * 4 + RC_CHUNK * RC_LH * 2, "the state's parts find room there");
    __shared__ float pair_s[4][RC_SUB][RC_SUB + 1], all_s[4][RC_D];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, seq = blockIdx.z;
    const int v_groups = a.vdim / RC_VT / a.v_each, head = blockIdx.y / v_groups, v_first = (blockIdx.y % v_groups) * a.v_each * RC_VT;
    const int chunk = a.portion.chunk0 + (int)blockIdx.x, t0 = a.cu_q[seq] + chunk * RC_CHUNK, n_here = min(RC_CHUNK, a.cu_q[seq + 1] - t0);
    if (n_here <= 0) return;
    const long long record = record_of<RC_CHUNK>(a.portion, a.cu_q, seq, chunk) * a.n_heads + head;
    const size_t width = (size_t)a.n_heads * RC_D;
    for (int i = threadIdx.x; i < RC_CHUNK * (RC_D / 8); i += 128) {
        const int row = i / 8, c = (i % 8) * 8;
        const bool there = row < n_here;
        const bf16 *ks = a.k + (size_t)t0 * a.k_stride + head * RC_D + c, *qs = a.q + (size_t)t0 * a.q_stride + head * RC_D + c;
        cp_async_16(k_s + row * RC_LH + c, there ? ks + (size_t)row * a.k_stride : ks, there);
        cp_async_16(q_s + row * RC_LH + c, there ? qs + (size_t)row * a.q_stride : qs, there);
    }
    for (int vt = 0; vt < a.v_each; ++vt)
        fetch_tile<RC_CHUNK, RC_VT>(v_all + vt * (RC_CHUNK * RC_VT * 2), a.v + (size_t)t0 * a.v_stride + head * a.vdim + v_first + vt * RC_VT, a.v_stride,
                                    n_here, threadIdx.x, 128);
    cp_async_commit();
    const float* w_src = (a.kind != 0 ? a.made : a.decay) + (size_t)t0 * width + head * RC_D;
#pragma unroll
    for (int i = threadIdx.x; i < RC_CHUNK * (RC_D / 4); i += 128) {
        const int row = i / 16, c = (i % 16) * 4;
        *reinterpret_cast<float4*>(w_s + row * RC_LD + c) =
            row < n_here ? *reinterpret_cast<const float4*>(w_src + row * width + c) : make_float4(1.f, 1.f, 1.f, 1.f);
    }
    constexpr int EACH = RC_VT * RC_D / 4 / 128;
    float4 held[EACH];
    const float* rec = a.records + record * RC_D * a.vdim + (size_t)v_first * RC_D;
#pragma unroll
    for (int u = 0; u < EACH; ++u) held[u] = *reinterpret_cast<const float4*>(rec + 4 * (threadIdx.x + 128 * u));
    cp_async_wait<0>();
    __syncthreads();

    // ---- the operands' weights: a thread takes a row of the state in two quarters
    {
        const int d = threadIdx.x & 63;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int sub = (threadIdx.x >> 6) * 2 + h, r0 = sub * RC_SUB;
            float upto = 1.f, behind = 1.f;
#pragma unroll
            for (int i = 0; i < RC_SUB; ++i) {
                const float w = w_s[(r0 + i) * RC_LD + d], q = __bfloat162float(q_s[(r0 + i) * RC_LH + d]) * a.q_scale;
                if (!BONUS) upto *= w;
                qh_s[(r0 + i) * RC_LD + d] = q * upto;
                if (BONUS) upto *= w;
            }
            all_s[sub][d] = upto;
#pragma unroll
            for (int i = RC_SUB - 1; i >= 0; --i) {
                const Thirds x = thirds(__bfloat162float(k_s[(r0 + i) * RC_LH + d]) * behind, 0.f);
                unsigned char* at = kh_s + tile_at<RC_D>(r0 + i, d >> 3) + (d & 7) * 2;
                *reinterpret_cast<unsigned short*>(at) = (unsigned short)x.hi;
                *reinterpret_cast<unsigned short*>(at + RC_PLANE) = (unsigned short)x.mid;
                *reinterpret_cast<unsigned short*>(at + 2 * RC_PLANE) = (unsigned short)x.lo;
                behind *= w_s[(r0 + i) * RC_LD + d];
            }
        }
    }
    // ---- the pairs of a quarter: lane (i, half) holds half of query i's row and walks the keys from i backwards, the decays
    // between gathering on it
    {
        const int i = lane & 15, half = lane >> 4, r0 = warp * RC_SUB;
        float2 qp[16];
#pragma unroll
        for (int c = 0; c < 32; c += 8) {
            const uint4 x = *reinterpret_cast<const uint4*>(q_s + (r0 + i) * RC_LH + half * 32 + c);
            const uint32_t p[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
            for (int e = 0; e < 4; ++e) qp[c / 2 + e] = make_float2(lower_bf16(p[e]) * a.q_scale, upper_bf16(p[e]) * a.q_scale);
        }
#pragma unroll 1
        for (int s = 0; s < RC_SUB; ++s) {
            const int j = max(i - s, 0);
            const bf16* kj = k_s + (r0 + j) * RC_LH + half * 32;
            const float* wj = w_s + (r0 + j) * RC_LD + half * 32;
            float2 sum[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};   // two multiply-adds an instruction
#pragma unroll
            for (int c = 0; c < 32; c += 8) {
                const uint4 x = *reinterpret_cast<const uint4*>(kj + c);
                const float4 wa = *reinterpret_cast<const float4*>(wj + c), wb = *reinterpret_cast<const float4*>(wj + c + 4);
                const uint32_t p[4] = {x.x, x.y, x.z, x.w};
                const float2 w[4] = {make_float2(wa.x, wa.y), make_float2(wa.z, wa.w), make_float2(wb.x, wb.y), make_float2(wb.z, wb.w)};
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    float2 k = make_float2(lower_bf16(p[e]), upper_bf16(p[e]));
                    if (BONUS && s == 0) {
                        const float* u = a.bonus + head * RC_D + half * 32 + c + 2 * e;
                        k.x *= u[0], k.y *= u[1];
                    }
                    sum[e & 1] = __ffma2_rn(qp[c / 2 + e], k, sum[e & 1]);
                    if (!BONUS || s > 0) qp[c / 2 + e] = __fmul2_rn(qp[c / 2 + e], w[e]);
                }
            }
            float total = (sum[0].x + sum[0].y) + (sum[1].x + sum[1].y);
            total += __shfl_xor_sync(0xffffffffu, total, 16);
            if (half == 0 && i >= s) pair_s[warp][i][i - s] = total;
        }
    }
#pragma unroll 1
    for (int vt = 0; vt < a.v_each; ++vt) {
        const unsigned char* v_s = v_all + vt * (RC_CHUNK * RC_VT * 2);
        const int v0 = v_first + vt * RC_VT;
        if (vt > 0) {
#pragma unroll
            for (int u = 0; u < EACH; ++u) held[u] = *reinterpret_cast<const float4*>(rec + (size_t)vt * RC_VT * RC_D + 4 * (threadIdx.x + 128 * u));
        }
        // A row of v that is not finite must not reach the tokens before it through a weight of zero: looked for here, kept apart below.
        int odd = 0;
#pragma unroll
        for (int i = 0; i < RC_CHUNK * RC_VT * 2 / 16 / 128; ++i) {
            const uint4 x = *reinterpret_cast<const uint4*>(v_s + 16 * (threadIdx.x + 128 * i));
            const uint32_t p[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
            for (int e = 0; e < 4; ++e) odd |= (p[e] & 0x7f80u) == 0x7f80u || (p[e] & 0x7f800000u) == 0x7f800000u;
        }
        // (and nobody reads the decays and the plain queries, or the state of the tile before, any more)
        const bool not_finite = __syncthreads_or(odd) != 0;
#pragma unroll
        for (int u = 0; u < EACH; ++u) {
            const int i = 4 * (threadIdx.x + 128 * u), row = i / RC_D, col = i % RC_D;
            const Thirds x = thirds(held[u].x, held[u].y), z = thirds(held[u].z, held[u].w);
            unsigned char* at = s_s + tile_at<RC_D>(row, col >> 3) + (col & 7) * 2;
            *reinterpret_cast<uint2*>(at) = make_uint2(x.hi, z.hi);
            *reinterpret_cast<uint2*>(at + RC_VT * RC_D * 2) = make_uint2(x.mid, z.mid);
            *reinterpret_cast<uint2*>(at + 2 * RC_VT * RC_D * 2) = make_uint2(x.lo, z.lo);
        }
        __syncthreads();

        const int g = lane >> 2, t2 = (lane & 3) * 2;
        // The products of the lesser parts, 2^8 times smaller, are summed apart; those of the leading parts 16 rows or tokens at a time
        // (MmaFirst). Errors against 64 bits, outputs / states, 2,048 tokens of 7 heads of 64 x 128, decays sigmoid(z)^(1/16): 1.20e-7 /
        // 6.0e-8, token by token 1.45e-7 / 1.14e-7 (the leading parts' sums left to the tensor cores: 2.5e-7 / 1.8e-7).
        float acc[RC_VT / 8][4], low[RC_VT / 8][4];
#pragma unroll
        for (int nt = 0; nt < RC_VT / 8; ++nt)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[nt][e] = low[nt][e] = 0.f;
        // rows g and g + 8 of this warp's queries: two neighbouring columns at 2 t and at 2 t + 8 of every 16
        float2 qf[RC_D / 16][4];
#pragma unroll
        for (int kd = 0; kd < RC_D / 16; ++kd)
#pragma unroll
            for (int r = 0; r < 4; ++r)
                qf[kd][r] = *reinterpret_cast<const float2*>(qh_s + (warp * RC_SUB + g + (r & 1) * 8) * RC_LD + kd * 16 + (r >> 1) * 8 + t2);
        // Both operands in three parts, the six largest products of the nine: sum[h] += A (16 x 16) B (16 x 8, h-th), low[h] likewise
        auto six = [&](const Thirds (&x)[4], const unsigned char* base, uint32_t plane, uint32_t at, float (&s0)[4], float (&s1)[4], float (&l0)[4],
                       float (&l1)[4]) {
            uint32_t hi[4], mid[4], lo[4], b[3][4];
#pragma unroll
            for (int r = 0; r < 4; ++r) hi[r] = x[r].hi, mid[r] = x[r].mid, lo[r] = x[r].lo;
#pragma unroll
            for (int p = 0; p < 3; ++p) ldmatrix_x4(b[p], base + p * plane + at);
            float sum[2][4];
            MmaFirst{}(sum[0], hi, b[0][0], b[0][1]);
            MmaFirst{}(sum[1], hi, b[0][2], b[0][3]);
#pragma unroll
            for (int e = 0; e < 4; ++e) s0[e] += sum[0][e], s1[e] += sum[1][e];
            mma_bf16_16816(l0, lo, b[0][0], b[0][1]);
            mma_bf16_16816(l1, lo, b[0][2], b[0][3]);
            mma_bf16_16816(l0, mid, b[1][0], b[1][1]);
            mma_bf16_16816(l1, mid, b[1][2], b[1][3]);
            mma_bf16_16816(l0, hi, b[2][0], b[2][1]);
            mma_bf16_16816(l1, hi, b[2][2], b[2][3]);
            mma_bf16_16816(l0, mid, b[0][0], b[0][1]);
            mma_bf16_16816(l1, mid, b[0][2], b[0][3]);
            mma_bf16_16816(l0, hi, b[1][0], b[1][1]);
            mma_bf16_16816(l1, hi, b[1][2], b[1][3]);
        };
        auto values = [&](int c, const float (&s)[2][4]) {   // acc += s (16 x 16 tokens of quarter c) v
            uint32_t part[3][4];
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const Thirds x = thirds(s[r >> 1][(r & 1) * 2], s[r >> 1][(r & 1) * 2 + 1]);
                part[0][r] = x.hi, part[1][r] = x.mid, part[2][r] = x.lo;
            }
            uint32_t b[RC_VT / 16][4];
#pragma unroll
            for (int vp = 0; vp < RC_VT / 16; ++vp) ldmatrix_x4_trans(b[vp], v_s + tile_at<RC_VT>(c * 16 + (lane & 15), vp * 2 + (lane >> 4)));
            float sum[RC_VT / 8][4];
#pragma unroll
            for (int vp = 0; vp < RC_VT / 16; ++vp) {
                MmaFirst{}(sum[2 * vp], part[0], b[vp][0], b[vp][1]);
                MmaFirst{}(sum[2 * vp + 1], part[0], b[vp][2], b[vp][3]);
            }
#pragma unroll
            for (int p = 2; p >= 1; --p)
#pragma unroll
                for (int vp = 0; vp < RC_VT / 16; ++vp) {
                    mma_bf16_16816(low[2 * vp], part[p], b[vp][0], b[vp][1]);
                    mma_bf16_16816(low[2 * vp + 1], part[p], b[vp][2], b[vp][3]);
                }
            add_sums(acc, sum);
        };
        // ---- this quarter's own pairs
        {
            float s[2][4];
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int row = g + (e >> 1) * 8, col = h * 8 + t2 + (e & 1);
                    s[h][e] = col <= row ? pair_s[warp][row][col] : 0.f;
                }
            if (!not_finite) {
                values(warp, s);
            } else {   // token by token, so that what lies behind a row is left out and not multiplied by zero
#pragma unroll 1
                for (int j = 0; j < RC_SUB; ++j) {
                    const float p0 = j <= g ? pair_s[warp][g][j] : 0.f, p1 = j <= g + 8 ? pair_s[warp][g + 8][j] : 0.f;
#pragma unroll
                    for (int nt = 0; nt < RC_VT / 8; ++nt) {
                        const uint32_t x = *reinterpret_cast<const uint32_t*>(v_s + tile_at<RC_VT>(warp * 16 + j, nt) + t2 * 2);
                        if (j <= g) acc[nt][0] = fmaf(p0, lower_bf16(x), acc[nt][0]), acc[nt][1] = fmaf(p0, upper_bf16(x), acc[nt][1]);
                        if (j <= g + 8) acc[nt][2] = fmaf(p1, lower_bf16(x), acc[nt][2]), acc[nt][3] = fmaf(p1, upper_bf16(x), acc[nt][3]);
                    }
                }
            }
        }
        // ---- the quarters before it, the nearest first; the decays of each gather on the queries
        for (int c = warp - 1; c >= 0; --c) {
            float s[2][4], s_low[2][4];
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int e = 0; e < 4; ++e) s[h][e] = s_low[h][e] = 0.f;
#pragma unroll
            for (int kd = 0; kd < RC_D / 16; ++kd) {
                Thirds x[4];
#pragma unroll
                for (int r = 0; r < 4; ++r) x[r] = thirds(qf[kd][r].x, qf[kd][r].y);
                six(x, kh_s, RC_PLANE, tile_at<RC_D>(c * 16 + (lane & 7) + ((lane >> 4) << 3), kd * 2 + ((lane >> 3) & 1)), s[0], s[1], s_low[0], s_low[1]);
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    const float2 all = *reinterpret_cast<const float2*>(&all_s[c][kd * 16 + (r >> 1) * 8 + t2]);
                    qf[kd][r].x *= all.x, qf[kd][r].y *= all.y;
                }
            }
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int e = 0; e < 4; ++e) s[h][e] += s_low[h][e];
            values(c, s);
        }
        // ---- the state before the chunk
#pragma unroll
        for (int kd = 0; kd < RC_D / 16; ++kd) {
            Thirds x[4];
#pragma unroll
            for (int r = 0; r < 4; ++r) x[r] = thirds(qf[kd][r].x, qf[kd][r].y);
#pragma unroll
            for (int vp = 0; vp < RC_VT / 16; ++vp)
                six(x, s_s, RC_VT * RC_D * 2, tile_at<RC_D>(vp * 16 + (lane & 7) + ((lane >> 4) << 3), kd * 2 + ((lane >> 3) & 1)), acc[2 * vp], acc[2 * vp + 1],
                    low[2 * vp], low[2 * vp + 1]);
        }
#pragma unroll
        for (int nt = 0; nt < RC_VT / 8; ++nt)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[nt][e] += low[nt][e];
        const int row = warp * RC_SUB + g, y_width = a.n_heads * a.vdim;
        float* y0 = a.y + (size_t)(t0 + row) * y_width + head * a.vdim + v0 + t2;
#pragma unroll
        for (int nt = 0; nt < RC_VT / 8; ++nt) {
            if (row < n_here) *reinterpret_cast<float2*>(y0 + nt * 8) = make_float2(acc[nt][0], acc[nt][1]);
            if (row + 8 < n_here) *reinterpret_cast<float2*>(y0 + 8 * (size_t)y_width + nt * 8) = make_float2(acc[nt][2], acc[nt][3]);
        }
    }
}

// q, k: bfloat16 [T][heads * 64], v: bfloat16 [T][heads * vdim], rows strided in whole eights and 16-byte aligned; decay: float32
// [T][heads * 64], 16-byte aligned; kind, decay_bias, inv_tau, bonus as in qf_outer_state_scan_rows; y: float32 [T][heads * vdim].
// scratch: float32, 16-byte aligned: [n_records][heads][64 * vdim + 64], then (each > 0) [n_seqs][heads][64 * vdim] for what passes from one
// portion to the next, then (kind not 0) [T][heads * 64]. n_records = n_tokens / 64 + n_seqs with each == 0, else n_seqs * each, and
// the call goes through `each` chunks of every sequence at a time.
QF_EXPORT int qf_row_chunks(const void* q, int q_stride, const void* k, int k_stride, const void* v, int v_stride, const float* decay,
                            const float* decay_bias, int kind, float inv_tau, const float* bonus, const int* cu_q, const int* slots,
                            int n_seqs, int max_q_len, float* state, long long slot_stride, long long s_offset, int n_heads, int dim,
                            int vdim, float q_scale, float* scratch, long long n_records, int each, float* y, cudaStream_t stream) {
    if (n_seqs <= 0 || max_q_len <= 0) return 0;
    if (dim != RC_D || vdim <= 0 || vdim % RC_VT || vdim > 512 || n_heads <= 0 || n_seqs > 65535 || (long long)n_heads * (vdim / RC_VT) > 65535 ||
        kind < 0 || kind > 2 || (kind != 0 && !decay_bias) || ((q_stride | k_stride | v_stride) & 7) ||
        (((uintptr_t)q | (uintptr_t)k | (uintptr_t)v | (uintptr_t)decay | (uintptr_t)scratch) & 15))
        return (int)cudaErrorInvalidValue;
    if (each < 0 || (each > 0 && n_records < (long long)n_seqs * each)) return (int)cudaErrorInvalidValue;
    float *whole = scratch + n_records * n_heads * dim * vdim, *carry = whole + n_records * n_heads * dim;
    float* made = carry + (each > 0 ? (long long)n_seqs * n_heads * dim * vdim : 0);
    RowChunkArgs a{(const bf16*)q, (const bf16*)k, (const bf16*)v, q_stride, k_stride, v_stride, decay, decay_bias, bonus, kind, inv_tau,
                         cu_q, slots, state, slot_stride, s_offset, n_heads, vdim, q_scale, scratch, whole, made, y, Portion{0, each, each > 0 ? carry : nullptr}, 1};
    const int chunks = (max_q_len + RC_CHUNK - 1) / RC_CHUNK;
    const size_t parts_smem = 3 * RC_PLANE + RC_CHUNK * RC_LH * 2 + (size_t)RC_CHUNK * vdim * 2;
    // A block of outputs takes two tiles of v one after the other, with the same weights, pairs and parts of the operands, where the blocks
    // still fill the SMs' two places each (3,079 tokens of 16 heads of 64 x 128: 96 microseconds with one, 83 with two); else one.
    const int v_tiles = vdim / RC_VT;
    const long long at_most = each > 0 ? (long long)min(each, (max_q_len + RC_CHUNK - 1) / RC_CHUNK) * n_seqs : n_records;
    a.v_each = v_tiles % 2 == 0 && at_most * n_heads * (v_tiles / 2) >= 2ll * qf_sm_count() ? 2 : 1;
    const size_t outputs_smem = 3 * RC_PLANE + 2 * RC_CHUNK * RC_LD * 4 + 2 * RC_CHUNK * RC_LH * 2 + (size_t)a.v_each * RC_CHUNK * RC_VT * 2;
    auto outputs = bonus ? row_outputs_kernel<true> : row_outputs_kernel<false>;
    cudaError_t e = cudaFuncSetAttribute(row_parts_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)parts_smem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(outputs, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)outputs_smem);
    const int at_once = each > 0 ? min(each, chunks) : chunks;
    for (int chunk0 = 0; chunk0 < chunks && e == cudaSuccess; chunk0 += at_once) {
        a.portion.chunk0 = chunk0;
        const int here = min(at_once, chunks - chunk0);
        e = launch_pdl(row_parts_kernel, dim3(here, n_heads, n_seqs), dim3(128), parts_smem, stream, a);
        if (e == cudaSuccess)
            e = launch_pdl(row_chain_kernel, dim3((vdim / 8 * (RC_D / 16) + 7) / 8, n_heads, n_seqs), dim3(256), 0, stream, a);
        if (e == cudaSuccess) e = launch_pdl(outputs, dim3(here, v_tiles / a.v_each * n_heads, n_seqs), dim3(128), outputs_smem, stream, a);
    }
    return (int)e;
}
