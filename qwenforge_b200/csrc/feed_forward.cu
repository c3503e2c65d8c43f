// The SwiGLU feed-forward of a step of up to eight rows as ONE kernel, for layers whose weights find room in the shared memory of all SMs:
//   x = rmsnorm(hidden) * norm_weight;  a = silu(x Wg^T) * (x Wu^T);  sums += a Wd^T
// A block owns `cols` of the intermediate columns: their gate and up rows, and the same columns of the down weight, are on their way into
// its shared memory before the kernel ahead has ended (no kernel writes weights), so that what is left behind the wait is a chain in one
// block: the token rows, gate and up on the tensor cores (mma.sync), the gate, the block's share of the down product, and 16-byte vector
// reductions of it into `sums`, float32 [rows][width]. As two kernels (skinny_gemm.cu) the activations went through the L2 behind a second
// kernel's launch. What bounds it is that chain, then the reductions, blocks x rows x width / 4 of them (218,000 for eight rows of 896 x 4,864; a
// row: 5.4 microseconds from the end of the kernel ahead to its own, 8.9 for the two kernels). A decode step at Qwen2.5-0.5B sizes, microseconds,
// two kernels / this one: 1 sequence of 1,024 tokens 627 / 525, 4 667 / 544, 8 675 / 569; 1 of 4,000 627 / 525, 8 680 / 606.
// `sums` is a buffer of its own, zero before the launch: added into the stream in place, a block's share would reach rows that other blocks are
// still reading. The next layer's QKV product reads stream and sums together, and its output projection (fold_project.cu) moves the sums into
// the stream and leaves zeros. The shares arrive in no fixed order, as there.
#include "skinny_common.cuh"

#define FF_THREADS 512
#define FF_WARPS (FF_THREADS / 32)
#define FF_MAX_ROWS 8
#define FF_MAX_COLS 128

struct FeedForwardArgs {
    const float* hidden;    // [rows][width]
    const bf16* norm_w;     // [width]
    const bf16* gate_up;    // [2 * inter][ldg]: gate rows, then up rows
    const bf16* down;       // [width][ldd]
    float* sums;            // [rows][width]
    int* err;
    float eps;
    int rows, width, inter, ldg, ldd, cols;
    int row_warps_log;      // 2 to the power of it: warps that share a token row
    int each, each_recip;   // warps of a gate/up tile; 65536 / each, rounded up (an integer division would be a part of the chain)
};

// Bytes between rows in shared memory: an odd number of 16-byte pieces, so that the eight rows of a ldmatrix meet no bank twice.
static __host__ __device__ inline int ff_stride(int elements) { return ((elements * 2 + 15) / 16 | 1) * 16; }

__device__ __forceinline__ void mma_bf16_16808(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t b) {
    asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};\n"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a0), "r"(a1), "r"(b));
}

__global__ void __launch_bounds__(FF_THREADS, 1) feed_forward_kernel(const FeedForwardArgs a) {
    extern __shared__ __align__(16) unsigned char ff_smem[];
    __shared__ __align__(8) uint64_t w_bar[1];
    __shared__ float ss_s[FF_WARPS], inv_s[FF_MAX_ROWS];
    const int wide = ff_stride(a.width), narrow = ff_stride(a.cols);
    unsigned char* w_s = ff_smem;                                  // [2 * cols][wide]: eight gate rows, the same eight up rows, ...
    unsigned char* x_s = w_s + (size_t)2 * a.cols * wide;          // [8][wide]
    unsigned char* d_s = x_s + (size_t)FF_MAX_ROWS * wide;         // [width][narrow]
    unsigned char* act_s = d_s + (size_t)a.width * narrow;         // [8][narrow]
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
    const int first = blockIdx.x * a.cols, here = min(a.cols, a.inter - first);   // (a multiple of eight, as inter and cols are)

    // ---- weights: a bulk copy per gate and up row; the down weight's pieces by 16 bytes
    if (warp == 0) {
        if (lane == 0) {
            mbar_init(&w_bar[0], 1);
            mbar_expect_tx(&w_bar[0], (uint32_t)(2 * here * a.width * 2));
        }
        __syncwarp();
        for (int r = lane; r < 2 * here; r += 32) {
            const int col = first + (r >> 4) * 8 + (r & 7), row = (r & 8) ? a.inter + col : col;
            bulk_copy_g2s(w_s + (size_t)r * wide, a.gate_up + (size_t)row * a.ldg, (uint32_t)a.width * 2, &w_bar[0]);
        }
    }
    {
        const int pieces = a.cols / 8, rows_on = FF_THREADS / pieces, pieces_on = FF_THREADS - rows_on * pieces;
        for (int n = threadIdx.x / pieces, c = threadIdx.x - n * pieces; n < a.width;) {
            cp_async_16(d_s + (size_t)n * narrow + c * 16, a.down + (size_t)n * a.ldd + first + (8 * c < here ? 8 * c : 0), 8 * c < here);
            n += rows_on, c += pieces_on;
            if (c >= pieces) c -= pieces, ++n;
        }
    }
    cp_async_commit();
    // columns beyond the last: zeros; token rows beyond the step's: zeros
    for (int i = threadIdx.x; i < 2 * (a.cols - here) * (wide / 16); i += FF_THREADS)
        reinterpret_cast<uint4*>(w_s + (size_t)2 * here * wide)[i] = make_uint4(0, 0, 0, 0);
    for (int i = threadIdx.x; i < (FF_MAX_ROWS - a.rows) * (wide / 16); i += FF_THREADS)
        reinterpret_cast<uint4*>(x_s + (size_t)a.rows * wide)[i] = make_uint4(0, 0, 0, 0);
    grid_launch_dependents();

    // ---- token rows: 16, 8, 4 or 2 warps a row, each a run of its columns
    const int share = 1 << a.row_warps_log, row = warp >> a.row_warps_log, run = (a.width / 4 + share - 1) >> a.row_warps_log << 2;
    const int c0 = (warp & (share - 1)) * run, c1 = min(a.width, c0 + run);
    uint2 norm_first[4];          // constants: asked for before the wait
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        const int c = c0 + (u * 32 + lane) * 4;
        norm_first[u] = row < a.rows && c < c1 ? *reinterpret_cast<const uint2*>(a.norm_w + c) : make_uint2(0u, 0u);
    }
    grid_dependency_wait();
    if (row < a.rows) {
        const float* h = a.hidden + (size_t)row * a.width;
        unsigned char* dst = x_s + (size_t)row * wide;
        float ss = 0.f;
        for (int base = c0; base < c1; base += 512) {
            float4 x[4];
            uint2 w[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int c = base + (u * 32 + lane) * 4;
                x[u] = c < c1 ? *reinterpret_cast<const float4*>(h + c) : make_float4(0.f, 0.f, 0.f, 0.f);
                w[u] = base == c0 ? norm_first[u] : c < c1 ? *reinterpret_cast<const uint2*>(a.norm_w + c) : make_uint2(0u, 0u);
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int c = base + (u * 32 + lane) * 4;
                if (c >= c1) continue;
                ss += x[u].x * x[u].x + x[u].y * x[u].y + x[u].z * x[u].z + x[u].w * x[u].w;
                const __nv_bfloat162 w01 = *reinterpret_cast<const __nv_bfloat162*>(&w[u].x), w23 = *reinterpret_cast<const __nv_bfloat162*>(&w[u].y);
                *reinterpret_cast<uint2*>(dst + c * 2) = make_uint2(pack_bf16(x[u].x * __low2float(w01), x[u].y * __high2float(w01)),
                                                                    pack_bf16(x[u].z * __low2float(w23), x[u].w * __high2float(w23)));
            }
        }
        ss = warp_sum(ss);
        if (lane == 0) ss_s[warp] = ss;
    }
    __syncthreads();
    if (threadIdx.x >= FF_THREADS - 32 && lane < a.rows) {         // (read behind the next barriers)
        float ss = 0.f;
        for (int p = 0; p < share; ++p) ss += ss_s[lane * share + p];
        inv_s[lane] = 1.0f / sqrtf(ss / (float)a.width + a.eps);
    }
    if (!mbar_wait(&w_bar[0], 0) && lane == 0) atomicOr(a.err, QF_ERR_COPY_TIMEOUT);

    // ---- gate and up: a tile is eight columns, its M side their gate and their up rows; the warps of a tile take blocks of 32 k in turn
    const int tiles = a.cols / 8, tile = warp * a.each_recip >> 16, n_kb = a.width / 32;
    float acc[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
    if (tile < tiles) {
        const unsigned char* w_lane = w_s + (size_t)(tile * 16 + (lane & 15)) * wide + (lane >> 4) * 16;
        const unsigned char* x_lane = x_s + (size_t)(lane & 7) * wide + (lane >> 3) * 16;
        for (int kb = warp - tile * a.each; kb < n_kb; kb += a.each) {
            uint32_t w0[4], w1[4], x[4];
            ldmatrix_x4(x, x_lane + kb * 64);
            ldmatrix_x4(w0, w_lane + kb * 64);
            ldmatrix_x4(w1, w_lane + kb * 64 + 32);
            mma_bf16_16816(acc[0], w0, x[0], x[1]);
            mma_bf16_16816(acc[1], w1, x[2], x[3]);
        }
    }
    __syncthreads();              // every warp is done with the gate and up rows: the parts of the sums take their place
    float* part = reinterpret_cast<float*>(w_s);                   // [FF_WARPS][4][32]
#pragma unroll
    for (int e = 0; e < 4; ++e) part[(warp * 4 + e) * 32 + lane] = acc[0][e] + acc[1][e];
    cp_async_wait<0>();
    __syncthreads();
    if (warp < tiles) {
        // the lane holds, of token rows 2 t and 2 t + 1, gate and up of the tile's column g
        float sum[4] = {0.f, 0.f, 0.f, 0.f};
        for (int w = 0; w < a.each; ++w)
#pragma unroll
            for (int e = 0; e < 4; ++e) sum[e] += part[((warp * a.each + w) * 4 + e) * 32 + lane];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int m = 2 * t + e;
            float out = 0.f;
            if (m < a.rows) {
                const float gate = sum[e] * inv_s[m], up = sum[2 + e] * inv_s[m];
                out = gate / (1.0f + expf(-gate)) * up;
            }
            *reinterpret_cast<bf16*>(act_s + (size_t)m * narrow + (warp * 8 + g) * 2) = __float2bfloat16_rn(out);
        }
    }
    __syncthreads();

    // ---- down: token rows are the M side (its second eight rows repeat the first and are dropped), 16 outputs a turn; the blocks begin at
    // different outputs, so that they do not all add into the same few lines at a time
    const int groups = a.width / 16, steps = a.cols / 16, from = (int)((blockIdx.x * 5u) % (unsigned)groups);
    const bool odd = lane & 1, rest = a.cols & 8;
    const unsigned char* act_lane = act_s + (size_t)(lane & 7) * narrow;
    for (int i = warp; i < groups; i += FF_WARPS) {
        const int n0 = (i + from < groups ? i + from : i + from - groups) * 16;
        float c[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
        for (int ks = 0; ks < steps; ++ks) {
            uint32_t x[4], w[4];
            ldmatrix_x4(x, act_lane + ks * 32 + (lane >> 4) * 16);
            ldmatrix_x4(w, d_s + (size_t)(n0 + (lane >> 4) * 8 + (lane & 7)) * narrow + ks * 32 + ((lane >> 3) & 1) * 16);
            mma_bf16_16816(c[0], x, w[0], w[1]);
            mma_bf16_16816(c[1], x, w[2], w[3]);
        }
        if (rest) {
            uint32_t x[2], w[2];
            ldmatrix_x2(x, act_lane + steps * 32);
            ldmatrix_x2(w, d_s + (size_t)(n0 + (lane & 15)) * narrow + steps * 32);
            mma_bf16_16808(c[0], x[0], x[1], w[0]);
            mma_bf16_16808(c[1], x[0], x[1], w[1]);
        }
        // neighbours swap one tile's pair: the even lane has four adjacent outputs of the first eight, the odd lane of the second
        const float s0 = odd ? c[0][0] : c[1][0], s1 = odd ? c[0][1] : c[1][1];
        const float r0 = __shfl_xor_sync(0xffffffffu, s0, 1), r1 = __shfl_xor_sync(0xffffffffu, s1, 1);
        if (g < a.rows) {
            const float4 sum = odd ? make_float4(r0, r1, c[1][0], c[1][1]) : make_float4(c[0][0], c[0][1], r0, r1);
            atomicAdd(reinterpret_cast<float4*>(a.sums + (size_t)g * a.width + n0 + (odd ? 8 : 0) + 4 * (t >> 1)), sum);
        }
    }
}

// hidden += sums; sums = 0: where what is pending is to be in the stream and no projection follows that takes it along.
__global__ void __launch_bounds__(256) take_sums_kernel(float* __restrict__ hidden, float* __restrict__ sums, long long n) {
    grid_chain_entry();
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    hidden[i] += sums[i];
    sums[i] = 0.f;
}

// Columns of a block and bytes of shared memory; 0 columns where the layer does not fit.
static int ff_columns(int rows, int width, int inter, int sms, size_t* smem) {
    if (rows < 1 || rows > FF_MAX_ROWS || width <= 0 || width % 32 || inter <= 0 || inter % 8 || sms <= 0) return 0;
    const int cols = ((inter + sms - 1) / sms + 7) / 8 * 8;
    if (cols > FF_MAX_COLS) return 0;
    *smem = (size_t)(2 * cols + FF_MAX_ROWS) * ff_stride(width) + (size_t)(width + FF_MAX_ROWS) * ff_stride(cols);
    const size_t parts = (size_t)FF_WARPS * 4 * 32 * 4;       // (take the gate and up rows' place)
    return *smem <= 226 * 1024 && (size_t)2 * cols * ff_stride(width) >= parts ? cols : 0;
}

// Blocks that the kernel would run with, 0 where it does not take the sizes.
QF_EXPORT int qf_feed_forward_blocks(int rows, int width, int inter) {
    size_t smem;
    const int cols = ff_columns(rows, width, inter, qf_sm_count(), &smem);
    return cols ? (inter + cols - 1) / cols : 0;
}

QF_EXPORT int qf_feed_forward(const FeedForwardArgs* args, cudaStream_t stream) {
    FeedForwardArgs a = *args;
    size_t smem;
    a.cols = ff_columns(a.rows, a.width, a.inter, qf_sm_count(), &smem);
    a.row_warps_log = a.rows == 1 ? 4 : a.rows == 2 ? 3 : a.rows <= 4 ? 2 : 1;
    a.each = a.cols ? FF_WARPS / (a.cols / 8) : 1;
    a.each_recip = (65536 + a.each - 1) / a.each;
    if (!a.cols || a.ldg < a.width || a.ldg % 8 || a.ldd < a.inter || a.ldd % 8) return (int)cudaErrorInvalidValue;
    if (((uintptr_t)a.hidden | (uintptr_t)a.gate_up | (uintptr_t)a.down | (uintptr_t)a.sums) % 16 || (uintptr_t)a.norm_w % 8) return (int)cudaErrorInvalidValue;
    cudaError_t e = cudaFuncSetAttribute(feed_forward_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
    return (int)launch_pdl(feed_forward_kernel, dim3((a.inter + a.cols - 1) / a.cols), dim3(FF_THREADS), smem, stream, a);
}

QF_EXPORT int qf_take_sums(float* hidden, float* sums, long long n, cudaStream_t stream) {
    if (n <= 0) return 0;
    return (int)launch_pdl(take_sums_kernel, dim3((unsigned)((n + 255) / 256)), dim3(256), 0, stream, hidden, sums, n);
}
