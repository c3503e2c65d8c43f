// What the recurrences written out over chunks of tokens share: float32 operands in three bfloat16 parts, tiles in shared memory.
#pragma once
#include "mma.cuh"

// x = hi + mid + lo, each a bfloat16 number (the upper half of a float32): cut off, subtract (exactly), twice.
struct Thirds {
    uint32_t hi, mid, lo;     // two neighbouring numbers each, the first in the lower half
};
__device__ __forceinline__ Thirds thirds(float x0, float x1) {
    Thirds r;
    uint32_t a = __float_as_uint(x0), b = __float_as_uint(x1);
    r.hi = __byte_perm(a, b, 0x7632);
    float s0 = x0 - __uint_as_float(a & 0xffff0000u), s1 = x1 - __uint_as_float(b & 0xffff0000u);
    a = __float_as_uint(s0), b = __float_as_uint(s1);
    r.mid = __byte_perm(a, b, 0x7632);
    s0 -= __uint_as_float(a & 0xffff0000u), s1 -= __uint_as_float(b & 0xffff0000u);
    r.lo = __byte_perm(__float_as_uint(s0), __float_as_uint(s1), 0x7632);
    return r;
}
__device__ __forceinline__ float lower_bf16(uint32_t pair) { return __uint_as_float(pair << 16); }
__device__ __forceinline__ float upper_bf16(uint32_t pair) { return __uint_as_float(pair & 0xffff0000u); }

// Byte offset of 16-byte piece `piece` of row `row` in a tile of WIDTH bfloat16 columns, pieces permuted so that eight
// neighbouring rows read at one piece lie in eight different bank groups.
template <int WIDTH>
__device__ __forceinline__ uint32_t tile_at(int row, int piece) {
    return (uint32_t)(row * (2 * WIDTH) + ((piece ^ (row & 7)) << 4));
}
// `rows` rows of a [.][WIDTH] tile from global rows `stride` elements apart; rows from n_here on become zeros.
template <int CHUNK, int WIDTH>
__device__ __forceinline__ void fetch_tile(unsigned char* dst, const bf16* src, int stride, int n_here, int first, int threads) {
    constexpr int PIECES = WIDTH / 8;
    for (int i = first; i < CHUNK * PIECES; i += threads) {
        const int row = i / PIECES, piece = i % PIECES;
        const bool there = row < n_here;
        cp_async_16(dst + tile_at<WIDTH>(row, piece), there ? src + (size_t)row * stride + piece * 8 : src, there);
    }
}
// The first record of a sequence: sequence s owns records cu_q[s] / CHUNK + s onwards, as many as its chunks at most.
template <int CHUNK> __device__ __forceinline__ long long first_record(const int* cu_q, int seq) { return cu_q[seq] / CHUNK + seq; }
