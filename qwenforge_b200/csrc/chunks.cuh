// What the recurrences written out over chunks of tokens share: float32 operands in three bfloat16 parts, tiles in shared memory.
#pragma once
#include "mma.cuh"

// x = hi + mid + lo, each a bfloat16 number: round to the nearest, subtract (exactly), twice; the last remainder is one as it stands. (Cut
// off instead of rounded, the remainders are up to twice as large and all of one sign, and what a product of two such sums
// leaves out adds up.)
struct Thirds {
    uint32_t hi, mid, lo;     // two neighbouring numbers each, the first in the lower half
};
__device__ __forceinline__ float lower_bf16(uint32_t pair) { return __uint_as_float(pair << 16); }
__device__ __forceinline__ float upper_bf16(uint32_t pair) { return __uint_as_float(pair & 0xffff0000u); }
__device__ __forceinline__ Thirds thirds(float x0, float x1) {
    Thirds r;
    r.hi = pack_bf16(x0, x1);
    float s0 = x0 - lower_bf16(r.hi), s1 = x1 - upper_bf16(r.hi);
    r.mid = pack_bf16(s0, s1);
    s0 -= lower_bf16(r.mid), s1 -= upper_bf16(r.mid);
    r.lo = __byte_perm(__float_as_uint(s0), __float_as_uint(s1), 0x7632);
    return r;
}

// A product of many decays with what its roundings left out beside it (the remainder of a product of two float32 is one itself): the
// scan rounds a state once a token, so a chunk's weights must not bring as many roundings of their own on top of its sums'.
struct Running {
    float value, rest;
    __device__ __forceinline__ void times(float w) {
        const float p = value * w, left = fmaf(value, w, -p);
        rest = fmaf(rest, w, left), value = p;
    }
    __device__ __forceinline__ void times(const Running& w) {
        const float p = value * w.value, left = fmaf(value, w.value, -p);
        rest = fmaf(value, w.rest, fmaf(rest, w.value, left)), value = p;
    }
    __device__ __forceinline__ float of(float x) const { return fmaf(x, value, x * rest); }   // x times the product, rounded once
};

// D = A[16x16] B[16x8], the first product of a sum of its own. The tensor cores cut a sum off behind its 24th bit, towards zero, with every
// product that is added to it. So the recurrences' sums over tokens and state rows are not left to them: the products of 16
// tokens or rows (least parts first) make a sum of their own, and that is added to the running one by a float32 addition, which rounds.
struct MmaFirst {
    __device__ __forceinline__ void operator()(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) const {
        asm volatile(
            "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};\n"
            : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
            : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
    }
};
struct MmaNext {
    __device__ __forceinline__ void operator()(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) const { mma_bf16_16816(d, a, b0, b1); }
};
// Two additions an instruction, each rounded as one alone.
template <int N> __device__ __forceinline__ void add_sums(float (*to)[4], const float (&sum)[N][4]) {
#pragma unroll
    for (int i = 0; i < N; ++i)
#pragma unroll
        for (int e = 0; e < 4; e += 2)
            asm("{\n\t.reg .b64 a, b;\n\tmov.b64 a, {%0, %1};\n\tmov.b64 b, {%2, %3};\n\tadd.rn.f32x2 a, a, b;\n\tmov.b64 {%0, %1}, a;\n\t}"
                : "+f"(to[i][e]), "+f"(to[i][e + 1])
                : "f"(sum[i][e]), "f"(sum[i][e + 1]));
}

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
// A call works through its chunks in portions of the same `each` chunks of every sequence, so that what it keeps per chunk has a bound:
// portion [chunk0, chunk0 + each). each == 0: all chunks at once.
struct Portion {
    int chunk0, each;
    float* carry;     // each > 0: a state per sequence [heads][D][vdim], [heads][D] between the portions of those that have no slot
};
// The record of a sequence's chunk, all at once: sequence s owns records cu_q[s] / CHUNK + s onwards, as many as its chunks at most.
template <int CHUNK> __device__ __forceinline__ long long record_of(const Portion& p, const int* cu_q, int seq, int chunk) {
    return p.each > 0 ? (long long)seq * p.each + chunk - p.chunk0 : (long long)cu_q[seq] / CHUNK + seq + chunk;
}
