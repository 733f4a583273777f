// A float32 product on tensor cores: every operand is the exact sum of three bfloat16 numbers
// (a0 = a rounded, a1 = a - a0 rounded, a2 = the rest: 3 x 8 bits hold float32's 24; Henry, Tang and Heinecke, "Leveraging the bfloat16
// Artificial Intelligence Datatype For Higher-Precision Computations", 2019), and of the nine products of parts six are summed, in float32
// accumulators.  What is left out (a1 b2, a2 b1, a2 b2) is at most 2^-24 of a term and 5.7e-9 of a whole product's norm; what bounds
// the error is the accumulator, which drops what falls off its end instead of rounding: so it never holds more than 64 terms, the
// parts' small products come first and the four steps of a0 b0 last, and everything above 64 terms is added in registers, rounded.
//
// The order of an output's sum depends on K alone: K is cut into blocks of 64, blocks into up to 4 or 8
// ranges (`fs_range_blocks`); a block is one chain of MMA steps of 16 terms (for each of its four steps
// x2 w0, x0 w2, x1 w1, x1 w0, x0 w1; then x0 w0 of the four); a range adds its blocks, the output its ranges, in
// ascending order, the bias last.  Step j of a block takes its terms 8 j .. 8 j + 7 and 32 + 8 j .. 32 + 8 j + 7 (so that
// eight lanes that read 16 bytes each of a row read 128 in a row).  `mma.sync` m16n8k16 and `tcgen05.mma` with K = 16 give the same bits
// for the same 16 terms wherever in a tile they stand and in whatever order (tests compare them), so steps of
// few tokens and of many take different kernels and a row's bits are the same in both.
//
// Relative error of whole products of normal numbers against 64 bits, float32 FMA chains / this: 896 terms 2.0e-7 / 9.7e-8,
// 4,864 terms 3.2e-7 / 1.15e-7.  One chain of 16 steps instead of four would have 2.3e-7 by itself, all of
// it towards zero.  What this cannot hold are operands below about 2^-109: their third parts are less than bfloat16's
// smallest number, and what is lost of an operand is at most 2^-134 (of 1e-38 some seven bits are left).  That goes for all that
// multiply parts: this product, attention_f32.cu and recurrent_chunks.cu.
#pragma once

#include "mma.cuh"

namespace somi {

constexpr int kFsBK = 64;                 // terms of a block
inline int fs_range_blocks(int blocks) {  // blocks of a range: 8 ranges from 2,048 terms on, else 4
    const int ranges = blocks >= 32 ? 8 : 4;
    return (blocks + ranges - 1) / ranges;
}

// (lo, hi) minus the pair of bfloat16 numbers p: exact where p is what (lo, hi) rounds to.
__device__ __forceinline__ void fs_rest(uint32_t p, float& lo, float& hi) {
    asm("{\n.reg .b16 l, h, m;\nmov.b32 {l, h}, %2;\nmov.b16 m, 0xBF80;\n"
        "fma.rn.f32.bf16 %0, l, m, %0;\nfma.rn.f32.bf16 %1, h, m, %1;\n}\n"
        : "+f"(lo), "+f"(hi)
        : "r"(p));
}
// Two numbers' parts, packed in pairs.
__device__ __forceinline__ void fs_split(float lo, float hi, uint32_t& p0, uint32_t& p1, uint32_t& p2) {
    p0 = pack_bf16(lo, hi);
    fs_rest(p0, lo, hi);
    p1 = pack_bf16(lo, hi);
    fs_rest(p1, lo, hi);
    p2 = pack_bf16(lo, hi);
}

// The sum as plain FMAs, for outputs that came out as infinity or NaN: an infinite operand has no second
// part (inf - inf), and one above bfloat16's range rounds to infinity.  Rare, so only correct.
__device__ __forceinline__ float fs_plain_sum(const float* x, const float* w, int K) {
    float s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f;
#pragma unroll 1
    for (int k = 0; k < K; k += 4) {      // (K is a multiple of 4)
        const float4 a = *reinterpret_cast<const float4*>(x + k), b = *reinterpret_cast<const float4*>(w + k);
        s0 = fmaf(a.x, b.x, s0);
        s1 = fmaf(a.y, b.y, s1);
        s2 = fmaf(a.z, b.z, s2);
        s3 = fmaf(a.w, b.w, s3);
    }
    return (s0 + s1) + (s2 + s3);
}
__device__ __forceinline__ bool fs_finite(float v) { return fabsf(v) <= 3.4028234664e38f; }
// Whether v is the sum of three parts: finite, and below (2 - 2^-8) 2^127, from where on bfloat16 rounds to infinity.
constexpr float kFsNoParts = 3.39617752923e38f;
__device__ __forceinline__ bool fs_has_parts(float v) { return fabsf(v) < kFsNoParts; }
// The larger magnitude, or NaN: below kFsNoParts only where all numbers have parts.
__device__ __forceinline__ float fs_largest(float m, float v) {
    asm("max.NaN.f32 %0, %0, %1;\n" : "+f"(m) : "f"(fabsf(v)));
    return m;
}

struct FsArgs {
    const float *x, *w, *bias;
    float* y;
    int M, N, K, batch, w_constant;
    long long ldx, ldy, bsx, bsw, bsy;
};

constexpr long long kFsMostApart = 0x7fffffffll / 144;

// Whether this way takes the product: from 512 terms on (64 terms in one chain have an error of 6.5e-8 here and of 4.4e-8
// as FMAs, 256 terms 7.4e-8 and 7.7e-8), up to what a cluster's shared memory holds of a row's blocks, with outputs for at
// least half a tile, and rows that can be read 16 bytes at a time and lie no more than `kFsMostApart` floats apart (a tile's
// are found by 32-bit offsets).  Never by the number of rows: a row's bits must not depend on it.
inline bool fs_takes(const FsArgs& a) {
    return a.ldx <= kFsMostApart && a.K >= 512 && a.K <= 20480 && a.N >= 64 && ((a.K | a.ldx | a.bsx | a.bsw) & 3) == 0 &&
           ((reinterpret_cast<uintptr_t>(a.x) | reinterpret_cast<uintptr_t>(a.w)) & 15) == 0;
}
int fs_launch_rows(const FsArgs& a, cudaStream_t stream);    // up to 16 rows (gemm_f32_rows.cu)
int fs_launch_tiles(const FsArgs& a, cudaStream_t stream);   // more (gemm_f32_tcgen05.cu)

}  // namespace somi
