// Shared by the two tcgen05 expert kernels (grouped_tc.cu: activations gathered per tile, any layout; grouped_tc_tiled.cu:
// tile-blocked activations): launch arguments, output modes, and the dequantization of packed codes to the F16 operand.
#pragma once

#include "experts.cuh"
#include "tc_ptx.cuh"

namespace sxb {

// kTcPartialBf16: kTcPartial with the per-slot dots stored as BF16 bits (N * 2 bytes a slot) - for the epilogue it is the
// plain gather's store on h rows.  A mode of its own, so that the per-token store code of every mode stays one short form.
// kTcHcUp: a dense projection whose epilogue is the stream combine of the hyper-connection up mix (TcHcUp below); the
// kernel for tile-blocked activations only.
enum TcMode { kTcGather = 0, kTcSwiglu = 1, kTcPartial = 2, kTcPartialBf16 = 3, kTcHcUp = 4 };

// kTcHcUp (kernels/hc_wmma.hip:244-272): the weight's rows are W_up's rows in the order that puts the H = 4 streams of an
// output column into adjacent tensor-memory lanes - row rb * 128 + q * 32 + l is stream l & 3 of column
// rb * 32 + q * 8 + (l >> 2) - so that a lane finishes z -> sigmoid(z) * x * inv * (1 + norm_w) for its stream and two
// shuffles add the four streams: u[t, j] = (1/4) sum_s ..., rounded once to the activation dtype.  No z in memory.
struct TcHcUp {
    const void *x;        // the streams X [M, 4 d], FP32 or BF16
    const float *inv;     // [M, 4]
    const float *norm_w;  // [4 d]
    void *u;              // [M, d] in x's dtype
    int64_t d;
    int f32;              // x and u are FP32 (else BF16)
};

struct TcArgs {
    const uint16_t *x;  // activations: BF16 or F16 bits, see x_kind
    const uint8_t *q;
    const uint16_t *scale, *minv;
    int64_t N, K;     // weight rows per expert, codes per row
    int64_t A, E;     // slots per token, experts in the view
    const int32_t *ws;
    RouteWords L;
    void *out;
    int x_kind;   // activations: 0 BF16, 1 F16 in natural k order, 2 F16 in this weight operand's k order (staged),
                  // 3 F16 "tile-blocked" (see tiled_offset): one bulk copy per k-block
    int out_f16;  // SwiGLU output h: 0 BF16, 1 F16 bits of its BF16 rounding, 2 the same in the Q4 operand's k order,
                  // 3 / 4 tile-blocked for a Q4 / Q8 down operand
    uint32_t *status;  // >= 3 words: {2, item, role} on a wait that ran out
    int64_t dense_M;   // > 0: a dense projection - no grouping workspace, one group holding rows 0 .. dense_M - 1 in order
    int dense_tile;    // its rows a tile (the kernel for tile-blocked activations), a multiple of 16
    unsigned long long wait_limit_ns;  // bound of every device-side wait
    int test_skip_slot;  // >= 0: CTA 0 never issues ring slot number test_skip_slot, so a wait runs out (tests only)
    TcHcUp hc;           // kTcHcUp only
};

// Eight weights = one 16-byte chunk of the A line, from one word of Q4 codes or two words of Q8 codes.
// w = code * s + m with one F16 rounding (kernels/wmma_gemm.hpp:116-129).
__device__ inline uint4 dequant_q4_word(uint32_t w, __half2 s, __half2 m) {
    const __half2 k1024 = __float2half2_rn(1024.f), k16th = __float2half2_rn(0.0625f);
    const uint32_t w8 = w >> 8;
    // (w & 0x000F000F) | 0x64006400 = (1024 + n0, 1024 + n4); the 0x00F0 nibbles give 1024 + 16 n.  The sixteenth goes to the code,
    // where it is exact: s / 16 would be an F16 subnormal from s < 2^-10 on, and short of bits from 2^-13 on.
    const __half2 p0 = __hsub2(u32_as_h2((w & 0x000F000Fu) | 0x64006400u), k1024);
    const __half2 p1 = __hmul2(__hsub2(u32_as_h2((w & 0x00F000F0u) | 0x64006400u), k1024), k16th);
    const __half2 p2 = __hsub2(u32_as_h2((w8 & 0x000F000Fu) | 0x64006400u), k1024);
    const __half2 p3 = __hmul2(__hsub2(u32_as_h2((w8 & 0x00F000F0u) | 0x64006400u), k1024), k16th);
    uint4 d;
    d.x = h2_as_u32(__hfma2(p0, s, m)), d.y = h2_as_u32(__hfma2(p1, s, m));
    d.z = h2_as_u32(__hfma2(p2, s, m)), d.w = h2_as_u32(__hfma2(p3, s, m));
    return d;
}
__device__ inline uint4 dequant_q8_words(uint32_t w0, uint32_t w1, __half2 s, __half2 m) {
    const __half2 k1024 = __float2half2_rn(1024.f);
    uint4 d;  // __byte_perm(w, 0x64646464, 0x4140) = (0x6400 | b0, 0x6400 | b1) = (1024 + b0, 1024 + b1)
    d.x = h2_as_u32(__hfma2(__hsub2(u32_as_h2(__byte_perm(w0, 0x64646464u, 0x4140)), k1024), s, m));
    d.y = h2_as_u32(__hfma2(__hsub2(u32_as_h2(__byte_perm(w0, 0x64646464u, 0x4342)), k1024), s, m));
    d.z = h2_as_u32(__hfma2(__hsub2(u32_as_h2(__byte_perm(w1, 0x64646464u, 0x4140)), k1024), s, m));
    d.w = h2_as_u32(__hfma2(__hsub2(u32_as_h2(__byte_perm(w1, 0x64646464u, 0x4342)), k1024), s, m));
    return d;
}

// The same weights times a power of two, with nothing but a mask before the multiply-add: a code n in the low mantissa bits
// of an F16 with a zero exponent field IS the subnormal n * 2^-24 (n * 2^-20 four bits further up), so
// fma(n * 2^-24, s * 2^k, m * 2^(k - 24)) is (n * s + m) * 2^(k - 24), rounded once as dequant_q4_word rounds it.  k is one
// per weight row, so that the accumulators of the row carry the factor 2^(k - 24) out of the contraction; s and m come in
// with their factors, s16 = s / 16.  Nine instructions per eight codes instead of eighteen (adding the 0x6400 and taking the
// 1024 off again): a 128 x 128 block took its four warps 202 SM cycles instead of 337.
// Rounding: s * 2^k < 2^15 for the row's largest s, so the row's largest weights lie between 2^-9 and 1/2 and keep their
// eleven bits; those of a group whose scale is 2^7 or more below the largest can lose bits to F16's subnormals, so rows with
// such groups go without a power of two (kScaleSpread in grouped_tc_tiled.cu).
__device__ inline uint4 dequant_q4_scaled(uint32_t w, __half2 s, __half2 s16, __half2 m) {
    const uint32_t w8 = w >> 8;
    uint4 d;
    d.x = h2_as_u32(__hfma2(u32_as_h2(w & 0x000F000Fu), s, m)), d.y = h2_as_u32(__hfma2(u32_as_h2(w & 0x00F000F0u), s16, m));
    d.z = h2_as_u32(__hfma2(u32_as_h2(w8 & 0x000F000Fu), s, m)), d.w = h2_as_u32(__hfma2(u32_as_h2(w8 & 0x00F000F0u), s16, m));
    return d;
}
__device__ inline uint4 dequant_q8_scaled(uint32_t w0, uint32_t w1, __half2 s, __half2 m) {
    uint4 d;  // __byte_perm(w, 0, 0x4140) = the subnormals (b0, b1) * 2^-24
    d.x = h2_as_u32(__hfma2(u32_as_h2(__byte_perm(w0, 0u, 0x4140)), s, m)), d.y = h2_as_u32(__hfma2(u32_as_h2(__byte_perm(w0, 0u, 0x4342)), s, m));
    d.z = h2_as_u32(__hfma2(u32_as_h2(__byte_perm(w1, 0u, 0x4140)), s, m)), d.w = h2_as_u32(__hfma2(u32_as_h2(__byte_perm(w1, 0u, 0x4342)), s, m));
    return d;
}

// grouped_tc_tiled.cu: the kernel for tile-blocked activations (a.x_kind == 3).  Same arguments, same outputs.
template <int BITS, int MODE>
int launch_tiled_tc(const char *fn, TcArgs a, int64_t G, cudaStream_t st);

}  // namespace sxb
