// Warp-level MMA with FP32 arithmetic for skinny products: 16 weight rows x 8 tokens x 16 k of BF16 operands, exact products, FP32
// sums.  An FP32 operand goes through as three BF16 planes, which together hold its 24 bits, each plane's products as exact.
//
// k inside a run of 32 is permuted the same way on both operands, which a dot product does not notice: lane (g = lane / 4, c = lane
// % 4) holds elements 8 c .. 8 c + 7 of its weight rows g and g + 8 and of its token g, i.e. whole runs of eight consecutive
// elements that a 16-byte load fetches; the run's first MMA takes elements 0 - 3, the second 4 - 7.
// Results: d[0], d[1] = row g x tokens 2 c, 2 c + 1; d[2], d[3] = row g + 8 x the same.
#pragma once

#include "common.cuh"

namespace sxb {

constexpr int kMmaRows = 16, kMmaTokens = 8, kMmaRun = 32;  // weight rows, tokens and k of a step

__device__ inline void mma_bf16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// d += a 32-k run: a, b = the lane's eight elements of rows g and g + 8, x = of its token, as BF16 pairs.
__device__ inline void mma_run(float (&d)[4], const uint4 &a, const uint4 &b, const uint4 &x) {
    mma_bf16(d, a.x, b.x, a.y, b.y, x.x, x.y);
    mma_bf16(d, a.z, b.z, a.w, b.w, x.z, x.w);
}

// Pairs of FP32 values in one instruction, each rounded as on its own.
__device__ inline uint64_t pair(float a, float b) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ inline void unpair(uint64_t v, float &a, float &b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ inline uint64_t mul_pair(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ inline uint64_t fma_pair(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ inline uint64_t add_pair(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

// Two FP32 values that fit BF16 as a pair (the first in the lower half).
__device__ inline uint32_t pack_bf16_exact(float lo, float hi) { return __byte_perm(__float_as_uint(lo), __float_as_uint(hi), 0x7632); }
// The upper sixteen bits of an FP32 value: a BF16, and what is left of the value is an FP32 with eight bits fewer.
__device__ inline float bf16_part(float v) { return __uint_as_float(__float_as_uint(v) & 0xffff0000u); }

// Eight FP32 values as three BF16 planes whose sum they are, bit for bit (down to BF16's smallest exponent).
__device__ inline void split_planes(const float (&v)[8], uint4 (&p)[3]) {
    uint32_t w[3][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float a = v[2 * i], b = v[2 * i + 1];
        const float a1 = a - bf16_part(a), b1 = b - bf16_part(b);
        w[0][i] = pack_bf16_exact(a, b), w[1][i] = pack_bf16_exact(a1, b1);
        w[2][i] = pack_bf16_exact(a1 - bf16_part(a1), b1 - bf16_part(b1));
    }
#pragma unroll
    for (int j = 0; j < 3; ++j) p[j] = make_uint4(w[j][0], w[j][1], w[j][2], w[j][3]);
}

// 2^23 plus the code whose weight scale * code + min comes nearest to zero.  Codes less that one, with the rest in the min (shifted_min), are
// as large as their weights: sums of codes as they are carry that code times sum(x), which the min takes off again, and the rounding of the larger
// sums stays; and less the middle of their range a weight of zero takes bits from the rest of its dot when its activation is large.
constexpr float kCodeBias = 0x1p23f;
template <int BITS>
__device__ inline float zero_code(float s, float m) {
    constexpr float kTop = (1 << BITS) - 1;
    float inv;  // any code is right, if not as good: an approximate reciprocal will do
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(inv) : "f"(s));
    return fmaf(__saturatef(inv * (m * (-1.f / kTop))), kTop, kCodeBias);  // NaN saturates to 0
}
__device__ inline float shifted_min(float s, float m, float zero) {
    const float z = zero - kCodeBias;
    return z > 0.f ? fmaf(z, s, m) : m;
}
// A row group's scale and zero code in a word, for the lanes that share the row.
template <int BITS>
__device__ inline void pack_group(uint16_t s, uint16_t m, uint32_t &word, float &min) {
    const float zero = zero_code<BITS>(bf16_bits_to_f32(s), bf16_bits_to_f32(m));
    word = (uint32_t)s << 16 | (__float_as_uint(zero) & 0xffu), min = shifted_min(bf16_bits_to_f32(s), bf16_bits_to_f32(m), zero);
}
__device__ inline float group_scale(uint32_t word) { return __uint_as_float(word & 0xffff0000u); }
__device__ inline float group_zero(uint32_t word) { return __uint_as_float((word & 0xffu) | 0x4B000000u); }

// The lane's eight codes of a row, less zero - 2^23, as BF16 pairs: Q8 from two words, Q4 from one (w1 unused).
template <int BITS>
__device__ inline uint4 codes_bf16(uint32_t w0, uint32_t w1, float zero) {
    uint32_t r[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        uint32_t lo, hi;  // 2^23 + code, less `zero`: no conversion instruction, which runs at a quarter rate
        if (BITS == 8) {
            const uint32_t w = i < 2 ? w0 : w1;
            lo = __byte_perm(w, 0x4B000000u, (i & 1) ? 0x7442 : 0x7440), hi = __byte_perm(w, 0x4B000000u, (i & 1) ? 0x7443 : 0x7441);
        } else {
            lo = 0x4B000000u | ((w0 >> (8 * i)) & 15u), hi = 0x4B000000u | ((w0 >> (8 * i + 4)) & 15u);
        }
        float a, b;
        unpair(add_pair(pair(__uint_as_float(lo), __uint_as_float(hi)), pair(-zero, -zero)), a, b);
        r[i] = pack_bf16_exact(a, b);
    }
    return make_uint4(r[0], r[1], r[2], r[3]);
}

// A lane's eight codes of a run: 8 bytes (Q8) or 4 (Q4).
template <int BITS>
struct Codes {
    uint32_t w[BITS / 4];
    __device__ inline void load(const uint8_t *p) {
        if constexpr (BITS == 8) {
            const uint2 v = __ldg(reinterpret_cast<const uint2 *>(p));
            w[0] = v.x, w[1] = v.y;
        } else {
            w[0] = __ldg(reinterpret_cast<const uint32_t *>(p));
        }
    }
    __device__ inline uint4 bf16(float zero = kCodeBias) const { return codes_bf16<BITS>(w[0], w[BITS / 4 - 1], zero); }
};

// Eights of tokens a CTA takes, 1, 2 or 4; the weights of a second group of tokens come from L2.  Two for 9 to 16 tokens, and below 64 where the last
// 32 would be at most half full (the hyper-connection mix of 40 tokens, d = 4096 Q8: 32 us, 39 with four; of 63 tokens: 45 and 41); from 64
// tokens on a group that is not full weighs little.
inline int token_eights(int64_t T) { return T <= 8 ? 1 : T <= 16 || (T < 64 && (T - 1) % 32 < 16) ? 2 : 4; }

// ---- the CTAs of a cluster -------------------------------------------------------------------------------------------
__device__ inline uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ inline void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
// A float of another CTA's shared memory, at the place that `p` has in this CTA's.
__device__ inline float ld_cluster(const float *p, uint32_t rank) {
    uint32_t a = (uint32_t)__cvta_generic_to_shared(p), r;
    float v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(r) : "memory");
    return v;
}

}  // namespace sxb
