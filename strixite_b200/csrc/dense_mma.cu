// Dense projections y = x W^T of Q8 weights with exact products (kernels/linear_q8.hpp linear_q8): the decode side's and small batches'
// quantized linears, the shared expert's among them.
//
// Products of BF16 activations with the integer codes on the warp-level tensor-core path (skinny_mma.cuh), FP32 sums, scale and min applied in
// FP32 per run of 32 codes: a row's dot is sum over its runs of scale * sum(x * code) + min * sum(x), as kernels/linear_q4.hip:175-199 forms
// it.  A CTA of eight warps owns 16 or 32 weight rows and up to 32 tokens; the warps take an eighth of the contraction each, whose codes a
// lane asks for four or eight runs ahead, with the activations in fragment order as they lie in memory; the warps' parts are added in
// order in shared memory.  Which runs a warp takes follows from K alone, so a row's bits depend neither on the batch nor on the tile.
//
// What bounds it: for few tokens a launch, the round trips to memory and the parts' meeting; for more the code conversions, once per
// 32 tokens.  The form before it (stream_mma.cu, which keeps Q4) staged a tile of 8 tokens as scaled F16 in every CTA and converted every
// code again for the next 8.  As CUDA graphs, us before -> now: 2048 x 4096, 1 / 16 / 37 / 150 tokens 9.5 -> 6.7, 12.0 -> 7.9,
// 21.7 -> 16.9, 41.4 -> 34.6; 4096 x 1024 7.3 -> 4.1, 8.2 -> 4.9, 13.5 -> 9.5, 23.9 -> 21.9; 8192 x 4096, 8 / 63 tokens 16.4 -> 13.7, 58.5 -> 48.0.
// Error against 64 bits (2-norms) 1.15e-7 .. 2.3e-7 -> 0.95e-7 .. 1.2e-7.  Q4, whose nibbles take more instructions to BF16 than to F16,
// was slower this way (8192 x 4096, 8 tokens: 13 -> 17) and stays there.

#include "experts.cuh"
#include "skinny_mma.cuh"

#include <algorithm>
#include <type_traits>

namespace sxb {
namespace {

constexpr int kDenseWarps = 8;

// What a token with one or more results that are not finite holds: infinities, NaN, or neither.
constexpr uint32_t kHoldsInf = 1u, kHoldsNan = 2u;
__device__ __noinline__ uint32_t odd_values(const uint16_t *x, int64_t K) {  // by a whole warp
    uint32_t inf = 0, nan = 0;
#pragma unroll 4
    for (int64_t e = threadIdx.x & 31; e < K / 8; e += 32) {
        const uint4 v = __ldg(reinterpret_cast<const uint4 *>(x) + e);
        const uint32_t xs[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const uint32_t lo = xs[i] & 0x7fffu, hi = xs[i] & 0x7fff0000u;
            inf |= (lo == 0x7f80u) | (hi == 0x7f800000u), nan |= (lo > 0x7f80u) | (hi > 0x7f800000u);
        }
    }
    return (__any_sync(0xffffffffu, inf != 0) ? kHoldsInf : 0u) | (__any_sync(0xffffffffu, nan != 0) ? kHoldsNan : 0u);
}

// The dot of one token with one weight row in FP64, by a whole warp: where the sums above left FP32's range - products of codes with
// activations beyond 2^120, or infinities - this says what the result is.  With an infinity among the activations the finite terms do not count.
__device__ __noinline__ float wide_dot(const uint16_t *x, const uint8_t *q, const uint16_t *scale, const uint16_t *minv, int64_t K, int64_t G, bool has_inf) {
    constexpr int kAhead = 4;  // pieces of eight in flight
    const int eights = (int)(K / 8), per_group = (int)(G / 8);
    double sum = 0.0;
    for (int e0 = threadIdx.x & 31; e0 < eights; e0 += 32 * kAhead) {
        uint4 v[kAhead];
        uint16_t sb[kAhead], mb[kAhead];
#pragma unroll
        for (int a = 0; a < kAhead; ++a) {
            const int e = min(e0 + 32 * a, eights - 1);
            v[a] = __ldg(reinterpret_cast<const uint4 *>(x) + e), sb[a] = __ldg(scale + e / per_group), mb[a] = __ldg(minv + e / per_group);
        }
#pragma unroll
        for (int a = 0; a < kAhead; ++a) {
            const int e = e0 + 32 * a;
            const uint32_t xs[4] = {v[a].x, v[a].y, v[a].z, v[a].w};
            const float s = bf16_bits_to_f32(sb[a]), m = bf16_bits_to_f32(mb[a]);
            bool odd = !isfinite(s) || !isfinite(m);
#pragma unroll
            for (int i = 0; i < 4; ++i) odd |= (xs[i] & 0x7f80u) == 0x7f80u || (xs[i] & 0x7f800000u) == 0x7f800000u;
            if (e >= eights || (has_inf && !odd)) continue;
            const uint2 w = __ldg(reinterpret_cast<const uint2 *>(q) + e);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const double code = (double)(((i < 4 ? w.x : w.y) >> (8 * (i & 3))) & 255u);
                sum += (code * s + m) * (double)__uint_as_float((i & 1) ? (xs[i / 2] & 0xffff0000u) : (xs[i / 2] << 16));
            }
        }
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
    return (float)sum;
}

// The results of a CTA's tile - sums [tokens][rows + 1] of tokens t0 .., weight rows n0 .. - that are not finite, formed again by all of its WARPS
// and stored: each token's activations are looked at once (a NaN among them: every result is NaN, as it is), then the warps share the
// weight rows.
// One thread walking the contraction for each such result, as it stood here before: 8 x 8192 x 4096 with a NaN or an infinity in one token 922 us,
// now 20 and 34; NaN in all tokens 3270, now 22; 128 rows with an infinity each 23500, now 1790; 16 and 88 us without.
template <int TOKENS, int ROWS, int WARPS, typename TOUT>
__device__ __noinline__ void form_again(const float (&sums)[TOKENS][ROWS + 1], const uint16_t *x, const uint8_t *q, const uint16_t *scale,
                                        const uint16_t *minv, int64_t t0, int64_t n0, int64_t M, int64_t N, int64_t K, int64_t G, TOUT *y) {
    __shared__ uint32_t holds[TOKENS];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int tt = warp; tt < TOKENS && t0 + tt < M; tt += WARPS) {
        bool bad = false;
        for (int r = lane; r < ROWS; r += 32) bad |= !isfinite(sums[tt][r]);
        const uint32_t h = __any_sync(0xffffffffu, bad) ? odd_values(x + (t0 + tt) * K, K) : 0u;
        if (lane == 0) holds[tt] = h;
    }
    __syncthreads();
    for (int r = warp; r < ROWS && n0 + r < N; r += WARPS)
        for (int tt = 0; tt < TOKENS && t0 + tt < M; ++tt) {
            if (isfinite(sums[tt][r]) || (holds[tt] & kHoldsNan)) continue;
            const int64_t n = n0 + r;
            const float wide = wide_dot(x + (t0 + tt) * K, q + n * K, scale + n * (K / G), minv + n * (K / G), K, G, (holds[tt] & kHoldsInf) != 0);
            if (lane == 0) store_from_f32(y, (t0 + tt) * N + n, wide);
        }
}

template <int BITS, int MT, int NT, typename TOUT>
__global__ void __launch_bounds__(32 * kDenseWarps, 2)
    dense_mma_kernel(const uint16_t *__restrict__ x, const uint8_t *__restrict__ q, const uint16_t *__restrict__ scale,
                     const uint16_t *__restrict__ minv, int64_t M, int64_t N, int64_t K, int64_t G, TOUT *__restrict__ y) {
    constexpr int kTok = kMmaTokens * NT, kRowsCta = kMmaRows * MT;
    constexpr int kAhead = MT == 2 || NT == 4 ? 4 : 8;           // runs whose codes a lane has in flight
    constexpr int kActs = NT == 4 ? 1 : (NT == 2 ? 2 : 4) / MT;  // ... whose activations
    constexpr int kRunBytes = kMmaRun * BITS / 8;
    __shared__ float part[kDenseWarps][kTok][kRowsCta + 1];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, c = lane & 3;
    const int64_t n0 = (int64_t)blockIdx.x * kRowsCta, row_bytes = K * BITS / 8, groups = K / G;
    const int runs = (int)(K / kMmaRun), lo = runs * warp / kDenseWarps, hi = runs * (warp + 1) / kDenseWarps, per_group = (int)(G / kMmaRun);
    int64_t row[2 * MT];  // rows past the end stream the last one; their sums are dropped
#pragma unroll
    for (int i = 0; i < 2 * MT; ++i) row[i] = min(n0 + 8 * i + g, N - 1);
    for (int64_t t0 = (int64_t)blockIdx.y * kTok; t0 < M; t0 += (int64_t)gridDim.y * kTok) {
        float acc[MT][NT][4];
#pragma unroll
        for (int m = 0; m < MT; ++m)
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) acc[m][nt][0] = acc[m][nt][1] = acc[m][nt][2] = acc[m][nt][3] = 0.f;
        for (int r0 = lo; r0 < hi; r0 += kAhead) {
            Codes<BITS> w[2 * MT][kAhead];
            uint32_t sm[2 * MT][kAhead / 4];  // (scale, min) for run r0 + 4 i + c: handed round by shuffles
#pragma unroll
            for (int e = 0; e < kAhead; ++e) {
                const int64_t r = min(r0 + e, hi - 1);
#pragma unroll
                for (int i = 0; i < 2 * MT; ++i) w[i][e].load(q + row[i] * row_bytes + r * kRunBytes + c * BITS);
            }
#pragma unroll
            for (int e = 0; e < kAhead / 4; ++e) {
                const int gi = min(r0 + 4 * e + c, hi - 1) / per_group;
#pragma unroll
                for (int i = 0; i < 2 * MT; ++i)
                    sm[i][e] = __ldg(scale + row[i] * groups + gi) | (uint32_t)__ldg(minv + row[i] * groups + gi) << 16;
            }
#pragma unroll
            for (int e0 = 0; e0 < kAhead; e0 += kActs) {
                if (r0 + e0 >= hi) break;
                uint4 xv[kActs][NT];
#pragma unroll
                for (int e = 0; e < kActs; ++e)
#pragma unroll
                    for (int nt = 0; nt < NT; ++nt) {
                        const int64_t t = t0 + nt * kMmaTokens + g;
                        xv[e][nt] = t < M && r0 + e0 + e < hi ? __ldg(reinterpret_cast<const uint4 *>(x + t * K + (int64_t)(r0 + e0 + e) * kMmaRun + 8 * c))
                                                              : make_uint4(0u, 0u, 0u, 0u);
                    }
#pragma unroll
                for (int e = 0; e < kActs; ++e) {
                    const int at = e0 + e;
                    if (r0 + at >= hi) break;
                    uint4 a[2 * MT];
                    float s[2 * MT], mn[2 * MT];
#pragma unroll
                    for (int i = 0; i < 2 * MT; ++i) {
                        const uint32_t p = __shfl_sync(0xffffffffu, sm[i][at / 4], (lane & ~3) + at % 4);
                        s[i] = __uint_as_float(p << 16), mn[i] = __uint_as_float(p & 0xffff0000u);
                        a[i] = w[i][at].bf16();
                    }
                    const uint4 ones = make_uint4(0x3f803f80u, 0x3f803f80u, 0x3f803f80u, 0x3f803f80u);
#pragma unroll
                    for (int nt = 0; nt < NT; ++nt) {
                        float sx[4] = {0.f, 0.f, 0.f, 0.f};
                        mma_run(sx, ones, ones, xv[e][nt]);
#pragma unroll
                        for (int m = 0; m < MT; ++m) {
                            float dot[4] = {0.f, 0.f, 0.f, 0.f};
                            mma_run(dot, a[2 * m], a[2 * m + 1], xv[e][nt]);
                            float(&o)[4] = acc[m][nt];
                            // the two terms meet before the sum does: they cancel by and large, and what they round is theirs alone
                            o[0] += fmaf(s[2 * m], dot[0], mn[2 * m] * sx[0]), o[1] += fmaf(s[2 * m], dot[1], mn[2 * m] * sx[1]);
                            o[2] += fmaf(s[2 * m + 1], dot[2], mn[2 * m + 1] * sx[0]), o[3] += fmaf(s[2 * m + 1], dot[3], mn[2 * m + 1] * sx[1]);
                        }
                    }
                }
            }
        }
        __syncthreads();  // the previous group's parts have been read
#pragma unroll
        for (int m = 0; m < MT; ++m)
#pragma unroll
            for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                for (int i = 0; i < 4; ++i) part[warp][nt * kMmaTokens + 2 * c + (i & 1)][m * kMmaRows + g + 8 * (i >> 1)] = acc[m][nt][i];
        __syncthreads();
        bool bad = false;
        for (int i = threadIdx.x; i < kTok * kRowsCta; i += 32 * kDenseWarps) {
            const int tt = i / kRowsCta, r = i % kRowsCta;
            const int64_t t = t0 + tt, n = n0 + r;
            if (t >= M || n >= N) continue;
            float sum = part[0][tt][r];
#pragma unroll
            for (int v = 1; v < kDenseWarps; ++v) sum += part[v][tt][r];
            store_from_f32(y, t * N + n, sum);
            part[0][tt][r] = sum, bad |= !isfinite(sum);
        }
        if (__syncthreads_or(bad)) form_again<kTok, kRowsCta, kDenseWarps>(part[0], x, q, scale, minv, t0, n0, M, N, K, G, y);
    }
}

}  // namespace

// x [M, K] BF16, y [M, N] BF16 or FP32; arguments checked by the caller.
template <int BITS>
int dense_mma(const char *fn, const void *x, const SxbQView *w, void *y, int64_t M, int out_act, cudaStream_t st) {
    const int NT = token_eights(M);
    const int64_t token_groups = (M + NT * kMmaTokens - 1) / (NT * kMmaTokens);
    // 32 rows a CTA where that leaves every SM one: half the reading of activations, and as many CTAs as are resident at once
    // (8 x 8192 x 4096: 14.1 us, 16.7 with 16); with 32 tokens the registers are better spent on those
    const int MT = NT < 4 && (w->N + 31) / 32 * token_groups >= sm_count() ? 2 : 1;
    const dim3 grid((unsigned)((w->N + kMmaRows * MT - 1) / (kMmaRows * MT)), (unsigned)std::min<int64_t>(token_groups, 65535));
    auto xb = static_cast<const uint16_t *>(x);
    auto go = [&](auto *yt) {
        using T = std::remove_pointer_t<decltype(yt)>;
#define SXB_DENSE(MTV, NTV) dense_mma_kernel<BITS, MTV, NTV, T><<<grid, 32 * kDenseWarps, 0, st>>>(xb, w->q, w->scale, w->minv, M, w->N, w->K, w->G, yt)
        if (NT == 4) SXB_DENSE(1, 4);
        else if (NT == 2 && MT == 1) SXB_DENSE(1, 2);
        else if (NT == 2) SXB_DENSE(2, 2);
        else if (MT == 1) SXB_DENSE(1, 1);
        else SXB_DENSE(2, 1);
#undef SXB_DENSE
    };
    if (out_act == SXB_ACT_F32) go(static_cast<float *>(y));
    else go(static_cast<uint16_t *>(y));
    SXB_CHECK_LAUNCH(fn, " BF16->", act_name(out_act), " M=", M, " N=", w->N, " K=", w->K, " G=", w->G);
    return SXB_OK;
}

template int dense_mma<8>(const char *, const void *, const SxbQView *, void *, int64_t, int, cudaStream_t);

}  // namespace sxb
