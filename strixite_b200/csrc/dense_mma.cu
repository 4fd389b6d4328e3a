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
// 32 tokens, and the activations' way through L1, once per 16 rows; for many rows of x see dense_rows_kernel.  The form before it (stream_mma.cu,
// which keeps Q4) staged a tile of 8 tokens as scaled F16 in every CTA and converted every code again for the next 8.  As CUDA graphs on weights that lie in L2,
// us before -> now: 2048 x 4096, 1 / 16 / 40 / 300 tokens 9.6 -> 6.4, 12.2 -> 7.7, 21.8 -> 15.1, 70 -> 55; 4096 x 1024 7.4 -> 4.1, 8.2 -> 4.7, 13.6 -> 8.4,
// 35.4 -> 36.0; 8192 x 4096, 8 / 63 / 300 tokens 16.4 -> 12.6, 56.8 -> 44.5, 205 -> 202; weights from HBM, 8 tokens 24.6 -> 20.5, 63 67.6 -> 55.3.
// Error against 64 bits (2-norms) 1.15e-7 .. 2.3e-7 -> 0.95e-7 .. 1.2e-7.  Q4, whose nibbles take more instructions to BF16 than to F16,
// was slower this way (8192 x 4096, 8 tokens: 13 -> 17) and stays there.

#include "experts.cuh"
#include "skinny_mma.cuh"

#include <algorithm>
#include <type_traits>

namespace sxb {
namespace {

constexpr int kDenseWarps = 8;
// Sums in shared memory lie [token][weight row], rows of four more: a fragment's lanes (tokens 2 c, rows g) meet every bank once, with one more
// four lanes met in one (dense_rows_kernel, 4096 x 4096 x 1024: 332 us, now 261).
constexpr int kPad = 4;

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

// The results of a CTA's tile - sums [tokens][rows] of tokens t0 .., weight rows n0 .. - that are not finite, formed again by all of its WARPS
// and stored: each token's activations are looked at once (a NaN among them: every result is NaN, as it is), then the warps share the
// weight rows.
// One thread walking the contraction for each such result, as it stood here before: 8 x 8192 x 4096 with a NaN or an infinity in one token 922 us,
// now 20 and 34; NaN in all tokens 3270, now 22; 128 rows with an infinity each 23500, now 1790; 16 and 88 us without.
template <int TOKENS, int ROWS, int WARPS, typename TOUT>
__device__ __noinline__ void form_again(const float (&sums)[TOKENS][ROWS + kPad], const uint16_t *x, const uint8_t *q, const uint16_t *scale,
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

// sum(x) over a run, of the lane's tokens 2 c and 2 c + 1.
__device__ inline uint64_t run_sums(const uint4 &x) {
    const uint4 ones = make_uint4(0x3f803f80u, 0x3f803f80u, 0x3f803f80u, 0x3f803f80u);
    float sx[4] = {0.f, 0.f, 0.f, 0.f};
    mma_run(sx, ones, ones, x);
    return pair(sx[0], sx[1]);
}
// acc += a run's share of the dots with P eights of tokens: a, s, mn = codes, scales and mins of the lane's rows, x = its tokens' activations, sx =
// the sums of its tokens 2 c and 2 c + 1.  An MMA's result is some 35 cycles away: the runs' second halves come after all of the first ones.
template <int P, int MT>
__device__ inline void add_runs(uint64_t (*acc)[MT][2], const uint4 (&a)[2 * MT], const float (&s)[2 * MT], const float (&mn)[2 * MT], const uint4 *x, const uint64_t *sx) {
    float dot[P][MT][4];
#pragma unroll
    for (int p = 0; p < P; ++p)
#pragma unroll
        for (int m = 0; m < MT; ++m) {
            dot[p][m][0] = dot[p][m][1] = dot[p][m][2] = dot[p][m][3] = 0.f;
            mma_bf16(dot[p][m], a[2 * m].x, a[2 * m + 1].x, a[2 * m].y, a[2 * m + 1].y, x[p].x, x[p].y);
        }
#pragma unroll
    for (int p = 0; p < P; ++p)
#pragma unroll
        for (int m = 0; m < MT; ++m) mma_bf16(dot[p][m], a[2 * m].z, a[2 * m + 1].z, a[2 * m].w, a[2 * m + 1].w, x[p].z, x[p].w);
#pragma unroll
    for (int p = 0; p < P; ++p)
#pragma unroll
        for (int m = 0; m < MT; ++m)
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int r = 2 * m + i;
                // the two terms meet before the sum does: they cancel by and large, and what they round is theirs alone
                acc[p][m][i] = add_pair(acc[p][m][i], fma_pair(pair(s[r], s[r]), pair(dot[p][m][2 * i], dot[p][m][2 * i + 1]), mul_pair(pair(mn[r], mn[r]), sx[p])));
            }
}

template <int MT, int NT, typename TOUT>
__global__ void __launch_bounds__(32 * kDenseWarps, 2)
    dense_mma_kernel(const uint16_t *__restrict__ x, const uint8_t *__restrict__ q, const uint16_t *__restrict__ scale,
                     const uint16_t *__restrict__ minv, int64_t M, int64_t N, int64_t K, int64_t G, TOUT *__restrict__ y) {
    behind_grid();
    constexpr int kTok = kMmaTokens * NT, kRowsCta = kMmaRows * MT;
    constexpr int kAhead = MT == 2 || NT == 4 ? 4 : 8;           // runs whose codes a lane has in flight
    constexpr int kActs = NT == 4 ? 1 : (NT == 2 ? 2 : 4) / MT;  // ... whose activations
    __shared__ float part[kDenseWarps][kTok][kRowsCta + kPad];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, c = lane & 3;
    const int64_t n0 = (int64_t)blockIdx.x * kRowsCta, groups = K / G;
    const int runs = (int)(K / kMmaRun), lo = runs * warp / kDenseWarps, hi = runs * (warp + 1) / kDenseWarps, per_group = (int)(G / kMmaRun);
    int64_t row[2 * MT];  // rows past the end stream the last one; their sums are dropped
#pragma unroll
    for (int i = 0; i < 2 * MT; ++i) row[i] = min(n0 + 8 * i + g, N - 1);
    const int64_t t0 = (int64_t)blockIdx.y * kTok;
    uint64_t acc[NT][MT][2];  // rows g + 16 m (+ 8), tokens 2 c and 2 c + 1 of each eight
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) acc[nt][m][0] = acc[nt][m][1] = 0;
    for (int r0 = lo; r0 < hi; r0 += kAhead) {
        Codes<8> w[2 * MT][kAhead];
        uint32_t sm[2 * MT][kAhead / 4];  // (scale, min) for run r0 + 4 i + c: handed round by shuffles
#pragma unroll
        for (int e = 0; e < kAhead; ++e) {
            const int64_t r = min(r0 + e, hi - 1);
#pragma unroll
            for (int i = 0; i < 2 * MT; ++i) w[i][e].load(q + row[i] * K + r * kMmaRun + 8 * c);
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
#pragma unroll
                for (int nt = 0; nt < NT; ++nt) {
                    const uint64_t sx = run_sums(xv[e][nt]);
                    add_runs<1, MT>(&acc[nt], a, s, mn, &xv[e][nt], &sx);
                }
            }
        }
    }
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int t = nt * kMmaTokens + 2 * c, r = m * kMmaRows + g + 8 * i;
                unpair(acc[nt][m][i], part[warp][t][r], part[warp][t + 1][r]);
            }
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

// ---- many rows of x: the same sums, bit for bit ------------------------------------------------------------------------
// A CTA takes 256 weight rows x 32 tokens, a warp 32 of the rows over the whole contraction, one of its eight parts after another.  The
// activations of 1024 k at a time lie in shared memory in fragment order with the sums of their runs, formed once for all rows; a warp's codes
// come straight from memory, four runs ahead, and nothing is waited for in between.
//
// What bounds it: the L1 pipe, at 79 % (codes 32 of a run's 90 wavefronts - eight rows, eight lines a load -, activations 16, scales), and the
// latencies between MMAs and sums with four warps a scheduler (issue slots 54 %, tensor pipe 30).  dense_mma_kernel reads the activations again for every 16
// rows and converts a code for 32 tokens as this does.  us, that -> this: 1024 x 8192 x 4096 648 -> 443, 4096 rows 2580 -> 1726, 4096 x 2048 x 4096
// 650 -> 443, 4096 x 4096 x 1024 447 -> 261; the form before these (stream_mma.cu) takes 593, 2390, 621 and 291.  Activations copied 64 k at
// a time by cp.async with a barrier a block: 1024 x 8192 x 4096 583.
constexpr int kRowsMT = 2, kRowsNT = 4;  // of a warp
constexpr int kRowsTile = kDenseWarps * kMmaRows * kRowsMT, kRowsTok = kMmaTokens * kRowsNT, kRowsChunk = 32;  // weight rows, tokens; runs in shared memory
constexpr size_t kRowsSmem = (size_t)kRowsChunk * kRowsTok * (kMmaRun * 2 + sizeof(float)) + (size_t)kRowsTok * (kRowsTile + kPad) * sizeof(float);

template <typename TOUT>
__global__ void __launch_bounds__(32 * kDenseWarps, 2)
    dense_rows_kernel(const uint16_t *__restrict__ x, const uint8_t *__restrict__ q, const uint16_t *__restrict__ scale,
                      const uint16_t *__restrict__ minv, int64_t M, int64_t N, int64_t K, int64_t G, TOUT *__restrict__ y) {
    constexpr int MT = kRowsMT, NT = kRowsNT, kAhead = 4, kP = 2;
    extern __shared__ __align__(16) unsigned char rows_smem[];
    uint4 *acts = reinterpret_cast<uint4 *>(rows_smem);                           // [run][nt][lane]
    uint64_t *sums = reinterpret_cast<uint64_t *>(acts + kRowsChunk * NT * 32);   // [run][nt][c]: of tokens 2 c and 2 c + 1
    using Total = float[kRowsTok][kRowsTile + kPad];
    Total &total = *reinterpret_cast<Total *>(sums + kRowsChunk * NT * 4);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, c = lane & 3, wr = kMmaRows * MT * warp;
    const int64_t n0 = (int64_t)blockIdx.x * kRowsTile, t0 = (int64_t)blockIdx.y * kRowsTok, groups = K / G;
    const int runs = (int)(K / kMmaRun), per_group = (int)(G / kMmaRun);
    const uint8_t *const tq = q + n0 * K + 8 * c;
    const uint16_t *const ts = scale + n0 * groups, *const tm = minv + n0 * groups;
    uint32_t q_at[2 * MT], s_at[2 * MT];  // rows past the end stream the last one; their sums are dropped
#pragma unroll
    for (int i = 0; i < 2 * MT; ++i) {
        const uint32_t row = (uint32_t)min((int64_t)(wr + 8 * i + g), N - 1 - n0);
        q_at[i] = row * (uint32_t)K, s_at[i] = row * (uint32_t)groups;
    }
    Codes<8> w[2 * MT][kAhead];
    uint16_t ns[2 * MT], nm[2 * MT];  // scale and min of every fourth group, of the next four: handed round by shuffles
    auto fetch = [&](int e, int r) {
#pragma unroll
        for (int i = 0; i < 2 * MT; ++i) w[i][e].load(tq + (q_at[i] + (uint32_t)(min(r, runs - 1) * kMmaRun)));
    };
    auto fetch_scales = [&](int g0) {
        const uint32_t gi = min(g0 + c, (int)groups - 1);
#pragma unroll
        for (int i = 0; i < 2 * MT; ++i) ns[i] = __ldg(ts + (s_at[i] + gi)), nm[i] = __ldg(tm + (s_at[i] + gi));
    };
#pragma unroll
    for (int e = 0; e < kAhead; ++e) fetch(e, e);
    fetch_scales(0);
    uint32_t sm[2 * MT];
    const int lg_group = per_group == 1 ? 0 : per_group == 2 ? 1 : 2;
    uint64_t acc[NT][MT][2];
    auto clear = [&]() {
#pragma unroll
        for (int m = 0; m < MT; ++m)
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) acc[nt][m][0] = acc[nt][m][1] = 0;
    };
    clear();
    int part = 0, part_end = runs / kDenseWarps;
    auto close_parts = [&](int r) {  // the parts that end before run r
        while (part < kDenseWarps && r == part_end) {
#pragma unroll
            for (int m = 0; m < MT; ++m) {  // all of a half's sums are read before any is written: one after another they cost 32 round trips
                float before[NT][2][2];
                auto at = [&](int nt, int i) { return &total[nt * kMmaTokens + 2 * c][wr + m * kMmaRows + g + 8 * i]; };
#pragma unroll
                for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        if (part > 0) before[nt][i][0] = at(nt, i)[0], before[nt][i][1] = at(nt, i)[kRowsTile + kPad];
                        else before[nt][i][0] = before[nt][i][1] = 0.f;
                    }
#pragma unroll
                for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        float p0, p1;
                        unpair(acc[nt][m][i], p0, p1);
                        at(nt, i)[0] = before[nt][i][0] + p0, at(nt, i)[kRowsTile + kPad] = before[nt][i][1] + p1;
                    }
            }
            clear();
            ++part, part_end = runs * (part + 1) / kDenseWarps;
        }
    };
    close_parts(0);
    for (int c0 = 0; c0 < runs; c0 += kRowsChunk) {
        const int here = min(kRowsChunk, runs - c0);
        __syncthreads();  // the chunk before has been read
        // a warp has four tokens, whose 16-byte pieces it loads two tokens at a time, all in flight at once
        const uint16_t *xc = x + (int64_t)c0 * kMmaRun;
#pragma unroll
        for (int j0 = 0; j0 < kRowsTok / kDenseWarps; j0 += 2) {
            constexpr int kPieces = kRowsChunk * 4 / 32;
            uint4 v[2][kPieces];
#pragma unroll
            for (int j = 0; j < 2; ++j)
#pragma unroll
                for (int m = 0; m < kPieces; ++m) {
                    const int64_t t = t0 + warp * (kRowsTok / kDenseWarps) + j0 + j;
                    v[j][m] = t < M && lane + 32 * m < here * 4 ? __ldg(reinterpret_cast<const uint4 *>(xc + t * K) + lane + 32 * m) : make_uint4(0u, 0u, 0u, 0u);
                }
#pragma unroll
            for (int j = 0; j < 2; ++j)
#pragma unroll
                for (int m = 0; m < kPieces; ++m) {
                    const int t = warp * (kRowsTok / kDenseWarps) + j0 + j, e = lane + 32 * m;
                    acts[(((e >> 2) * NT + (t >> 3)) << 5) + ((t & 7) << 2) + (e & 3)] = v[j][m];
                }
        }
        __syncthreads();
        for (int i = warp; i < here * NT; i += kDenseWarps) {
            const uint64_t sx = run_sums(acts[i * 32 + lane]);
            if (g == 0) sums[i * 4 + c] = sx;
        }
        __syncthreads();
        for (int r0 = c0; r0 < c0 + here; r0 += kAhead) {
            if ((r0 >> lg_group) % 4 == 0 && (r0 & (per_group - 1)) == 0) {
#pragma unroll
                for (int i = 0; i < 2 * MT; ++i) sm[i] = ns[i] | (uint32_t)nm[i] << 16;
                fetch_scales((r0 >> lg_group) + 4);
            }
#pragma unroll
            for (int e = 0; e < kAhead; ++e) {
                const int r = r0 + e;
                if (r >= runs) break;
                uint4 a[2 * MT];
                float s[2 * MT], mn[2 * MT];
#pragma unroll
                for (int i = 0; i < 2 * MT; ++i) {
                    const uint32_t p = __shfl_sync(0xffffffffu, sm[i], (lane & ~3) + ((r >> lg_group) & 3));
                    s[i] = __uint_as_float(p << 16), mn[i] = __uint_as_float(p & 0xffff0000u);
                    a[i] = w[i][e].bf16();
                }
                fetch(e, r + kAhead);
#pragma unroll
                for (int nt = 0; nt < NT; nt += kP) {
                    uint4 xv[kP];
                    uint64_t sx[kP];
#pragma unroll
                    for (int p = 0; p < kP; ++p) {
                        const int at = (r - c0) * NT + nt + p;
                        xv[p] = acts[at * 32 + lane], sx[p] = sums[at * 4 + c];
                    }
                    add_runs<kP, MT>(&acc[nt], a, s, mn, xv, sx);
                }
                close_parts(r + 1);
            }
        }
    }
    __syncthreads();
    bool bad = false;
    static_assert(kRowsTile == 32 * kDenseWarps, "a thread has a weight row");
    const int64_t n = n0 + threadIdx.x;
#pragma unroll 8
    for (int tt = 0; tt < kRowsTok; ++tt)
        if (t0 + tt < M && n < N) {
            const float sum = total[tt][threadIdx.x];
            store_from_f32(y, (t0 + tt) * N + n, sum);
            bad |= !isfinite(sum);
        }
    if (__syncthreads_or(bad)) form_again<kRowsTok, kRowsTile, kDenseWarps>(total, x, q, scale, minv, t0, n0, M, N, K, G, y);
}

}  // namespace

// x [M, K] BF16, y [M, N] BF16 or FP32; arguments checked by the caller.
int dense_q8(const char *fn, const void *x, const SxbQView *w, void *y, int64_t M, int out_act, cudaStream_t st) {
    auto xb = static_cast<const uint16_t *>(x);
    // Two CTAs of dense_rows_kernel an SM: it is taken where its waves are at least three quarters full and the other form would take tokens by 32
    // too.  As measured, us (dense_mma_kernel / this one): 80 CTAs 55 / 84 (300 x 2048 x 4096), 160 37 / 50 (300 x 4096 x 1024), 256 166 / 130
    // (1024 x 2048 x 4096), 320 205 / 214, 512 114 / 78 (1024 x 4096 x 1024).
    const dim3 rows_grid((unsigned)((w->N + kRowsTile - 1) / kRowsTile), (unsigned)((M + kRowsTok - 1) / kRowsTok));
    const int64_t rows_ctas = (int64_t)rows_grid.x * rows_grid.y, at_once = 2 * (int64_t)sm_count();
    if (M >= 64 && rows_ctas * 4 >= (rows_ctas + at_once - 1) / at_once * at_once * 3) {
        auto go_rows = [&](auto *yt) -> int {
            auto kern = dense_rows_kernel<std::remove_pointer_t<decltype(yt)>>;
            SXB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kRowsSmem), fn, ": reserving shared memory");
            kern<<<rows_grid, 32 * kDenseWarps, kRowsSmem, st>>>(xb, w->q, w->scale, w->minv, M, w->N, w->K, w->G, yt);
            SXB_CHECK_LAUNCH(fn, " BF16->", act_name(out_act), " M=", M, " N=", w->N, " K=", w->K, " G=", w->G);
            return SXB_OK;
        };
        return out_act == SXB_ACT_F32 ? go_rows(static_cast<float *>(y)) : go_rows(static_cast<uint16_t *>(y));
    }
    const int NT = token_eights(M);
    const int64_t token_groups = (M + NT * kMmaTokens - 1) / (NT * kMmaTokens);
    // 32 rows a CTA where that leaves every SM one: half the reading of activations, and as many CTAs as are resident at once
    // (8 x 8192 x 4096: 14.1 us, 16.7 with 16); with 32 tokens the registers are better spent on those
    const int MT = NT < 4 && (w->N + 31) / 32 * token_groups >= sm_count() ? 2 : 1;
    const dim3 grid((unsigned)((w->N + kMmaRows * MT - 1) / (kMmaRows * MT)), (unsigned)token_groups);  // at most 16384: 524280 rows of x, 32 a CTA
    auto go = [&](auto *yt) {
        using T = std::remove_pointer_t<decltype(yt)>;
#define SXB_DENSE(MTV, NTV) launch_behind(dense_mma_kernel<MTV, NTV, T>, grid, 32 * kDenseWarps, 0, st, 1, xb, w->q, w->scale, w->minv, M, w->N, w->K, w->G, yt)
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

}  // namespace sxb
