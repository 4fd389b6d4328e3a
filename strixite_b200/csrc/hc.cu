// The hyper-connection mix that produces the MoE block's input (kernels/hc.hpp:36-50, call site
// runtime/qwen4exp.cpp:2801-2831, 3144): from the H = 4 residual streams X [T, H*d]
//   hc_mix_down   h [T, r] = silu(a / H) and w_in [T, H] = 2 sigmoid(a / H), a = sum_s inv_s * (W'_s . X_s) over the rows of
//                 the folded, quantized down weight W' [r (+ H), H*d]; inv [T, H] = 1 / sqrt(mean(X_s^2) + eps)
//   hc_mix_up     u [T, d] = (1/H) sum_s sigmoid(W_up[s*d + j] . h) * X_s[j] * inv_s * (1 + norm_w[s*d + j]), W_up chunk-major
// Everything inside is FP32 (kernels/hc.hpp:8-11); u is rounded once to the activation dtype.  A quantized row's dot with
// a 32-code chunk is scale * sum(x * code) + min * sum(x) (kernels/hc.hip:117-123, 206-211): the weights are never
// rounded to a dequantized value.
//
// Both are small-matrix, many-launch kernels (a few MB of weights, ~97 mixes per decoded token upstream): what bounds them is the round
// trips of one launch, as long as the arithmetic stays out of the way.  As FP32 multiply-adds, one a code and token behind a conversion
// of every code, it did not; on the tensor cores (skinny_mma.cuh: exact products of integer codes with BF16 activations, or with the three
// BF16 planes of FP32 ones, FP32 sums) the same numbers are a few hundred MMAs a warp.  Both halves as a CUDA graph, d = 4096, Q8, us before ->
// now: r = 320, one token 16.9 -> 12.6, 16 tokens 42.2 -> 15.7, 64 158 -> 40, 300 525 -> 136; r = 32, 16 tokens 17.9 -> 10.7; r = 1024, 99.5 -> 31.9.
// Against 64 bits, FP32 streams of 16 tokens, h 4.0e-7 -> 1.4e-7 and u 5.7e-7 -> 0.9e-7 (2-norms).  ncu, 16 tokens from HBM: issue slots 25 and
// 32 %, tensor pipe 9 and 13 %, DRAM 6 and 7 %; the warps wait for loads (long scoreboard) and, in the down half, for the cluster.
//   down: 16 weight rows by a cluster of eight CTAs, an eighth of the row each (an eighth lies in one stream), which a CTA's eight warps share;
//         a lane's codes are all asked for at once, its activations come from L2 in fragment order as they lie; the parts meet in shared
//         memory, then across the cluster.
//   up:   a CTA owns 16 output columns, a warp their rows in one stream; h goes to shared memory once, as planes in fragment order; the
//         H streams of a column meet in shared memory.

#include "experts.cuh"
#include "skinny_mma.cuh"

#include <algorithm>
#include <cmath>

namespace sxb {
namespace {

constexpr int kStreams = 4;
constexpr int kChunk = 32;  // codes per chunk: 16 bytes of Q4, 32 of Q8
constexpr int64_t kMaxRank = 1024;
static_assert(kChunk == kMmaRun, "a chunk is a run of the MMA's k");

__device__ inline float sigmoid_f32(float z) { return 1.0f / (1.0f + expf(-z)); }

// A lane's eight activations of a chunk of its token, as the BF16 planes they consist of.
template <typename T>
struct Acts;
template <>
struct Acts<uint16_t> {
    static constexpr int kPlanes = 1;
    uint4 v;
    __device__ inline void load(const uint16_t *p) { v = __ldg(reinterpret_cast<const uint4 *>(p)); }
    __device__ inline void clear() { v = make_uint4(0u, 0u, 0u, 0u); }
    __device__ inline void planes(uint4 (&pl)[1]) const { pl[0] = v; }
    __device__ inline float sum_sq(float s) const {
        const uint32_t w4[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float lo = __uint_as_float(w4[i] << 16), hi = __uint_as_float(w4[i] & 0xffff0000u);
            s = fmaf(lo, lo, s), s = fmaf(hi, hi, s);
        }
        return s;
    }
};
template <>
struct Acts<float> {
    static constexpr int kPlanes = 3;
    float4 a, b;
    __device__ inline void load(const float *p) { a = __ldg(reinterpret_cast<const float4 *>(p)), b = __ldg(reinterpret_cast<const float4 *>(p) + 1); }
    __device__ inline void clear() { a = b = make_float4(0.f, 0.f, 0.f, 0.f); }
    __device__ inline void planes(uint4 (&pl)[3]) const {
        const float f[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
        split_planes(f, pl);
    }
    __device__ inline float sum_sq(float s) const {
        const float f[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
        for (int i = 0; i < 8; ++i) s = fmaf(f[i], f[i], s);
        return s;
    }
};

// hc_mix_down.  grid = (8 x row tiles, token groups of 8 NT), clusters of eight CTAs along x.
// A chunk's share of a dot is scale * sum(x * code) + min * sum(x), as the header of this file says; sum(x) comes from an MMA of its own with
// a matrix of ones for weights, which leaves it in the lanes that need it.  sum(x^2), the same for every weight row, costs a few
// instructions a chunk and is formed by every cluster for itself.
constexpr int kDownWarps = 8, kParts = 8;
constexpr int kCodesAhead = 8;  // chunks whose codes a lane has in flight: d = 4096 gives a warp eight
template <typename T, int NT> constexpr int kActsAhead = sizeof(T) == 2 ? (NT == 4 ? 1 : 4) : (NT == 1 ? 4 : 1);  // ... whose activations

template <typename T, int BITS, int NT>
__global__ void __launch_bounds__(32 * kDownWarps, 2) hc_down_kernel(const T *__restrict__ x, const uint8_t *__restrict__ q,
                                                                     const uint16_t *__restrict__ scale, const uint16_t *__restrict__ minv,
                                                                     int64_t R, int64_t K, int64_t G, int64_t d, int r, float eps, int64_t Tn,
                                                                     float *__restrict__ h, float *__restrict__ w_in, float *__restrict__ inv) {
    constexpr int kTok = kMmaTokens * NT, kAhead = kActsAhead<T, NT>;
    __shared__ float part[kDownWarps][kTok][kMmaRows + 1];  // + 1: the finishing threads of a token read different banks
    __shared__ float part_sq[kDownWarps][kTok];
    __shared__ float cta_part[kTok][kMmaRows], cta_sq[kTok];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, c = lane & 3;
    const int rank = (int)cluster_rank();
    const int64_t n0 = (int64_t)(blockIdx.x / kParts) * kMmaRows, t0 = (int64_t)blockIdx.y * kTok;
    // rows past the end stream the last one; their sums are dropped
    const int64_t row_bytes = K * BITS / 8, groups = K / G, ra = min(n0 + g, R - 1), rb = min(n0 + g + 8, R - 1);
    const int per_part = (int)(K / kChunk) / kParts, lo = rank * per_part + per_part * warp / kDownWarps,
              hi = rank * per_part + per_part * (warp + 1) / kDownWarps;
    const uint8_t *qa = q + ra * row_bytes + c * BITS, *qb = q + rb * row_bytes + c * BITS;
    float acc[NT][4], sq[NT];
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) acc[nt][0] = acc[nt][1] = acc[nt][2] = acc[nt][3] = sq[nt] = 0.f;
    for (int c0 = lo; c0 < hi; c0 += kCodesAhead) {
        Codes<BITS> wa[kCodesAhead], wb[kCodesAhead];
        uint32_t sz_a[kCodesAhead / 4], sz_b[kCodesAhead / 4];  // scales, zero codes and mins of rows a and b for chunks c0 + 4 i + c:
        float mn_a[kCodesAhead / 4], mn_b[kCodesAhead / 4];     // handed round by shuffles
#pragma unroll
        for (int e = 0; e < kCodesAhead; ++e) {
            const int ch = min(c0 + e, hi - 1);
            wa[e].load(qa + (int64_t)ch * (kChunk * BITS / 8)), wb[e].load(qb + (int64_t)ch * (kChunk * BITS / 8));
        }
#pragma unroll
        for (int i = 0; i < kCodesAhead / 4; ++i) {
            const int64_t gi = (int64_t)min(c0 + 4 * i + c, hi - 1) * kChunk / G;
            pack_group<BITS>(__ldg(scale + ra * groups + gi), __ldg(minv + ra * groups + gi), sz_a[i], mn_a[i]);
            pack_group<BITS>(__ldg(scale + rb * groups + gi), __ldg(minv + rb * groups + gi), sz_b[i], mn_b[i]);
        }
#pragma unroll
        for (int e0 = 0; e0 < kCodesAhead; e0 += kAhead) {
            if (c0 + e0 >= hi) break;
            Acts<T> xv[kAhead][NT];
#pragma unroll
            for (int e = 0; e < kAhead; ++e)
#pragma unroll
                for (int nt = 0; nt < NT; ++nt) {
                    const int64_t t = t0 + nt * kMmaTokens + g;
                    if (t < Tn && c0 + e0 + e < hi) xv[e][nt].load(x + t * K + (int64_t)(c0 + e0 + e) * kChunk + 8 * c);
                    else xv[e][nt].clear();
                }
#pragma unroll
            for (int e = 0; e < kAhead; ++e) {
                const int i = e0 + e;
                if (c0 + i >= hi) break;
                const int from = (lane & ~3) + i % 4;
                const uint32_t w_a = __shfl_sync(0xffffffffu, sz_a[i / 4], from), w_b = __shfl_sync(0xffffffffu, sz_b[i / 4], from);
                const float m_a = __shfl_sync(0xffffffffu, mn_a[i / 4], from), m_b = __shfl_sync(0xffffffffu, mn_b[i / 4], from);
                const float s_a = group_scale(w_a), s_b = group_scale(w_b);
                const uint4 va = wa[i].bf16(group_zero(w_a)), vb = wb[i].bf16(group_zero(w_b)), ones = make_uint4(0x3f803f80u, 0x3f803f80u, 0x3f803f80u, 0x3f803f80u);
#pragma unroll
                for (int nt = 0; nt < NT; ++nt) {
                    uint4 pl[Acts<T>::kPlanes];
                    xv[e][nt].planes(pl);
                    float dot[4] = {0.f, 0.f, 0.f, 0.f}, sx[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                    for (int p = Acts<T>::kPlanes - 1; p >= 0; --p) mma_run(dot, va, vb, pl[p]), mma_run(sx, ones, ones, pl[p]);
                    acc[nt][0] = fmaf(s_a, dot[0], fmaf(m_a, sx[0], acc[nt][0])), acc[nt][1] = fmaf(s_a, dot[1], fmaf(m_a, sx[1], acc[nt][1]));
                    acc[nt][2] = fmaf(s_b, dot[2], fmaf(m_b, sx[0], acc[nt][2])), acc[nt][3] = fmaf(s_b, dot[3], fmaf(m_b, sx[1], acc[nt][3]));
                    sq[nt] = xv[e][nt].sum_sq(sq[nt]);
                }
            }
        }
    }
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
        const int t = nt * kMmaTokens + 2 * c;
        part[warp][t][g] = acc[nt][0], part[warp][t + 1][g] = acc[nt][1];
        part[warp][t][g + 8] = acc[nt][2], part[warp][t + 1][g + 8] = acc[nt][3];
        sq[nt] += __shfl_xor_sync(0xffffffffu, sq[nt], 1);
        sq[nt] += __shfl_xor_sync(0xffffffffu, sq[nt], 2);
        if (c == 0) part_sq[warp][nt * kMmaTokens + g] = sq[nt];
    }
    __syncthreads();
    for (int i = threadIdx.x; i < kTok * kMmaRows; i += 32 * kDownWarps) {
        float sum = 0.f;
#pragma unroll
        for (int w = 0; w < kDownWarps; ++w) sum += part[w][i / kMmaRows][i % kMmaRows];
        cta_part[i / kMmaRows][i % kMmaRows] = sum;
    }
    if (threadIdx.x < kTok) {
        float sum = 0.f;
#pragma unroll
        for (int w = 0; w < kDownWarps; ++w) sum += part_sq[w][threadIdx.x];
        cta_sq[threadIdx.x] = sum;
    }
    cluster_sync();
    // A CTA of the cluster finishes every eighth token: its sixteen rows' dots, their streams' inverse RMS, the activation.
    if (threadIdx.x < NT * kMmaRows) {
        const int tt = rank + kParts * (threadIdx.x / kMmaRows), row = threadIdx.x % kMmaRows;
        const int64_t n = n0 + row, t = t0 + tt;
        if (n < R && t < Tn) {
            float dots[kParts], sqs[kParts];
#pragma unroll
            for (int p = 0; p < kParts; ++p) dots[p] = ld_cluster(&cta_part[tt][row], p), sqs[p] = ld_cluster(&cta_sq[tt], p);
            float a = 0.f;
#pragma unroll
            for (int st = 0; st < kStreams; ++st) {
                const float rms = 1.0f / sqrtf((sqs[2 * st] + sqs[2 * st + 1]) / (float)d + eps);
                a = fmaf(rms, dots[2 * st] + dots[2 * st + 1], a);
                if (n == 0) inv[t * kStreams + st] = rms;
            }
            const float z = a / (float)kStreams;
            if (n < r) h[t * r + n] = z * sigmoid_f32(z);
            else w_in[t * kStreams + (n - r)] = 2.0f * sigmoid_f32(z);
        }
    }
    cluster_sync();  // no CTA leaves while another may still read its shared memory
}

// hc_mix_up.  grid = (d / 16, token groups of 8 NT); warp s owns rows s * d + 16 blockIdx.x .. + 15 of W_up, whose chunks lie side by side in
// the chunk-major layout.  h is an FP32 number and stays one: three BF16 planes.
constexpr int kUpCols = kMmaRows;  // output columns per CTA
constexpr int kUpAhead = 12;       // chunks of codes in flight per warp: r = 320 has ten

template <typename T, int BITS, int NT>
__global__ void __launch_bounds__(32 * kStreams) hc_up_kernel(const float *__restrict__ h, const uint8_t *__restrict__ q,
                                                              const uint16_t *__restrict__ scale, const uint16_t *__restrict__ minv, int64_t G,
                                                              const T *__restrict__ x, const float *__restrict__ norm_w,
                                                              const float *__restrict__ inv, int64_t d, int r, int64_t Tn, bool vec_h, T *__restrict__ u) {
    constexpr int kTok = kMmaTokens * NT;
    extern __shared__ __align__(16) unsigned char up_smem[];
    const int chunks = r / kChunk;
    uint4 *planes = reinterpret_cast<uint4 *>(up_smem);                      // [chunk][nt][plane][lane]
    float *hsum = reinterpret_cast<float *>(planes + (size_t)chunks * NT * 3 * 32);  // [chunk][token]
    __shared__ float part[kStreams][kTok][kUpCols + 1];
    const int lane = threadIdx.x & 31, s = threadIdx.x >> 5, g = lane >> 2, c = lane & 3;
    const int64_t N = kStreams * d, j0 = (int64_t)blockIdx.x * kUpCols, row = s * d + j0 + g, t0 = (int64_t)blockIdx.y * kTok;
    // the first chunks' codes are asked for before anything else
    Codes<BITS> wa[kUpAhead], wb[kUpAhead];
    uint16_t sa[kUpAhead / 4], sb[kUpAhead / 4], ma[kUpAhead / 4], mb[kUpAhead / 4];  // of chunk 4 i + c: the four lanes of a row share it
    auto fetch = [&](int slot, int ch) {
        const uint8_t *p = q + ((int64_t)ch * N + row) * (kChunk * BITS / 8) + c * BITS;
        wa[slot].load(p), wb[slot].load(p + 8 * (kChunk * BITS / 8));
    };
    auto fetch_scales = [&](int slot, int ch) {
        const int64_t gi = (int64_t)min(ch + c, chunks - 1) * kChunk / G * N + row;
        sa[slot] = __ldg(scale + gi), ma[slot] = __ldg(minv + gi), sb[slot] = __ldg(scale + gi + 8), mb[slot] = __ldg(minv + gi + 8);
    };
#pragma unroll
    for (int a = 0; a < kUpAhead; ++a)
        if (a < chunks) fetch(a, a);
#pragma unroll
    for (int i = 0; i < kUpAhead / 4; ++i)
        if (4 * i < chunks) fetch_scales(i, 4 * i);
    // what the tokens' terms take beside z: the lane's tokens are 2 c and 2 c + 1 of each eight, its columns g and g + 8
    float xi[NT][4];
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int64_t t = t0 + nt * kMmaTokens + 2 * c + (i & 1);
            xi[nt][i] = t < Tn ? load_as_f32(x, t * N + row + 8 * (i >> 1)) * inv[t * kStreams + s] * (1.0f + norm_w[row + 8 * (i >> 1)]) : 0.f;
        }
    constexpr int kStage = 5;  // runs of h a warp has in flight: one at a time, each iteration was a round trip to L2
    for (int i0 = s; i0 < chunks * NT; i0 += kStage * kStreams) {
        float v[kStage][8];
#pragma unroll
        for (int b = 0; b < kStage; ++b) {
            const int i = i0 + b * kStreams, ch = i / NT;
            const int64_t t = t0 + i % NT * kMmaTokens + g;
            const float *hp = h + t * r + ch * kChunk + 8 * c;
#pragma unroll
            for (int k = 0; k < 8; ++k) v[b][k] = 0.f;
            if (i < chunks * NT && t < Tn) {
                if (vec_h) {
                    const float4 p = reinterpret_cast<const float4 *>(hp)[0], q4 = reinterpret_cast<const float4 *>(hp)[1];
                    v[b][0] = p.x, v[b][1] = p.y, v[b][2] = p.z, v[b][3] = p.w, v[b][4] = q4.x, v[b][5] = q4.y, v[b][6] = q4.z, v[b][7] = q4.w;
                } else {
#pragma unroll
                    for (int k = 0; k < 8; ++k) v[b][k] = hp[k];
                }
            }
        }
#pragma unroll
        for (int b = 0; b < kStage; ++b) {
            const int i = i0 + b * kStreams;
            if (i >= chunks * NT) break;
            uint4 pl[3];
            split_planes(v[b], pl);
#pragma unroll
            for (int p = 0; p < 3; ++p) planes[(i * 3 + p) * 32 + lane] = pl[p];
            float sum = ((v[b][0] + v[b][1]) + (v[b][2] + v[b][3])) + ((v[b][4] + v[b][5]) + (v[b][6] + v[b][7]));
            sum += __shfl_xor_sync(0xffffffffu, sum, 1);
            sum += __shfl_xor_sync(0xffffffffu, sum, 2);
            if (c == 0) hsum[i / NT * kTok + i % NT * kMmaTokens + g] = sum;
        }
    }
    __syncthreads();
    float acc[NT][4];
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) acc[nt][0] = acc[nt][1] = acc[nt][2] = acc[nt][3] = 0.f;
    for (int c0 = 0; c0 < chunks; c0 += kUpAhead) {
        uint32_t sz_a = 0, sz_b = 0;
        float mn_a = 0.f, mn_b = 0.f;
#pragma unroll
        for (int a = 0; a < kUpAhead; ++a) {
            const int ch = c0 + a;
            if (ch >= chunks) break;
            if (a % 4 == 0) {
                pack_group<BITS>(sa[a / 4], ma[a / 4], sz_a, mn_a), pack_group<BITS>(sb[a / 4], mb[a / 4], sz_b, mn_b);
                if (ch + kUpAhead < chunks) fetch_scales(a / 4, ch + kUpAhead);
            }
            const int from = (lane & ~3) + a % 4;
            const uint32_t w_a = __shfl_sync(0xffffffffu, sz_a, from), w_b = __shfl_sync(0xffffffffu, sz_b, from);
            const float m_a = __shfl_sync(0xffffffffu, mn_a, from), m_b = __shfl_sync(0xffffffffu, mn_b, from);
            const float s_a = group_scale(w_a), s_b = group_scale(w_b);
            const uint4 va = wa[a].bf16(group_zero(w_a)), vb = wb[a].bf16(group_zero(w_b));
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) {
                float dot[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                for (int p = 2; p >= 0; --p) mma_run(dot, va, vb, planes[((ch * NT + nt) * 3 + p) * 32 + lane]);
                const float2 hs = *reinterpret_cast<const float2 *>(hsum + ch * kTok + nt * kMmaTokens + 2 * c);
                acc[nt][0] = fmaf(s_a, dot[0], fmaf(m_a, hs.x, acc[nt][0])), acc[nt][1] = fmaf(s_a, dot[1], fmaf(m_a, hs.y, acc[nt][1]));
                acc[nt][2] = fmaf(s_b, dot[2], fmaf(m_b, hs.x, acc[nt][2])), acc[nt][3] = fmaf(s_b, dot[3], fmaf(m_b, hs.y, acc[nt][3]));
            }
            if (ch + kUpAhead < chunks) fetch(a, ch + kUpAhead);  // the slot's codes are spent
        }
    }
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int i = 0; i < 4; ++i) part[s][nt * kMmaTokens + 2 * c + (i & 1)][g + 8 * (i >> 1)] = sigmoid_f32(acc[nt][i]) * xi[nt][i];
    __syncthreads();
    for (int i = threadIdx.x; i < kTok * kUpCols; i += 32 * kStreams) {
        const int tt = i / kUpCols, j = i % kUpCols;
        if (t0 + tt >= Tn) break;
        float sum = 0.f;
#pragma unroll
        for (int k = 0; k < kStreams; ++k) sum += part[k][tt][j];
        store_from_f32(u, (t0 + tt) * d + j0 + j, sum / (float)kStreams);
    }
}

// Row-major Q4 / Q8 -> chunk-major (formats/q4.hpp:41-55): 32-code chunk c of row n at q[(c * N + n) * chunk bytes], group
// g's scale / min at [g * N + n].
__global__ void __launch_bounds__(256) chunk_major_kernel(const uint8_t *__restrict__ q, const uint16_t *__restrict__ scale,
                                                          const uint16_t *__restrict__ minv, int64_t N, int64_t K, int64_t G, int chunk_bytes,
                                                          uint8_t *__restrict__ qo, uint16_t *__restrict__ so, uint16_t *__restrict__ mo) {
    const int64_t chunks = K / kChunk, groups = K / G, words = chunk_bytes / 4;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < N * chunks * words; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t w = i % words, nc = i / words, c = nc % chunks, n = nc / chunks;
        reinterpret_cast<uint32_t *>(qo)[(c * N + n) * words + w] = reinterpret_cast<const uint32_t *>(q)[(n * chunks + c) * words + w];
    }
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < N * groups; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t g = i % groups, n = i / groups;
        so[g * N + n] = scale[i], mo[g * N + n] = minv[i];
    }
}

int check_hc_shape(const char *fn, int64_t T, int64_t H, int64_t d) {
    SXB_CHECK(H == kStreams, fn, ": H = ", H, " streams, only ", kStreams, " is supported");
    SXB_CHECK(T >= 1 && T <= 65535, fn, ": T = ", T, " tokens, expected 1..65535");
    SXB_CHECK(d >= kChunk && d <= (1 << 20) && d % kChunk == 0, fn, ": d = ", d, ", expected a multiple of ", kChunk, " up to ", 1 << 20);
    return SXB_OK;
}
int check_hc_weight(const char *fn, const SxbQView *w) {
    SXB_CHECK(w != nullptr && w->q != nullptr && w->scale != nullptr && w->minv != nullptr, fn, ": null weight pointer");
    SXB_CHECK(w->G == 32 || w->G == 64 || w->G == 128, fn, ": group size ", w->G, " unsupported (32, 64 or 128)");
    SXB_CHECK(w->K >= w->G && w->K % w->G == 0, fn, ": K = ", w->K, " must be a positive multiple of group size ", w->G);
    SXB_CHECK(aligned16(w->q), fn, ": code array ", (const void *)w->q, " must be 16-byte aligned for vector loads");
    return SXB_OK;
}

template <int BITS>
int mix_down(const void *x, const SxbQView *w, int64_t T, int64_t H, int64_t d, int64_t r, int inject, float eps, float *h, float *w_in,
             float *inv, int act, sxb_stream_t stream) {
    const char *fn = "hc_mix_down";
    if (int rc = check_hc_shape(fn, T, H, d)) return rc;
    if (int rc = check_hc_weight(fn, w)) return rc;
    SXB_CHECK(act_ok(act), fn, ": unsupported activation dtype ", act);
    SXB_CHECK(x != nullptr && h != nullptr && inv != nullptr, fn, ": null pointer (x=", x, ", h=", (const void *)h, ", inv=", (const void *)inv, ")");
    SXB_CHECK((inject != 0) == (w_in != nullptr), fn, ": w_in must be given exactly when inject (inject=", inject, ", w_in=", (const void *)w_in, ")");
    SXB_CHECK(r >= 1 && r <= kMaxRank, fn, ": r = ", r, ", expected 1..", kMaxRank);
    SXB_CHECK(w->K == H * d, fn, ": weight K = ", w->K, " != H*d = ", H * d);
    const int64_t R = r + (inject ? H : 0);
    SXB_CHECK(w->N == R, fn, ": weight has ", w->N, " rows, expected r", inject ? " + H" : "", " = ", R);
    SXB_CHECK(aligned16(x), fn, ": x ", x, " must be 16-byte aligned");
    SXB_CHECK(std::isfinite(eps) && eps > 0.f, fn, ": eps must be finite and > 0, got ", eps);
    SXB_CHECK((w->K / kChunk) % kParts == 0, fn, ": H*d = ", w->K, " must be a multiple of ", kChunk * kParts, " (eight parts of whole chunks a row)");
    // The longest row of streams is part of the interface (a token's streams and its chunks' sums in 196 KB); the kernel itself would take a longer one.
    const size_t per_token = (size_t)w->K * act_bytes(act) + (size_t)(w->K / kChunk) * 8;
    SXB_CHECK(per_token <= 200 * 1024 - 4352, fn, ": H*d = ", w->K, " is longer than the mix takes (", act_name(act), ": at most ",
              (200 * 1024 - 4352) / (4 * act_bytes(act) + 1) * 4 / (kChunk * kParts) * (kChunk * kParts), ")");
    const int NT = act == SXB_ACT_F32 ? std::min(2, token_eights(T)) : token_eights(T);
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeClusterDimension, attr.val.clusterDim.x = kParts, attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.gridDim = dim3((unsigned)((R + kMmaRows - 1) / kMmaRows * kParts), (unsigned)((T + NT * kMmaTokens - 1) / (NT * kMmaTokens)));
    cfg.blockDim = dim3(32 * kDownWarps), cfg.stream = static_cast<cudaStream_t>(stream), cfg.attrs = &attr, cfg.numAttrs = 1;
    auto launch = [&](auto kern, auto *xt) {
        return cudaLaunchKernelEx(&cfg, kern, xt, w->q, w->scale, w->minv, R, w->K, w->G, d, (int)r, eps, T, h, w_in, inv);
    };
    cudaError_t e;
    if (act == SXB_ACT_F32) {
        auto xt = static_cast<const float *>(x);
        e = NT == 1 ? launch(hc_down_kernel<float, BITS, 1>, xt) : launch(hc_down_kernel<float, BITS, 2>, xt);
    } else {
        auto xt = static_cast<const uint16_t *>(x);
        e = NT == 1 ? launch(hc_down_kernel<uint16_t, BITS, 1>, xt) : NT == 2 ? launch(hc_down_kernel<uint16_t, BITS, 2>, xt) : launch(hc_down_kernel<uint16_t, BITS, 4>, xt);
    }
    SXB_CUDA(e, fn, ": launching T=", T, " R=", R, " K=", w->K);
    SXB_CHECK_LAUNCH(fn, " Q", BITS, " ", act_name(act), " T=", T, " R=", R, " K=", w->K, " G=", w->G);
    return SXB_OK;
}

// Shared memory of hc_up_kernel.  The limit that a launch asks for is the function's, one for all threads of the process: it is always that of the
// longest rank, or a call of a short one would lower it between another thread's request and launch.
constexpr size_t up_smem_bytes(int64_t r, int NT) { return (size_t)(r / kChunk) * NT * (3 * 32 * sizeof(uint4) + kMmaTokens * sizeof(float)); }
static_assert(up_smem_bytes(kMaxRank, 4) <= 200 * 1024, "with its static shared memory an SM has it");

template <int BITS>
int mix_up(const float *h, const SxbQView *w, const void *x, const float *norm_w, const float *inv, int64_t T, int64_t H, int64_t d,
           void *u, int act, sxb_stream_t stream) {
    const char *fn = "hc_mix_up";
    if (int rc = check_hc_shape(fn, T, H, d)) return rc;
    if (int rc = check_hc_weight(fn, w)) return rc;
    SXB_CHECK(act_ok(act), fn, ": unsupported activation dtype ", act);
    SXB_CHECK(h != nullptr && x != nullptr && norm_w != nullptr && inv != nullptr && u != nullptr, fn, ": null pointer (h=", (const void *)h,
              ", x=", x, ", norm_w=", (const void *)norm_w, ", inv=", (const void *)inv, ", u=", u, ")");
    SXB_CHECK(w->N == H * d, fn, ": W_up has ", w->N, " rows, expected H*d = ", H * d);
    SXB_CHECK(w->K >= kChunk && w->K <= kMaxRank && w->K % kChunk == 0, fn, ": W_up K (the rank r) = ", w->K, ", expected a multiple of ",
              kChunk, " up to ", kMaxRank);
    SXB_CHECK(apart(u, T * d * act_bytes(act), x, T * H * d * act_bytes(act)), fn, ": u overlaps the streams x");
    const int64_t r = w->K;
    const int NT = token_eights(T);
    const size_t smem = up_smem_bytes(r, NT);
    const bool vec_h = aligned16(h);
    auto st = static_cast<cudaStream_t>(stream);
#define SXB_HC_UP(TYPE, NTV)                                                                                                           \
    do {                                                                                                                               \
        auto kern = hc_up_kernel<TYPE, BITS, NTV>;                                                                                     \
        SXB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)up_smem_bytes(kMaxRank, NTV)), fn, ": reserving shared memory"); \
        const dim3 grid((unsigned)(d / kUpCols), (unsigned)((T + NTV * kMmaTokens - 1) / (NTV * kMmaTokens)));                          \
        kern<<<grid, 32 * kStreams, smem, st>>>(h, w->q, w->scale, w->minv, w->G, static_cast<const TYPE *>(x), norm_w, inv, d, (int)r, T,  \
                                                vec_h, static_cast<TYPE *>(u));                                                        \
    } while (0)
#define SXB_HC_UP_T(TYPE)                    \
    do {                                     \
        if (NT == 4) SXB_HC_UP(TYPE, 4);     \
        else if (NT == 2) SXB_HC_UP(TYPE, 2);\
        else SXB_HC_UP(TYPE, 1);             \
    } while (0)
    if (act == SXB_ACT_F32) SXB_HC_UP_T(float);
    else SXB_HC_UP_T(uint16_t);
#undef SXB_HC_UP_T
#undef SXB_HC_UP
    SXB_CHECK_LAUNCH(fn, " Q", BITS, " ", act_name(act), " T=", T, " d=", d, " r=", r, " G=", w->G, " NT=", NT);
    return SXB_OK;
}

}  // namespace
}  // namespace sxb

using namespace sxb;

extern "C" {

int sxb_hc_mix_down_q4(const void *x, const SxbQView *w, int64_t T, int64_t H, int64_t d, int64_t r, int inject, float eps, float *h,
                       float *w_in, float *inv, int act, sxb_stream_t stream) {
    return mix_down<4>(x, w, T, H, d, r, inject, eps, h, w_in, inv, act, stream);
}
int sxb_hc_mix_down_q8(const void *x, const SxbQView *w, int64_t T, int64_t H, int64_t d, int64_t r, int inject, float eps, float *h,
                       float *w_in, float *inv, int act, sxb_stream_t stream) {
    return mix_down<8>(x, w, T, H, d, r, inject, eps, h, w_in, inv, act, stream);
}
int sxb_hc_mix_up_q4(const float *h, const SxbQView *w_up, const void *x, const float *norm_w, const float *inv, int64_t T, int64_t H,
                     int64_t d, void *u, int act, sxb_stream_t stream) {
    return mix_up<4>(h, w_up, x, norm_w, inv, T, H, d, u, act, stream);
}
int sxb_hc_mix_up_q8(const float *h, const SxbQView *w_up, const void *x, const float *norm_w, const float *inv, int64_t T, int64_t H,
                     int64_t d, void *u, int act, sxb_stream_t stream) {
    return mix_up<8>(h, w_up, x, norm_w, inv, T, H, d, u, act, stream);
}

int sxb_to_chunk_major(const SxbQView *w, int bits, uint8_t *q, uint16_t *scale, uint16_t *minv, sxb_stream_t stream) {
    const char *fn = "to_chunk_major";
    if (int rc = check_hc_weight(fn, w)) return rc;
    SXB_CHECK(bits == 4 || bits == 8, fn, ": ", bits, "-bit codes unsupported (4 or 8)");
    SXB_CHECK(q != nullptr && scale != nullptr && minv != nullptr, fn, ": null output pointer");
    SXB_CHECK(w->N >= 1 && w->K % kChunk == 0, fn, ": chunk-major needs K % 32 == 0 (32-code chunks), got K = ", w->K);
    SXB_CHECK(reinterpret_cast<uintptr_t>(q) % 16 == 0, fn, ": output codes must be 16-byte aligned");
    const int64_t words = w->N * (w->K / kChunk) * (bits == 4 ? 4 : 8);
    const unsigned blocks = (unsigned)std::min<int64_t>((words + 255) / 256, (int64_t)sm_count() * 8);
    chunk_major_kernel<<<blocks, 256, 0, static_cast<cudaStream_t>(stream)>>>(w->q, w->scale, w->minv, w->N, w->K, w->G, bits == 4 ? 16 : 32, q,
                                                                             scale, minv);
    SXB_CHECK_LAUNCH(fn, " N=", w->N, " K=", w->K, " G=", w->G, " bits=", bits);
    return SXB_OK;
}

}  // extern "C"
