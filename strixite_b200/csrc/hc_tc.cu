// The hyper-connection mix for multi-token forwards on the tensor cores (kernels/hc_wmma.hpp:34-47, kernels/hc_wmma.hip):
// the same math and weight layouts as hc.cu's per-token forms, with the numerics of the reference's matrix-unit path -
// x and h rounded once to F16, the weights dequantized to F16 (code * scale + min, one rounding), FP32 accumulation over
// each product's whole K range; norms, gates and the stream combine in FP32.
//
//   down  runs on this library's tcgen05 expert kernel: a = sum_s inv[t, s] * (W'_s . X_s[t]) is a grouped projection with the H streams as H "experts": slot t * H + s
//         holds the row X_s[t] (X [T, H*d] read as [T*H, d] IS that slot-major matrix), expert s the weight's column range
//         [s d, (s + 1) d) restacked as rows [s Rp, (s + 1) Rp) of a [H * Rp, d] view (Rp = R rounded up to 16, the padding
//         rows zero).  One pass over X computes inv and writes the tile-blocked F16 operand; the grouping workspace of that
//         regular pattern is written by formula under that pass (no ids, no sort); the grouped kernel leaves FP32 per-slot dots; a last pass
//         folds them with inv, in stream order (kernels/hc_wmma.hip:136-150), into h and w_in.
//   up    z = h W_up^T is a dense projection of h [T, r] on W_up [H*d, r], r padded to a multiple of 128 by zero groups, its rows in the order
//         that makes the four streams of an output column neighbours in tensor memory; the kernel's epilogue is the stream combine itself,
//         u = (1/H) sum_s sigmoid(z_s) * X_s * inv_s * (1 + norm_w_s) (kernels/hc_wmma.hip:244-272), so z never exists
//         in memory.  Ranks up to 512: a kernel of its own (hc_up_tc_kernel).  Above: the general kernel, on W_up un-chunked to row-major.
// The re-layouts of weights (a few MB) are done per call into the caller's workspace: the views an engine holds
// stay the reference's (row-major folded down weight, chunk-major up weight), shared with the per-token kernels.

#include "grouped_tc.cuh"
#include "skinny_mma.cuh"

#include <algorithm>
#include <cmath>

namespace sxb {
namespace {

constexpr int kStreams = 4;
constexpr int kChunk = 32;           // codes per chunk of the chunk-major layout
constexpr int64_t kMaxRank = 1024;

inline int64_t up16(int64_t v) { return (v + 15) / 16 * 16; }
inline int64_t up128(int64_t v) { return (v + 127) / 128 * 128; }
inline size_t al256(size_t v) { return (v + 255) / 256 * 256; }

// Eight FP32 values -> one 16-byte chunk of F16 in the k order of a BITS-bit weight operand ([0 4 1 5 2 6 3 7] for Q4).
template <int BITS>
__device__ inline uint4 f16_chunk(const float (&f)[8]) {
    uint4 o;
    if (BITS == 4) {
        o.x = h2_as_u32(__floats2half2_rn(f[0], f[4])), o.y = h2_as_u32(__floats2half2_rn(f[1], f[5]));
        o.z = h2_as_u32(__floats2half2_rn(f[2], f[6])), o.w = h2_as_u32(__floats2half2_rn(f[3], f[7]));
    } else {
        o.x = h2_as_u32(__floats2half2_rn(f[0], f[1])), o.y = h2_as_u32(__floats2half2_rn(f[2], f[3]));
        o.z = h2_as_u32(__floats2half2_rn(f[4], f[5])), o.w = h2_as_u32(__floats2half2_rn(f[6], f[7]));
    }
    return o;
}
// Eight consecutive activations starting at element i (a multiple of 8) as FP32.
__device__ inline void load8(const float *p, int64_t i, float (&f)[8]) {
    const float4 a = __ldg(reinterpret_cast<const float4 *>(p + i)), b = __ldg(reinterpret_cast<const float4 *>(p + i) + 1);
    f[0] = a.x, f[1] = a.y, f[2] = a.z, f[3] = a.w, f[4] = b.x, f[5] = b.y, f[6] = b.z, f[7] = b.w;
}
__device__ inline void load8(const uint16_t *p, int64_t i, float (&f)[8]) {
    const uint4 u = __ldg(reinterpret_cast<const uint4 *>(p + i));
    const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) f[2 * j] = __uint_as_float(w[j] << 16), f[2 * j + 1] = __uint_as_float(w[j] & 0xffff0000u);
}

// ---- down ----------------------------------------------------------------------------------------------------------

struct DownStack {
    const uint8_t *q;  // the folded down weight [R, H*d]
    const uint16_t *scale, *minv;
    int64_t R, Rp, G;
    uint32_t *qo;      // its per-stream stacks [H * Rp, d]
    uint16_t *so, *mo;
    RouteWords L;      // the grouping workspace of T slots a stream
    int32_t *ws;
};

// The folded down weight [R, H*d] -> per-stream stacks [H * Rp, d]: codes, scales and mins of columns [s d, (s + 1) d) of
// row n become row s * Rp + n; rows n >= R are zero codes with zero scale and min.  And the grouping workspace.
__device__ __noinline__ void prepare_down(const DownStack &k, int64_t T, int64_t d, int bits, int64_t first, int64_t stride) {
    const int64_t row_vecs = d * bits / 128, row_groups = d / k.G;  // 16-byte pieces a stream's row
    const uint4 *qi = reinterpret_cast<const uint4 *>(k.q);
    uint4 *qv = reinterpret_cast<uint4 *>(k.qo);
    for (int64_t i = first; i < kStreams * k.Rp * row_vecs; i += stride) {
        const int64_t w = i % row_vecs, sn = i / row_vecs, n = sn % k.Rp, s = sn / k.Rp;
        qv[i] = n < k.R ? __ldg(qi + (n * kStreams + s) * row_vecs + w) : make_uint4(0u, 0u, 0u, 0u);
    }
    for (int64_t i = first; i < kStreams * k.Rp * row_groups; i += stride) {
        const int64_t g = i % row_groups, sn = i / row_groups, n = sn % k.Rp, s = sn / k.Rp;
        const int64_t at = (n * kStreams + s) * row_groups + g;
        k.so[i] = n < k.R ? k.scale[at] : (uint16_t)0, k.mo[i] = n < k.R ? k.minv[at] : (uint16_t)0;
    }
    write_regular_routes(k.L, T, k.ws, first, stride);
}

// One pass over X [T, H*d]: inv[t, s] = 1 / sqrt(mean(X_s[t]^2) + eps) (kernels/hc_wmma.hip:25-45; skipped when the caller
// has it), and the row X_s[t] as F16 in the tile-blocked form at the position the pack gives slot t * H + s: bucket s
// starts at s * T and holds its slots in ascending order, and a row's swizzle depends on its place in its tile modulo 8
// only, which is t modulo 8 for every tile size in use.  A warp per row, rows in position order.
// The launch's first `stack_blocks` CTAs meanwhile restack the weight and write the grouping workspace (as launches of their own those took 10 us
// of a 4096-token mix, which the pass over X now hides).
template <typename TX, int BITS>
__global__ void __launch_bounds__(256) hc_stage_down_kernel(const TX *__restrict__ x, int64_t T, int64_t d, float eps, bool want_inv,
                                                            float *__restrict__ inv, unsigned char *__restrict__ xs, const __grid_constant__ DownStack k,
                                                            int stack_blocks) {
    if ((int)blockIdx.x < stack_blocks) {
        prepare_down(k, T, d, BITS, (int64_t)blockIdx.x * blockDim.x + threadIdx.x, (int64_t)stack_blocks * blockDim.x);
        return;
    }
    const int lane = threadIdx.x & 31;
    const int64_t warps = (int64_t)((int)gridDim.x - stack_blocks) * (blockDim.x >> 5), S = T * kStreams;
    const int chunks = (int)(d / 8);
    for (int64_t pos = (int64_t)((int)blockIdx.x - stack_blocks) * (blockDim.x >> 5) + (threadIdx.x >> 5); pos < S; pos += warps) {
        const int64_t s = pos / T, t = pos % T;
        const TX *row = x + (t * kStreams + s) * d;
        float ssq = 0.f;
        for (int k8 = lane; k8 < chunks; k8 += 128) {
            float f[4][8];
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (k8 + 32 * u < chunks) load8(row, (int64_t)(k8 + 32 * u) * 8, f[u]);
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int kk = k8 + 32 * u;
                if (kk < chunks) {
#pragma unroll
                    for (int j = 0; j < 8; ++j) ssq = fmaf(f[u][j], f[u][j], ssq);
                    *reinterpret_cast<uint4 *>(xs + tiled_offset(S, kk >> 3, pos, (int)(t & 7), kk & 7)) = f16_chunk<BITS>(f[u]);
                }
            }
        }
        if (want_inv) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) ssq += __shfl_xor_sync(0xffffffffu, ssq, o);
            if (lane == 0) inv[t * kStreams + s] = 1.0f / sqrtf(ssq / (float)d + eps);
        }
    }
}

// a = sum_s inv[t, s] * P[t * H + s, n] in stream order, z = a / H, h = silu(z) for n < r, w_in = 2 sigmoid(z) after
// (kernels/hc_wmma.hip:136-150).
__global__ void __launch_bounds__(256) hc_finish_down_kernel(const float *__restrict__ partial, const float *__restrict__ inv, int64_t T,
                                                             int64_t R, int64_t Rp, int64_t r, float *__restrict__ h,
                                                             float *__restrict__ w_in) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= T * R) return;
    const int64_t t = i / R, n = i % R;
    float a = 0.f;
#pragma unroll
    for (int s = 0; s < kStreams; ++s) a = fmaf(inv[t * kStreams + s], partial[(t * kStreams + s) * Rp + n], a);
    const float z = a / (float)kStreams;
    if (n < r) h[t * r + n] = z / (1.0f + expf(-z));
    else w_in[t * kStreams + (n - r)] = 2.0f / (1.0f + expf(-z));
}

// ---- inject + inv --------------------------------------------------------------------------------------------------

// kernels/hc_wmma.hip:47-73 hc_inject_inv: X[t, s d + j] = stored(fma(w_in[t, s], y[t, j], X[t, s d + j])) and inv[t, s]
// from the stored values, in one pass.  A CTA per token; a thread takes columns j and updates their four streams.
template <typename TX>
__global__ void __launch_bounds__(256) hc_inject_inv_kernel(TX *__restrict__ x, const float *__restrict__ w_in, const TX *__restrict__ y,
                                                            int64_t d, float eps, float *__restrict__ inv) {
    __shared__ float red[kStreams][8];
    const int64_t t = blockIdx.x;
    TX *xr = x + t * kStreams * d;
    float wi[kStreams], ssq[kStreams] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int s = 0; s < kStreams; ++s) wi[s] = w_in[t * kStreams + s];
    for (int64_t j = threadIdx.x; j < d; j += blockDim.x) {
        const float v = load_as_f32(y, t * d + j);
#pragma unroll
        for (int s = 0; s < kStreams; ++s) {
            store_from_f32(xr, s * d + j, fmaf(wi[s], v, load_as_f32(xr, s * d + j)));
            const float kept = load_as_f32(xr, s * d + j);  // the stored (rounded) value, as the next mix reads it
            ssq[s] = fmaf(kept, kept, ssq[s]);
        }
    }
#pragma unroll
    for (int s = 0; s < kStreams; ++s) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) ssq[s] += __shfl_xor_sync(0xffffffffu, ssq[s], o);
        if ((threadIdx.x & 31) == 0) red[s][threadIdx.x >> 5] = ssq[s];
    }
    __syncthreads();
    if (threadIdx.x < kStreams) {
        float sum = 0.f;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) sum += red[threadIdx.x][w];
        inv[t * kStreams + threadIdx.x] = 1.0f / sqrtf(sum / (float)d + eps);
    }
}

// ---- up ------------------------------------------------------------------------------------------------------------

// Chunk-major W_up [N = 4 d, r] (32-code chunk c of row n at word (c N + n) * cw, group g's scale / min at [g N + n]) ->
// row-major [N, Kp] with Kp >= r: the chunks and groups past r are zero codes, zero scale, zero min.  Row
// rb * 128 + q * 32 + l of the result is W_up's row s d + j with s = l & 3, j = rb * 32 + q * 8 + (l >> 2): the order in
// which the up mix's epilogue wants the rows in tensor-memory lanes (TcHcUp).
__device__ inline int64_t up_source_row(int64_t row, int64_t d) {
    const int64_t rb = row >> 7, q = (row >> 5) & 3, l = row & 31;
    return (l & 3) * d + rb * 32 + q * 8 + (l >> 2);
}
__global__ void __launch_bounds__(256) hc_unchunk_up_kernel(const uint8_t *__restrict__ q, const uint16_t *__restrict__ scale,
                                                            const uint16_t *__restrict__ minv, int64_t d, int64_t r, int64_t Kp, int64_t G,
                                                            int bits, uint32_t *__restrict__ qo, uint16_t *__restrict__ so,
                                                            uint16_t *__restrict__ mo) {
    const int64_t N = kStreams * d;
    const int64_t cv = bits / 4, chunks = r / kChunk, chunks_p = Kp / kChunk, groups = r / G, groups_p = Kp / G;  // cv: 16-byte pieces a chunk
    const int64_t stride = (int64_t)gridDim.x * blockDim.x, first = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const uint4 *qi = reinterpret_cast<const uint4 *>(q);
    uint4 *qv = reinterpret_cast<uint4 *>(qo);
    for (int64_t i = first; i < N * chunks_p * cv; i += stride) {
        const int64_t w = i % cv, nc = i / cv, c = nc % chunks_p, n = up_source_row(nc / chunks_p, d);
        qv[i] = c < chunks ? __ldg(qi + (c * N + n) * cv + w) : make_uint4(0u, 0u, 0u, 0u);
    }
    for (int64_t i = first; i < N * groups_p; i += stride) {
        const int64_t g = i % groups_p, n = up_source_row(i / groups_p, d);
        so[i] = g < groups ? scale[g * N + n] : (uint16_t)0, mo[i] = g < groups ? minv[g * N + n] : (uint16_t)0;
    }
}

// h [M, r] FP32 -> F16, tile-blocked in the rows' own order (a dense projection's operand), r padded to Kp with zeros.
template <int BITS>
__global__ void __launch_bounds__(256) hc_stage_h_kernel(const float *__restrict__ h, int64_t M, int64_t r, int64_t Kp,
                                                         unsigned char *__restrict__ hs) {
    const int64_t chunks_p = Kp / 8;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < M * chunks_p; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t t = i / chunks_p;
        const int kk = (int)(i % chunks_p);
        float f[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        if ((int64_t)kk * 8 < r) load8(h + t * r, (int64_t)kk * 8, f);
        *reinterpret_cast<uint4 *>(hs + tiled_offset(M, kk >> 3, t, (int)(t & 7), kk & 7)) = f16_chunk<BITS>(f);
    }
}

// ---- up, ranks up to 512: a kernel of its own ------------------------------------------------------------------------

// z = h W_up^T and the stream combine for 128 rows of W_up - 32 output columns, their four streams in neighbouring tensor-memory lanes (up_source_row) -
// against up to 128 tokens an item.  The contraction is short (r = 320: three steps of 128 k), so what an item costs is everything but its products: on
// the general kernel, whose items dequantize their rows again for every 128 tokens, look for their powers of two and pass through its rings,
// 11200 SM cycles, of which the MMAs take 1500.  Here a CTA takes neighbouring items, the tokens of a row block one after another, and the
// block's weights stay in tensor memory: dequantized once or twice a CTA, straight from the chunk-major codes.
// Warps: sixteen for the epilogue, four producers, MMA issue, copies of h, copies of X.  Waits are bounded; one that runs out raises the CTA's abort
// flag and is recorded in the library's status words.  4096 tokens, d = 4096, r = 320, Q8: 169 us and 6 for the re-layout -> 97, 6500 SM cycles an
// item.  What bounds it: the epilogue's warps - latencies of shared memory and the special-function unit (33 % busy), issue slots 46 %.
constexpr int kUpTile = 128, kUpSubBytes = kUpTile * 128, kUpStageBytes = 2 * kUpSubBytes, kUpSteps = 4;  // steps of 128 k at most
constexpr int kUpEpiWarps = 16, kUpProducer = kUpEpiWarps, kUpMma = kUpEpiWarps + 4, kUpCopy = kUpEpiWarps + 5, kUpXCopy = kUpEpiWarps + 6,
              kUpThreads = 32 * (kUpEpiWarps + 7);
constexpr int kUpACols = 256;   // first tensor-memory column of the weights, behind two accumulators of 128
constexpr int kUpGroup = kUpEpiWarps / 2;  // epilogue warps that share an item; the two groups take items by turns
constexpr int kUpScaleBufs = 4; // row blocks whose powers of two are kept: the epilogue is two accumulators behind at most
template <typename TX> constexpr int kUpXBytes = 4 * kUpTile * 32 * (int)sizeof(TX);  // an item's X: 128 tokens x 4 streams x 32 columns
template <typename TX> constexpr int kUpBuf = kUpXBytes<TX> + kUpTile * 16;           // and inv
template <typename TX> constexpr int kUpStages = sizeof(TX) == 2 ? 4 : 2;             // what shared memory holds beside two of them

struct HcUpArgs {
    const unsigned char *hs;  // h, tile-blocked F16 [M, Kp]
    const uint8_t *q;         // chunk-major W_up
    const uint16_t *scale, *minv;
    const float *inv, *norm_w;
    void *u;
    int64_t M, d;
    int r, G, steps;
    uint32_t *status;
    unsigned long long wait_limit_ns;
    int test_skip_slot;  // >= 0: CTA 0 never issues the copies of that stage fill of h, so that a wait runs out (tests only)
};

// 2^v and 1 / v on the special-function unit, results below 2^-126 as zero: the one is added to one, the other is of a sum of one or more.
__device__ inline float exp2_ftz(float v) {
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
    return r;
}
__device__ inline float rcp_ftz(float v) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
    return r;
}
__device__ inline void store_rounded(float *p, float v) { *p = v; }
__device__ inline void store_rounded(uint16_t *p, float v) { *p = __bfloat16_as_ushort(__float2bfloat16_rn(v)); }

template <int BITS, typename TX>
__global__ void __launch_bounds__(kUpThreads, 1) hc_up_tc_kernel(const HcUpArgs a, const __grid_constant__ CUtensorMap xmap) {
    constexpr int kStages = kUpStages<TX>;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char *smem = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    __shared__ uint64_t b_full[kStages], b_empty[kStages], acc_full[2], acc_empty[2], x_full[2], x_empty[2], w_full, w_free, drain_bar;
    __shared__ float row_scale[kUpScaleBufs][128];
    __shared__ uint32_t tmem_base_smem;
    __shared__ int abort_flag;
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31, quad = warp & 3;
    const int tiles = (int)((a.M + kUpTile - 1) / kUpTile);
    const int64_t items = (a.d / 32) * tiles;
    const int64_t i0 = items * blockIdx.x / gridDim.x, i1 = items * (blockIdx.x + 1) / gridDim.x;  // item i: row block i / tiles, tokens of tile i % tiles
    volatile int *abort_v = &abort_flag;

    if (threadIdx.x == 0) {
        for (int s = 0; s < kStages; ++s) mbar_init(&b_full[s], 1), mbar_init(&b_empty[s], 1);
        for (int h = 0; h < 2; ++h) mbar_init(&acc_full[h], 1), mbar_init(&acc_empty[h], kUpGroup), mbar_init(&x_full[h], 1), mbar_init(&x_empty[h], kUpGroup);
        mbar_init(&w_full, 4), mbar_init(&w_free, 1), mbar_init(&drain_bar, 1);
        abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == kUpMma) {  // all 512 columns: one CTA per SM
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_smem)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_base_smem;
    auto raise_abort = [&](int64_t item, int role) {
        if (atomicExch(&abort_flag, 1) == 0 && atomicCAS(&a.status[0], 0u, 2u) == 0u) a.status[1] = (uint32_t)item, a.status[2] = (uint32_t)role;
    };
    unsigned char *const x_bufs = smem + kStages * kUpStageBytes;
    auto cnt_of = [&](int tile) { return (int)min((int64_t)kUpTile, a.M - (int64_t)tile * kUpTile); };
    bool copied = false;  // this thread has issued bulk copies

    if (warp >= kUpProducer && warp < kUpMma) {
        // ===================== weights: a lane a row =====================
        const int64_t N = kStreams * a.d;
        const int chunks = a.r / kChunk, groups = a.r / a.G;
        int block = 0;
        for (int64_t rb = i0 / tiles; rb * tiles < i1; ++rb, ++block) {
            const int64_t n = up_source_row(rb * 128 + quad * 32 + lane, a.d);
            // The row's power of two, or none for the quadrant, as the general kernel chooses it (kScaleSpread in grouped_tc_tiled.cu).
            int hi = 0x400, lo = 0x7fff;  // over v = max(|scale| 2^8, |min|) as BF16 bits; 0x400 = an empty group
            for (int g = 0; g < groups; ++g) {
                const int v = max(((int)__ldg(a.scale + g * N + n) & 0x7fff) + 0x400, (int)__ldg(a.minv + g * N + n) & 0x7fff);
                hi = max(hi, v);
                if (v != 0x400) lo = min(lo, v);
            }
            const int e = min(max((hi >> 7) - 8, 127 - 24), 127 + 15);
            const bool natural = __any_sync(0xffffffffu, e > 127 - 10 && lo != 0x7fff && (lo >> 7) - 8 < e - 6);
            const float scale = __int_as_float((127 + 14 + 127 - e) << 23), scale_min = scale * 0x1p-24f;
            row_scale[block % kUpScaleBufs][quad * 32 + lane] = natural ? 1.f : __uint_as_float(((127u + 24u + 127u) << 23) - __float_as_uint(scale));  // undoes it: 2^(24 - k)
            if (block > 0) {  // the MMAs of the block before have read their weights
                const bool ok = mbar_wait(&w_free, (uint32_t)(block - 1) & 1u, abort_v, a.wait_limit_ns);
                if (!__all_sync(0xffffffffu, ok)) {
                    if (lane == 0) raise_abort(rb * tiles, 1);
                    break;
                }
            }
            tc_fence_after();
            const uint32_t to = tmem + ((uint32_t)(quad * 32) << 16) + kUpACols;
#pragma unroll 2
            for (int c = 0; c < a.steps * 4; ++c) {  // 32 codes -> 16 columns
                uint4 dq[4];
                const bool in = c < chunks;
                const int64_t at = (int64_t)(in ? c : 0) * N + n, gi = (int64_t)((in ? c : 0) * kChunk / a.G) * N + n;
                const float sc = in ? bf16_bits_to_f32(__ldg(a.scale + gi)) : 0.f, mn = in ? bf16_bits_to_f32(__ldg(a.minv + gi)) : 0.f;
                const uint4 *src = reinterpret_cast<const uint4 *>(a.q) + at * (BITS / 4);
                const uint4 v0 = __ldg(src), v1 = BITS == 8 ? __ldg(src + (BITS / 8)) : v0;
                if (natural) {
                    const __half2 s2 = __float2half2_rn(sc), m2 = __float2half2_rn(mn);
                    if (BITS == 4) dq[0] = dequant_q4_word(v0.x, s2, m2), dq[1] = dequant_q4_word(v0.y, s2, m2), dq[2] = dequant_q4_word(v0.z, s2, m2), dq[3] = dequant_q4_word(v0.w, s2, m2);
                    else dq[0] = dequant_q8_words(v0.x, v0.y, s2, m2), dq[1] = dequant_q8_words(v0.z, v0.w, s2, m2), dq[2] = dequant_q8_words(v1.x, v1.y, s2, m2), dq[3] = dequant_q8_words(v1.z, v1.w, s2, m2);
                } else {
                    const __half2 s2 = __float2half2_rn(sc * scale), m2 = __float2half2_rn(mn * scale_min), s16 = __hmul2(s2, __float2half2_rn(0.0625f));
                    if (BITS == 4) dq[0] = dequant_q4_scaled(v0.x, s2, s16, m2), dq[1] = dequant_q4_scaled(v0.y, s2, s16, m2), dq[2] = dequant_q4_scaled(v0.z, s2, s16, m2), dq[3] = dequant_q4_scaled(v0.w, s2, s16, m2);
                    else dq[0] = dequant_q8_scaled(v0.x, v0.y, s2, m2), dq[1] = dequant_q8_scaled(v0.z, v0.w, s2, m2), dq[2] = dequant_q8_scaled(v1.x, v1.y, s2, m2), dq[3] = dequant_q8_scaled(v1.z, v1.w, s2, m2);
                }
                __syncwarp();
                tc_st16(to + (uint32_t)c * 16u, dq);
            }
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&w_full);
        }
    } else if (warp == kUpCopy) {
        // ===================== activations: two bulk copies a step =====================
        if (elect_one()) {
            const int64_t line = a.M * 128;  // bytes from one 64-k sub-tile to the next
            uint32_t count = 0;
            for (int64_t i = i0; i < i1 && !*abort_v; ++i) {
                const int tile = (int)(i % tiles);
                const uint32_t bytes = (uint32_t)cnt_of(tile) * 128u;
                const unsigned char *src = a.hs + (int64_t)tile * kUpTile * 128;
                for (int st = 0; st < a.steps; ++st, ++count, src += 2 * line) {
                    const uint32_t stage = count % kStages;
                    if (!mbar_wait(&b_empty[stage], ((count / kStages) & 1u) ^ 1u, abort_v, a.wait_limit_ns)) {
                        raise_abort(i, 5);
                        break;
                    }
                    if (blockIdx.x == 0 && (int)count == a.test_skip_slot) continue;
                    const uint32_t dst = smem_u32(smem) + stage * (uint32_t)kUpStageBytes;
                    mbar_expect_tx(&b_full[stage], 2 * bytes);
                    bulk_g2s(dst, src, bytes, &b_full[stage]);
                    bulk_g2s(dst + kUpSubBytes, src + line, bytes, &b_full[stage]);
                    copied = true;
                }
            }
        }
        __syncwarp();
    } else if (warp == kUpXCopy) {
        // ===================== X and inv, an item ahead: a row is a stream of a token, 16-byte chunks swizzled =====================
        // (by 16-byte asynchronous copies of the epilogue's lanes, each to a row of its own, X took a third of the epilogue's time)
        if (elect_one()) {
            uint32_t count = 0;
            for (int64_t i = i0; i < i1 && !*abort_v; ++i, ++count) {
                const uint32_t half = count & 1u;
                if (!mbar_wait(&x_empty[half], ((count >> 1) & 1u) ^ 1u, abort_v, a.wait_limit_ns)) {
                    raise_abort(i, 5);
                    break;
                }
                const int tile = (int)(i % tiles), x0 = (int)(i / tiles) * 32, y0 = tile * 4 * kUpTile;
                const uint32_t dst = smem_u32(x_bufs) + half * (uint32_t)kUpBuf<TX>, inv_bytes = (uint32_t)cnt_of(tile) * 16u;
                mbar_expect_tx(&x_full[half], (uint32_t)kUpXBytes<TX> + inv_bytes);
                tma_load_2d(dst, &xmap, x0, y0, &x_full[half]);  // rows past the last token read as zeros
                tma_load_2d(dst + kUpXBytes<TX> / 2, &xmap, x0, y0 + 2 * kUpTile, &x_full[half]);
                bulk_g2s(dst + kUpXBytes<TX>, a.inv + (int64_t)tile * kUpTile * 4, inv_bytes, &x_full[half]);
                copied = true;
            }
        }
        __syncwarp();
    } else if (warp == kUpMma) {
        // ===================== MMA issue: the whole warp, uniform control flow =====================
        const uint32_t leader = elect_one() ? 1u : 0u;
        const uint64_t desc0 = smem_desc(smem_u32(smem));
        uint32_t count = 0, acc_count = 0;
        int block = -1;
        int64_t rb_at = -1;
        bool ok = true;
        for (int64_t i = i0; i < i1 && ok; ++i, ++acc_count) {
            const int64_t rb = i / tiles;
            if (rb != rb_at) {
                rb_at = rb, ++block;
                ok = __all_sync(0xffffffffu, mbar_wait(&w_full, (uint32_t)block & 1u, abort_v, a.wait_limit_ns));
                if (!ok) {
                    if (leader) raise_abort(i, 3);
                    break;
                }
            }
            const uint32_t half = acc_count & 1u;
            ok = __all_sync(0xffffffffu, mbar_wait(&acc_empty[half], ((acc_count >> 1) & 1u) ^ 1u, abort_v, a.wait_limit_ns));
            if (!ok) {
                if (leader) raise_abort(i, 2);
                break;
            }
            tc_fence_after();
            const uint32_t idesc = __reduce_max_sync(0xffffffffu, instr_desc((cnt_of((int)(i % tiles)) + 15) & ~15));
            for (int st = 0; st < a.steps; ++st, ++count) {
                const uint32_t stage = count % kStages;
                ok = __all_sync(0xffffffffu, mbar_wait(&b_full[stage], (count / kStages) & 1u, abort_v, a.wait_limit_ns));
                if (!ok) {
                    if (leader) raise_abort(i, 3);
                    break;
                }
                tc_fence_after();
                tc_step_ts<kUpSubBytes>(leader, tmem + half * (uint32_t)kUpTile, tmem + (uint32_t)(kUpACols + st * 64), (uint32_t)desc0 + stage * (uint32_t)(kUpStageBytes / 16),
                                        (uint32_t)(desc0 >> 32), idesc, st != 0);
                tc_commit_if(leader, &b_empty[stage]);
            }
            if (ok) tc_commit_if(leader, &acc_full[half]);
            if (ok && (i + 1) / tiles != rb) tc_commit_if(leader, &w_free);  // the last item of the block: its weights have been read
        }
        tc_commit_if(leader, &drain_bar);  // not given up while aborting: tensor memory must not be released under an MMA
        mbar_wait(&drain_bar, 0u, nullptr, a.wait_limit_ns);
        __syncwarp();
    } else if (warp < kUpEpiWarps) {
        // ===================== epilogue: the stream combine (TcHcUp) =====================
        // Lane = (stream s = lane & 3, output column j); a warp has 64 of the item's tokens, 32 a pass and every other 32.  One accumulator and one buffer of X belong to
        // a group, and while one group's warps are at the special-function unit, which bounds the terms, the other's are at shuffles and stores.
        constexpr int es = sizeof(TX), kRowBytes = 32 * es;
        const int s = lane & 3, jj = lane >> 2, tok0 = ((warp >> 2) & 1) * 32;
        const uint32_t half = (uint32_t)(warp / kUpGroup);
        // this lane's element of a token at even / odd place: row 4 tok + s, column quad * 8 + jj, its chunk swizzled (64-byte rows by row >> 1 & 3,
        // 128-byte rows by row & 7)
        const TX *xs_[2];
#pragma unroll
        for (int p = 0; p < 2; ++p) {
            const int chunk = (quad * 8 + jj) * es / 16, swz = es == 2 ? p * 2 + (s >> 1) : p * 4 + s;
            xs_[p] = reinterpret_cast<const TX *>(x_bufs + half * (uint32_t)kUpBuf<TX> + (4 * (tok0 + p) + s) * kRowBytes + ((chunk ^ swz) << 4) + (jj * es) % 16);
        }
        const float *ivs = reinterpret_cast<const float *>(x_bufs + half * (uint32_t)kUpBuf<TX> + kUpXBytes<TX>) + tok0 * 4 + s;
        const bool b0 = (lane & 1) != 0, b1 = (lane & 2) != 0;
        const int mine = (b0 ? 2 : 0) + (b1 ? 1 : 0);  // which of a group's four tokens this lane ends up with
        uint32_t phase = 0;
        for (int64_t i = i0 + half; i < i1; i += 2, phase ^= 1u) {
            const int64_t rb = i / tiles, j = rb * 32 + quad * 8 + jj;
            const int tile = (int)(i % tiles), live = cnt_of(tile) - tok0;
            const float nwp = 1.0f + __ldg(a.norm_w + (int64_t)s * a.d + j);
            const bool ok = mbar_wait(&x_full[half], phase, abort_v, a.wait_limit_ns) && mbar_wait(&acc_full[half], phase, abort_v, a.wait_limit_ns);
            if (!__all_sync(0xffffffffu, ok)) {
                if (lane == 0) raise_abort(i, 4);
                break;
            }
            tc_fence_after();
            // sigmoid(z) = 1 / (1 + 2^(-z log2 e)), with the row's power of two taken out of z on the way
            const float nz = -1.44269504f * row_scale[(int)(rb - i0 / tiles) % kUpScaleBufs][quad * 32 + lane];
            const uint64_t nz2 = pair(nz, nz), nwp2 = pair(nwp, nwp), one2 = pair(1.0f, 1.0f);
            TX *up = static_cast<TX *>(a.u) + ((int64_t)tile * kUpTile + tok0 + mine) * a.d + j;
#pragma unroll 1
            for (int p = 0; p < 2; ++p, up += 64 * a.d) {
                const int left = live - 64 * p;
                float va[16], vb[16];
                const uint32_t tcol = tmem + ((uint32_t)(quad * 32) << 16) + half * (uint32_t)kUpTile + (uint32_t)(tok0 + 64 * p);
                if (left > 0) tc_ld16x2(tcol, tcol + 16u, va, vb);
                if (p == 1) {
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&acc_empty[half]);
                }
                // First every token's term of this lane's stream, in place of its accumulator (shared-memory reads and arithmetic only: a store
                // to u in between would fence the next token's reads behind it, both being generic addresses).  Then the four streams of a
                // column - lanes l, l ^ 1, l ^ 2, l ^ 3 - four tokens at a time by a reduce-scatter: three shuffles instead of the eight of
                // four butterflies, and it leaves each of the four lanes with the sum of one token, which that lane stores.
                if (left > 0) {
#pragma unroll
                    for (int t = 0; t < 32; t += 2) {  // two tokens' factors in one instruction, each rounded as on its own (4096 tokens 104.8 -> 101.3 us under load, 1024 36.9 -> 34.8, 77 18.2 -> 16.4)
                        float (&v)[16] = t < 16 ? va : vb;
                        const int q = t & 15;
                        float e0, e1;
                        unpair(mul_pair(pair(v[q], v[q + 1]), nz2), e0, e1);
                        unpair(add_pair(one2, pair(exp2_ftz(e0), exp2_ftz(e1))), e0, e1);
                        const uint64_t x2 = pair(load_as_f32(xs_[0], p * 8192 + (t >> 1) * 256), load_as_f32(xs_[1], p * 8192 + (t >> 1) * 256));
                        const uint64_t c2 = mul_pair(mul_pair(x2, pair(ivs[p * 256 + t * 4], ivs[p * 256 + t * 4 + 4])), nwp2);
                        unpair(mul_pair(c2, pair(rcp_ftz(e0), rcp_ftz(e1))), v[q], v[q + 1]);
                    }
                }
                if (p == 1) {
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&x_empty[half]);
                }
                if (left > 0) {
#pragma unroll
                    for (int k = 0; k < 8; ++k) {
                        const float ta = k < 4 ? va[4 * k] : vb[4 * k - 16], tb = k < 4 ? va[4 * k + 1] : vb[4 * k - 15];
                        const float tc = k < 4 ? va[4 * k + 2] : vb[4 * k - 14], td = k < 4 ? va[4 * k + 3] : vb[4 * k - 13];
                        // lanes with bit 0 clear keep tokens a, b and send c, d; the others the reverse
                        const float k0 = (b0 ? tc : ta) + __shfl_xor_sync(0xffffffffu, b0 ? ta : tc, 1);
                        const float k1 = (b0 ? td : tb) + __shfl_xor_sync(0xffffffffu, b0 ? tb : td, 1);
                        // lanes with bit 1 clear keep the first of the two and send the second; the others the reverse
                        const float sum = (b1 ? k1 : k0) + __shfl_xor_sync(0xffffffffu, b1 ? k0 : k1, 2);
                        if (4 * k + mine < left) store_rounded(up + (int64_t)(4 * k) * a.d, sum * 0.25f);
                    }
                }
            }
        }
    }

    // An aborting CTA must not return under copies into its own shared memory: their issuer lets a generous time pass.
    if (*abort_v && copied)
        for (const unsigned long long t0 = global_ns(); global_ns() - t0 < 50000ull;) {}
    tc_fence_before();
    __syncthreads();
    if (warp == kUpMma) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
    }
}

template <int BITS, typename TX>
int launch_hc_up(const char *fn, const HcUpArgs &a, const void *x, cudaStream_t st) {
    const size_t smem = (size_t)kUpStages<TX> * kUpStageBytes + (size_t)2 * kUpBuf<TX> + 1024;
    // X as [4 T, d], boxes of 32 columns x 256 rows
    CUtensorMap xmap;
    if (int rc = tensor_map_2d(fn, x, sizeof(TX) == 2 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, sizeof(TX), (uint64_t)a.d, (uint64_t)(kStreams * a.M),
                               (uint64_t)a.d * sizeof(TX), 32u, 256u, sizeof(TX) == 2 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B, &xmap))
        return rc;
    auto kern = hc_up_tc_kernel<BITS, TX>;
    SXB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem), fn, ": reserving shared memory");
    const int64_t items = a.d / 32 * ((a.M + kUpTile - 1) / kUpTile);
    kern<<<(unsigned)std::min<int64_t>(items, sm_count()), kUpThreads, smem, st>>>(a, xmap);
    SXB_CHECK_LAUNCH(fn, " T=", a.M, " d=", a.d, " r=", a.r);
    return SXB_OK;
}

// ---- hosts ---------------------------------------------------------------------------------------------------------

int check_shape(const char *fn, int64_t T, int64_t H, int64_t d, const SxbQView *w, int act) {
    SXB_CHECK(H == kStreams, fn, ": H = ", H, " streams, only ", kStreams, " is supported");
    SXB_CHECK(T >= 1 && T <= 65535, fn, ": T = ", T, " tokens, expected 1..65535");
    SXB_CHECK(d >= 128 && d <= (1 << 20) && d % 128 == 0, fn, ": d = ", d, ", the tensor-core mix needs a multiple of 128 up to ", 1 << 20);
    SXB_CHECK(act_ok(act), fn, ": unsupported activation dtype ", act);
    SXB_CHECK(w != nullptr && w->q != nullptr && w->scale != nullptr && w->minv != nullptr, fn, ": null weight pointer");
    SXB_CHECK(w->G == 32 || w->G == 64 || w->G == 128, fn, ": group size ", w->G, " unsupported (32, 64 or 128)");
    SXB_CHECK(w->K >= w->G && w->K % w->G == 0, fn, ": K = ", w->K, " must be a positive multiple of group size ", w->G);
    SXB_CHECK(aligned16(w->q), fn, ": code array ", (const void *)w->q, " must be 16-byte aligned");
    return SXB_OK;
}

// Parts of the down mix's workspace, in bytes from its start; the grouping workspace comes first, so that
// sxb_check_grouped_status reads the caller's pointer as it is.
struct DownWs {
    size_t route, route_bytes, wq, wscale, wmin, xs, partial, total;
};
DownWs down_ws(int64_t T, int64_t d, int64_t R, int bits, int64_t G) {
    const int64_t Rp = up16(R), S = T * kStreams;
    DownWs L{};
    size_t at = 0;
    auto take = [&](size_t bytes) { const size_t o = at; at += al256(bytes); return o; };
    L.route_bytes = (size_t)route_words(S, 1, kStreams).total * 4;
    L.route = take(L.route_bytes);
    L.wq = take((size_t)kStreams * Rp * d * bits / 8), L.wscale = take((size_t)kStreams * Rp * (d / G) * 2), L.wmin = take((size_t)kStreams * Rp * (d / G) * 2);
    L.xs = take((size_t)S * d * 2), L.partial = take((size_t)S * Rp * 4);
    L.total = at;
    return L;
}

template <int BITS>
int mix_down_tc(const void *x, const SxbQView *w, int64_t T, int64_t H, int64_t d, int64_t r, int inject, float eps, float *h, float *w_in,
                float *inv, void *ws, size_t ws_bytes, int act, int inv_ready, sxb_stream_t stream) {
    const char *fn = "hc_mix_down_wmma";
    if (int rc = check_shape(fn, T, H, d, w, act)) return rc;
    SXB_CHECK(d % w->G == 0, fn, ": d = ", d, " not a multiple of group size ", w->G, " (each stream's K range must start a group)");
    SXB_CHECK(x != nullptr && h != nullptr && inv != nullptr && ws != nullptr, fn, ": null pointer (x=", x, ", h=", (const void *)h,
              ", inv=", (const void *)inv, ", ws=", ws, ")");
    SXB_CHECK((inject != 0) == (w_in != nullptr), fn, ": w_in must be given exactly when inject (inject=", inject, ", w_in=", (const void *)w_in, ")");
    SXB_CHECK(r >= 1 && r <= kMaxRank, fn, ": r = ", r, ", expected 1..", kMaxRank);
    const int64_t R = r + (inject ? H : 0), Rp = up16(R), S = T * kStreams;
    SXB_CHECK(w->K == H * d && w->N == R, fn, ": weight [", w->N, ", ", w->K, "], expected [r", inject ? " + H" : "", " = ", R, ", H*d = ", H * d, "]");
    SXB_CHECK(aligned16(x) && reinterpret_cast<uintptr_t>(ws) % 256 == 0, fn, ": x must be 16-byte and the workspace 256-byte aligned");
    SXB_CHECK(std::isfinite(eps) && eps > 0.f, fn, ": eps must be finite and > 0, got ", eps);
    const DownWs L = down_ws(T, d, R, BITS, w->G);
    SXB_CHECK(ws_bytes >= L.total, fn, ": workspace of ", ws_bytes, " bytes, needs ", L.total);
    auto *base = static_cast<unsigned char *>(ws);
    auto st = static_cast<cudaStream_t>(stream);
    auto *partial = reinterpret_cast<float *>(base + L.partial);
    SxbQView stacked{base + L.wq, reinterpret_cast<uint16_t *>(base + L.wscale), reinterpret_cast<uint16_t *>(base + L.wmin), kStreams * Rp, d, w->G};

    const DownStack stack{w->q, w->scale, w->minv, R, Rp, w->G, reinterpret_cast<uint32_t *>(base + L.wq), reinterpret_cast<uint16_t *>(base + L.wscale),
                          reinterpret_cast<uint16_t *>(base + L.wmin), route_words(S, 1, kStreams), reinterpret_cast<int32_t *>(base + L.route)};
    const int64_t stack_vecs = kStreams * Rp * d * BITS / 128;
    const unsigned stage_blocks = (unsigned)std::min<int64_t>((S + 7) / 8, (int64_t)sm_count() * 8);
    const int stack_blocks = (int)std::min<int64_t>((stack_vecs + 255) / 256, (int64_t)sm_count() * 2);
    if (act == SXB_ACT_F32)
        hc_stage_down_kernel<float, BITS><<<stage_blocks + stack_blocks, 256, 0, st>>>(static_cast<const float *>(x), T, d, eps, inv_ready == 0, inv, base + L.xs,
                                                                                       stack, stack_blocks);
    else
        hc_stage_down_kernel<uint16_t, BITS><<<stage_blocks + stack_blocks, 256, 0, st>>>(static_cast<const uint16_t *>(x), T, d, eps, inv_ready == 0, inv,
                                                                                          base + L.xs, stack, stack_blocks);
    SXB_CHECK_LAUNCH(fn, " staging the streams, T=", T, " d=", d);
    if (int rc = tc_partial_grouped<BITS>(fn, base + L.xs, &stacked, kStreams, base + L.route, L.route_bytes, S, 1, partial, SXB_ACT_F16_TILED,
                                          BITS == 4 ? 3 : 4, false, stream))
        return rc;
    hc_finish_down_kernel<<<(unsigned)((T * R + 255) / 256), 256, 0, st>>>(partial, inv, T, R, Rp, r, h, w_in);
    SXB_CHECK_LAUNCH(fn, " Q", BITS, " ", act_name(act), " T=", T, " R=", R, " d=", d, " G=", w->G);
    return SXB_OK;
}

// Parts of the up mix's workspace.  The un-chunked weight is the general kernel's: up to rank 512 its place stays unused (the size is part of the
// interface, which a host may have stored).
struct UpWs {
    size_t wq, wscale, wmin, hs, total;
};
UpWs up_ws(int64_t T, int64_t d, int64_t r, int bits, int64_t G) {
    const int64_t Kp = up128(r), N = kStreams * d;
    UpWs L{};
    size_t at = 0;
    auto take = [&](size_t bytes) { const size_t o = at; at += al256(bytes); return o; };
    L.wq = take((size_t)N * Kp * bits / 8), L.wscale = take((size_t)N * (Kp / G) * 2), L.wmin = take((size_t)N * (Kp / G) * 2);
    L.hs = take((size_t)T * Kp * 2);
    L.total = at;
    return L;
}

template <int BITS>
int mix_up_tc(const float *h, const SxbQView *w, const void *x, const float *norm_w, const float *inv, int64_t T, int64_t H, int64_t d,
              void *u, void *ws, size_t ws_bytes, int act, sxb_stream_t stream) {
    const char *fn = "hc_mix_up_wmma";
    if (int rc = check_shape(fn, T, H, d, w, act)) return rc;
    SXB_CHECK(h != nullptr && x != nullptr && norm_w != nullptr && inv != nullptr && u != nullptr && ws != nullptr, fn, ": null pointer (h=",
              (const void *)h, ", x=", x, ", norm_w=", (const void *)norm_w, ", inv=", (const void *)inv, ", u=", u, ", ws=", ws, ")");
    SXB_CHECK(w->N == H * d, fn, ": W_up has ", w->N, " rows, expected H*d = ", H * d);
    SXB_CHECK(w->K >= kChunk && w->K <= kMaxRank && w->K % kChunk == 0, fn, ": W_up K (the rank r) = ", w->K, ", expected a multiple of ", kChunk,
              " up to ", kMaxRank);
    // inv: both kernels fetch a token's four of it as one 16-byte piece
    SXB_CHECK(aligned16(h) && aligned16(x) && aligned16(norm_w) && aligned16(inv) && aligned16(u) && reinterpret_cast<uintptr_t>(ws) % 256 == 0, fn,
              ": h, x, norm_w, inv and u must be 16-byte and the workspace 256-byte aligned");
    SXB_CHECK(w->K % 8 == 0, fn, ": r = ", w->K, " must be a multiple of 8");
    SXB_CHECK(apart(u, T * d * act_bytes(act), x, T * H * d * act_bytes(act)), fn, ": u overlaps the streams x");
    const int64_t r = w->K, Kp = up128(r), N = H * d;
    const UpWs L = up_ws(T, d, r, BITS, w->G);
    SXB_CHECK(ws_bytes >= L.total, fn, ": workspace of ", ws_bytes, " bytes, needs ", L.total);
    auto *base = static_cast<unsigned char *>(ws);
    auto st = static_cast<cudaStream_t>(stream);
    SxbQView rows{base + L.wq, reinterpret_cast<uint16_t *>(base + L.wscale), reinterpret_cast<uint16_t *>(base + L.wmin), N, Kp, w->G};

    const unsigned stage_blocks = (unsigned)std::min<int64_t>((T * (Kp / 8) + 255) / 256, (int64_t)sm_count() * 8);
    hc_stage_h_kernel<BITS><<<stage_blocks, 256, 0, st>>>(h, T, r, Kp, base + L.hs);
    SXB_CHECK_LAUNCH(fn, " staging h, T=", T, " r=", r);
    if (Kp <= kUpSteps * 128) {
        HcUpArgs a{base + L.hs, w->q, w->scale, w->minv, inv, norm_w, u, T, d, (int)r, (int)w->G, (int)(Kp / 128), nullptr, wait_limit_ns(), test_skip_slot()};
        if (int rc = library_status_words(fn, &a.status)) return rc;
        return act == SXB_ACT_F32 ? launch_hc_up<BITS, float>(fn, a, x, st) : launch_hc_up<BITS, uint16_t>(fn, a, x, st);
    }
    const int64_t vecs = N * Kp * BITS / 128;
    hc_unchunk_up_kernel<<<(unsigned)std::min<int64_t>((vecs + 255) / 256, (int64_t)sm_count() * 8), 256, 0, st>>>(
        w->q, w->scale, w->minv, d, r, Kp, w->G, BITS, reinterpret_cast<uint32_t *>(base + L.wq), reinterpret_cast<uint16_t *>(base + L.wscale),
        reinterpret_cast<uint16_t *>(base + L.wmin));
    SXB_CHECK_LAUNCH(fn, " un-chunking the weight, N=", N, " r=", r);
    return tc_hc_up<BITS>(fn, base + L.hs, &rows, x, inv, norm_w, u, T, d, act == SXB_ACT_F32, stream);
}

}  // namespace
}  // namespace sxb

using namespace sxb;

extern "C" {

size_t sxb_hc_mix_down_wmma_workspace_bytes(int64_t T, int64_t H, int64_t d, int64_t R, int bits, int64_t G) {
    if (T < 1 || T > 65535 || H != kStreams || d < 128 || d % 128 != 0 || R < 1 || R > kMaxRank + kStreams || (bits != 4 && bits != 8) ||
        (G != 32 && G != 64 && G != 128)) {
        last_error() = cat("hc_mix_down_wmma_workspace_bytes: T = ", T, ", H = ", H, ", d = ", d, ", R = ", R, ", bits = ", bits, ", G = ", G);
        return 0;
    }
    return down_ws(T, d, R, bits, G).total;
}
int sxb_hc_mix_down_wmma_q4(const void *x, const SxbQView *w, int64_t T, int64_t H, int64_t d, int64_t r, int inject, float eps, float *h,
                            float *w_in, float *inv, void *ws, size_t ws_bytes, int act, int inv_ready, sxb_stream_t stream) {
    return mix_down_tc<4>(x, w, T, H, d, r, inject, eps, h, w_in, inv, ws, ws_bytes, act, inv_ready, stream);
}
int sxb_hc_mix_down_wmma_q8(const void *x, const SxbQView *w, int64_t T, int64_t H, int64_t d, int64_t r, int inject, float eps, float *h,
                            float *w_in, float *inv, void *ws, size_t ws_bytes, int act, int inv_ready, sxb_stream_t stream) {
    return mix_down_tc<8>(x, w, T, H, d, r, inject, eps, h, w_in, inv, ws, ws_bytes, act, inv_ready, stream);
}

int sxb_hc_inject_inv(void *x, const float *w_in, const void *y, int64_t T, int64_t H, int64_t d, float eps, float *inv, int act,
                      sxb_stream_t stream) {
    const char *fn = "hc_inject_inv";
    SXB_CHECK(H == kStreams, fn, ": H = ", H, " streams, only ", kStreams, " is supported");
    SXB_CHECK(T >= 1 && T <= 0x7fffffff && d >= 1 && d <= (1 << 20), fn, ": T = ", T, ", d = ", d);
    SXB_CHECK(x != nullptr && w_in != nullptr && y != nullptr && inv != nullptr, fn, ": null pointer (x=", x, ", w_in=", (const void *)w_in,
              ", y=", y, ", inv=", (const void *)inv, ")");
    SXB_CHECK(std::isfinite(eps) && eps > 0.f, fn, ": eps must be finite and > 0, got ", eps);
    SXB_CHECK(act_ok(act), fn, ": unsupported activation dtype ", act);
    SXB_CHECK(apart(x, T * H * d * act_bytes(act), y, T * d * act_bytes(act)), fn, ": y overlaps the streams x");
    auto st = static_cast<cudaStream_t>(stream);
    if (act == SXB_ACT_F32)
        hc_inject_inv_kernel<float><<<(unsigned)T, 256, 0, st>>>(static_cast<float *>(x), w_in, static_cast<const float *>(y), d, eps, inv);
    else
        hc_inject_inv_kernel<uint16_t><<<(unsigned)T, 256, 0, st>>>(static_cast<uint16_t *>(x), w_in, static_cast<const uint16_t *>(y), d, eps, inv);
    SXB_CHECK_LAUNCH(fn, " ", act_name(act), " T=", T, " d=", d);
    return SXB_OK;
}

size_t sxb_hc_mix_up_wmma_workspace_bytes(int64_t T, int64_t H, int64_t d, int64_t r, int bits, int64_t G) {
    if (T < 1 || T > 65535 || H != kStreams || d < 128 || d % 128 != 0 || r < kChunk || r > kMaxRank || r % kChunk != 0 ||
        (bits != 4 && bits != 8) || (G != 32 && G != 64 && G != 128)) {
        last_error() = cat("hc_mix_up_wmma_workspace_bytes: T = ", T, ", H = ", H, ", d = ", d, ", r = ", r, ", bits = ", bits, ", G = ", G);
        return 0;
    }
    return up_ws(T, d, r, bits, G).total;
}
int sxb_hc_mix_up_wmma_q4(const float *h, const SxbQView *w_up, const void *x, const float *norm_w, const float *inv, int64_t T, int64_t H,
                          int64_t d, void *u, void *ws, size_t ws_bytes, int act, sxb_stream_t stream) {
    return mix_up_tc<4>(h, w_up, x, norm_w, inv, T, H, d, u, ws, ws_bytes, act, stream);
}
int sxb_hc_mix_up_wmma_q8(const float *h, const SxbQView *w_up, const void *x, const float *norm_w, const float *inv, int64_t T, int64_t H,
                          int64_t d, void *u, void *ws, size_t ws_bytes, int act, sxb_stream_t stream) {
    return mix_up_tc<8>(h, w_up, x, norm_w, inv, T, H, d, u, ws, ws_bytes, act, stream);
}

}  // extern "C"
