// The router-logits projection, the step right before the MoE router: logits [M, N] = x [M, K] * W^T (+ bias), FP32 out
// (runtime/qwen4exp.cpp:3149-3155; kernels/linear.hip:82-132 linear_bf16w, kernels/linear_wmma.hip:115-151
// linear_bf16w_wmma), and the residual add that closes a sublayer.
//
// Two forms, by regime:
//   * streaming (decode, a few dozen tokens): sixteen weight rows by a cluster of CTAs, each warp a part of their contraction against
//     sixteen tokens at a time, up to 64 a CTA, on the warp-level tensor-core path, FP32 weights as three BF16 planes split in registers;
//   * tcgen05 (prefill, thousands of tokens): a plain tensor-core GEMM with both operands staged by tensor copies.  The
//     weight is the reference's BF16 [N, K], or an FP32 one split once, at load time, into P BF16 "planes"
//     W = W1 + W2 (+ W3) (each plane the BF16 rounding of what the planes before it left over), so that the products
//     x * Wp are exact BF16 x BF16 products and their FP32 sum carries 16 (P = 2) or 24 (P = 3) bits of the weight.
//     The tokens sit on the MMA's M (128 a tile), the weight rows on its N, as many as suit the launch (gemm_shape); accumulators
//     double-buffered in tensor memory; warp 0 issues the copies, warp 1 the MMAs, warps 2-5 are the epilogue (bias add, FP32 store).
// Every device-side wait is bounded; one that runs out is recorded in the library's status words (see
// sxb_check_dense_status) and the kernel returns.

#include "experts.cuh"
#include "skinny_mma.cuh"
#include "tc_ptx.cuh"

#include <algorithm>
#include <cmath>

namespace sxb {
namespace {

// ---- streaming form ------------------------------------------------------------------------------------------

constexpr int kStreamSplit = 8, kStreamWarps = 8;  // CTAs of a cluster, and warps of a CTA, that share 16 weight rows
constexpr int kStreamEights = 8;                   // eights of tokens a CTA takes at most

// A lane's eight consecutive weights of a row: the BF16 planes they consist of.
template <typename TW>
struct Weights;
template <>
struct Weights<uint16_t> {
    static constexpr int kPlanes = 1, kAhead = 4;
    uint4 v;
    __device__ inline void load(const uint16_t *p) { v = __ldg(reinterpret_cast<const uint4 *>(p)); }
    __device__ inline void clear() { v = make_uint4(0u, 0u, 0u, 0u); }
    __device__ inline void planes(uint4 (&pl)[1]) const { pl[0] = v; }
};
template <>
struct Weights<float> {
    static constexpr int kPlanes = 3, kAhead = 2;
    float4 a, b;
    __device__ inline void load(const float *p) { a = __ldg(reinterpret_cast<const float4 *>(p)), b = __ldg(reinterpret_cast<const float4 *>(p) + 1); }
    __device__ inline void clear() { a = b = make_float4(0.f, 0.f, 0.f, 0.f); }
    __device__ inline void planes(uint4 (&pl)[3]) const {
        const float f[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
        split_planes(f, pl);
    }
};

// Whether a token's activations hold a NaN, and its dot with an FP32 weight row; by a whole warp.
__device__ __noinline__ bool row_has_nan(const uint16_t *x, int64_t K) {
    uint32_t nan = 0;
#pragma unroll 4
    for (int64_t e = threadIdx.x & 31; e < K / 8; e += 32) {
        const uint4 v = __ldg(reinterpret_cast<const uint4 *>(x) + e);
        const uint32_t xs[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) nan |= ((xs[i] & 0x7fffu) > 0x7f80u) | ((xs[i] & 0x7fff0000u) > 0x7f800000u);
    }
    return __any_sync(0xffffffffu, nan != 0);
}
__device__ __noinline__ float plain_dot(const uint16_t *x, const float *w, int64_t K) {
    double sum = 0.0;
#pragma unroll 2
    for (int64_t e = threadIdx.x & 31; e < K / 8; e += 32) {
        const uint4 v = __ldg(reinterpret_cast<const uint4 *>(x) + e);
        const float4 a = __ldg(reinterpret_cast<const float4 *>(w) + 2 * e), b = __ldg(reinterpret_cast<const float4 *>(w) + 2 * e + 1);
        const float f[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
        const uint32_t xs[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int i = 0; i < 8; ++i) sum += (double)f[i] * (double)__uint_as_float((i & 1) ? (xs[i / 2] & 0xffff0000u) : (xs[i / 2] << 16));
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
    return (float)sum;
}
// The sum of a lane whose result came out NaN, formed again by its whole converged warp.  An infinity times a plane that is zero, or split into planes, is NaN:
// the plain sum says what it is; a NaN among the token's activations, looked at once for all its rows, leaves nothing to say.  (One thread
// walking the contraction for each such result, as it stood here before: 128 x 513 x 4096 with NaN in every token 885 us, now 71; 32 without.)
__device__ inline float formed_again(bool bad, float sum, int64_t t, int64_t n, const uint16_t *x, const float *w, int64_t K) {
    const int lane = threadIdx.x & 31;
    int64_t seen = -1;
    bool nan = false;
    for (uint32_t todo = __ballot_sync(0xffffffffu, bad); todo != 0; todo &= todo - 1) {
        const int from = __ffs(todo) - 1;
        const int64_t t_of = __shfl_sync(0xffffffffu, t, from), n_of = __shfl_sync(0xffffffffu, n, from);
        if (t_of != seen) seen = t_of, nan = row_has_nan(x + t_of * K, K);
        if (nan) continue;
        const float plain = plain_dot(x + t_of * K, w + n_of * K, K);
        if (lane == from) sum = plain;
    }
    return sum;
}

// y[m, n] = sum_k x[m, k] * w[n, k] (+ bias[n]).  grid = (8 x tiles of 16 rows, groups of 8 NT tokens), clusters of eight CTAs along x:
// the warps of a cluster take the row's runs of 32 k by turns of a 64th each, ask for all their weights at once (K = 4096 FP32: two
// runs a warp), and the parts are added in order, across the warps in shared memory and then across the cluster.  FP32 weights go
// through the tensor cores as three BF16 planes (skinny_mma.cuh): exact products, each plane's sum apart, so that the arithmetic is
// no less than an FP32 multiply-add chain's (error against 64 bits 1.1e-7 -> 0.9e-7) and a token costs an MMA's column of it, not 16 dots
// a CTA whether they live or not.  513 x 4096 FP32, as a CUDA graph: 1 token 8.1 -> 4.1 us, 16 11.7 -> 4.5, 37 29 -> 6.1, 127 82 -> 14.
// Above sixteen tokens a warp keeps its weights, split, for one pair of eights after another: the same sums, FP32 8192 x 4096, 300 tokens 1230 -> 513 us
// (with groups of sixteen each was another CTA, which loaded and split them again).  What bounds it: the launch, one round trip to memory, the meeting of the parts.
template <typename TW, typename TOUT, int NT>
__global__ void __launch_bounds__(32 * kStreamWarps, 2)
    logits_stream_kernel(const uint16_t *__restrict__ x, const TW *__restrict__ w, const float *__restrict__ bias, int64_t M,
                         int64_t N, int64_t K, TOUT *__restrict__ y, int64_t ld) {
    behind_grid();
    constexpr int kTok = kMmaTokens * NT, kBatch = NT < 2 ? NT : 2, kAhead = Weights<TW>::kAhead, P = Weights<TW>::kPlanes;
    constexpr bool kKept = NT > kBatch;  // the split weights stay in registers for one batch of tokens after another
    __shared__ float part[kStreamWarps][kTok][kMmaRows + 1];
    __shared__ float cta_part[kTok][kMmaRows];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, c = lane & 3;
    const int rank = (int)cluster_rank();
    const int64_t n0 = (int64_t)(blockIdx.x / kStreamSplit) * kMmaRows;
    const TW *wa = w + min(n0 + g, N - 1) * K + 8 * c, *wb = w + min(n0 + g + 8, N - 1) * K + 8 * c;  // rows past the end: the last one
    const int64_t runs = (K + kMmaRun - 1) / kMmaRun, at = rank * kStreamWarps + warp, parts = kStreamSplit * kStreamWarps;
    const int64_t lo = runs * at / parts, hi = runs * (at + 1) / parts;
    for (int64_t t0 = (int64_t)blockIdx.y * kTok; t0 < M; t0 += (int64_t)gridDim.y * kTok) {
        const int live = (int)min((int64_t)NT, (M - t0 + kMmaTokens - 1) / kMmaTokens);  // eights of tokens in this group
        float acc[kBatch][4];  // of up to kBatch eights; more have their sums in `part` itself
#pragma unroll
        for (int b = 0; b < kBatch; ++b) acc[b][0] = acc[b][1] = acc[b][2] = acc[b][3] = 0.f;
        for (int64_t r0 = lo; (kKept && r0 == lo) || r0 < hi; r0 += kAhead) {  // a warp without runs: parts of zero
            Weights<TW> va[kAhead], vb[kAhead];
            bool in[kAhead];
#pragma unroll
            for (int e = 0; e < kAhead; ++e) {
                const int64_t k = (r0 + e) * kMmaRun;
                in[e] = r0 + e < hi && k + 8 * c < K;
                if (in[e]) va[e].load(wa + k), vb[e].load(wb + k);
                else va[e].clear(), vb[e].clear();
            }
            uint4 xv[kBatch][kAhead], pa[kAhead][P], pb[kAhead][P];
            auto fetch = [&](int nt0) {
#pragma unroll
                for (int b = 0; b < kBatch; ++b)
#pragma unroll
                    for (int e = 0; e < kAhead; ++e) {
                        const int64_t t = t0 + (nt0 + b) * kMmaTokens + g;
                        xv[b][e] = in[e] && t < M ? __ldg(reinterpret_cast<const uint4 *>(x + t * K + (r0 + e) * kMmaRun + 8 * c)) : make_uint4(0u, 0u, 0u, 0u);
                    }
            };
            fetch(0);
            if constexpr (kKept) {
#pragma unroll
                for (int e = 0; e < kAhead; ++e) va[e].planes(pa[e]), vb[e].planes(pb[e]);
            }
#pragma unroll 1
            for (int nt0 = 0; nt0 < (kKept ? live : 1); nt0 += kBatch) {
                float dot[kBatch][P][4];
#pragma unroll
                for (int b = 0; b < kBatch; ++b)
#pragma unroll
                    for (int p = 0; p < P; ++p) dot[b][p][0] = dot[b][p][1] = dot[b][p][2] = dot[b][p][3] = 0.f;
#pragma unroll
                for (int e = 0; e < kAhead; ++e) {
                    if (r0 + e >= hi) break;
                    if constexpr (!kKept) va[e].planes(pa[e]), vb[e].planes(pb[e]);
#pragma unroll
                    for (int p = 0; p < P; ++p)
#pragma unroll
                        for (int b = 0; b < kBatch; ++b) mma_run(dot[b][p], pa[e][p], pb[e][p], xv[b][e]);
                }
                if (kKept && nt0 + kBatch < live) fetch(nt0 + kBatch);
#pragma unroll
                for (int b = 0; b < kBatch; ++b)
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        float sum = dot[b][P - 1][i];
#pragma unroll
                        for (int p = P - 2; p >= 0; --p) sum += dot[b][p][i];
                        if constexpr (kKept) {
                            float &to = part[warp][(nt0 + b) * kMmaTokens + 2 * c + (i & 1)][g + 8 * (i >> 1)];
                            to = r0 == lo ? sum : to + sum;
                        } else {
                            acc[b][i] += sum;
                        }
                    }
            }
        }
        if constexpr (!kKept) {
#pragma unroll
            for (int b = 0; b < kBatch; ++b)
#pragma unroll
                for (int i = 0; i < 4; ++i) part[warp][b * kMmaTokens + 2 * c + (i & 1)][g + 8 * (i >> 1)] = acc[b][i];
        }
        __syncthreads();
        for (int i = threadIdx.x; i < (kKept ? live * kMmaTokens : kTok) * kMmaRows; i += 32 * kStreamWarps) {
            float sum = 0.f;
#pragma unroll
            for (int v = 0; v < kStreamWarps; ++v) sum += part[v][i / kMmaRows][i % kMmaRows];
            cta_part[i / kMmaRows][i % kMmaRows] = sum;
        }
        cluster_sync();
        // a CTA finishes every eighth token of the group
        if (warp < (NT * kMmaRows + 31) / 32) {
            const int tt = rank + kStreamSplit * ((int)threadIdx.x / kMmaRows), row = lane % kMmaRows;
            const int64_t n = n0 + row, t = t0 + tt;
            const bool out = threadIdx.x < NT * kMmaRows && n < N && t < M;
            float sum = 0.f;
            if (out) {
                float v[kStreamSplit];
#pragma unroll
                for (int p = 0; p < kStreamSplit; ++p) v[p] = ld_cluster(&cta_part[tt][row], p);
#pragma unroll
                for (int p = 0; p < kStreamSplit; ++p) sum += v[p];
            }
            if constexpr (P > 1) sum = formed_again(out && isnan(sum), sum, t, n, x, w, K);
            if (out) store_from_f32(y, t * ld + n, sum + (bias != nullptr ? bias[n] : 0.f));
        }
        cluster_sync();  // the parts have been read: the next group may overwrite them, or the CTA leave
    }
}

// x_out = bf16(x + y): the residual add that closes the sublayer (the reference injects into its four residual streams
// with hc_inject, kernels/hc.hpp:52-54; this is the single-stream case with weight 1).  Eight elements a thread.
template <typename TY>
__global__ void __launch_bounds__(256) residual_add_kernel(const uint4 *__restrict__ x, const TY *__restrict__ y, uint4 *__restrict__ out,
                                                           int64_t chunks) {
    behind_grid();
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < chunks; i += (int64_t)gridDim.x * blockDim.x) {
        const uint4 xv = x[i];
        const uint32_t u[4] = {xv.x, xv.y, xv.z, xv.w};
        float yv[8];
        if constexpr (sizeof(TY) == 4) {
            const float4 a = reinterpret_cast<const float4 *>(y)[2 * i], b = reinterpret_cast<const float4 *>(y)[2 * i + 1];
            yv[0] = a.x, yv[1] = a.y, yv[2] = a.z, yv[3] = a.w, yv[4] = b.x, yv[5] = b.y, yv[6] = b.z, yv[7] = b.w;
        } else {
            const uint4 a = reinterpret_cast<const uint4 *>(y)[i];
            const uint32_t v[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
            for (int j = 0; j < 4; ++j) yv[2 * j] = __uint_as_float(v[j] << 16), yv[2 * j + 1] = __uint_as_float(v[j] & 0xffff0000u);
        }
        uint32_t o[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const uint32_t lo = f32_to_bf16_bits(__uint_as_float(u[j] << 16) + yv[2 * j]);
            const uint32_t hi = f32_to_bf16_bits(__uint_as_float(u[j] & 0xffff0000u) + yv[2 * j + 1]);
            o[j] = lo | (hi << 16);
        }
        out[i] = make_uint4(o[0], o[1], o[2], o[3]);
    }
}

// ---- tcgen05 form ----------------------------------------------------------------------------------------------

constexpr int kGemmThreads = 192;      // warp 0 copies, warp 1 MMA issue, warps 2-5 epilogue
constexpr int kTile = 128;             // tokens of a tile (MMA M); the planes' rows are padded to as many
constexpr int kGemmBK = 64;            // k per stage: one 128-byte swizzle line of BF16
constexpr int kXBytes = kTile * kGemmBK * 2;  // 16 KB: a stage's activations; a plane's part is 128 bytes a weight row
constexpr int kMaxStages = 8;
constexpr int kMaxPlanes = 3;
constexpr int kMaxRows = 256;          // weight rows of a tile (MMA N), a multiple of 16: two accumulators fill tensor memory
constexpr int kGemmTmemCols = 512;
constexpr int kEpiCols = 16, kEpiPitch = kEpiCols + 1;  // the epilogue's transpose: 32 tokens x 16 rows a warp
constexpr int kEpiBytes = 4 * 32 * kEpiPitch * 4;
constexpr size_t kGemmSmem = 230400;   // of 232448 bytes; the rest is for the barriers

struct GemmArgs {
    const float *bias;
    float *logits;
    int64_t M, N, Npad, K, ld;
    int planes, stages, rows;  // rows: of a tile
    uint32_t *status;
    unsigned long long wait_limit_ns;
    int test_skip_slot;  // >= 0: CTA 0 never issues the copies of that stage fill, so that a wait runs out (tests only)
};

// Instruction descriptor for kind::f16 with BF16 operands: D FP32 (bits [4,6) = 1), A and B BF16 (bits [7,10) and
// [10,13) = 1), both K-major, N >> 3 at bits [17,23), M >> 4 at bits [24,29).
__device__ inline uint32_t instr_desc_bf16(int n_cols) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n_cols >> 3) << 17) | ((128u >> 4) << 24);
}
// D[tmem] (+)= A[smem] * B[smem] over 64 k, both 128-byte-swizzled: four MMAs, issued by the lane with leader = 1 of a whole warp under uniform
// control flow, so that descriptors stay in uniform registers.
__device__ inline void tc_kblock_ss(uint32_t leader, uint32_t d, uint32_t a_lo, uint32_t b_lo, uint32_t hi, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p, q, one;\n\t.reg .b32 x1, x2, x3, y1, y2, y3;\n\t.reg .b64 a0, a1, a2, a3, b0, b1, b2, b3;\n\t"
        "setp.ne.b32 p, %5, 0;\n\tsetp.ne.b32 q, %6, 0;\n\tsetp.eq.b32 one, 0, 0;\n\t"
        "add.u32 x1, %1, 2;\n\tadd.u32 x2, %1, 4;\n\tadd.u32 x3, %1, 6;\n\tadd.u32 y1, %2, 2;\n\tadd.u32 y2, %2, 4;\n\tadd.u32 y3, %2, 6;\n\t"
        "mov.b64 a0, {%1, %3};\n\tmov.b64 a1, {x1, %3};\n\tmov.b64 a2, {x2, %3};\n\tmov.b64 a3, {x3, %3};\n\t"
        "mov.b64 b0, {%2, %3};\n\tmov.b64 b1, {y1, %3};\n\tmov.b64 b2, {y2, %3};\n\tmov.b64 b3, {y3, %3};\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], a0, b0, %4, p;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], a1, b1, %4, one;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], a2, b2, %4, one;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], a3, b3, %4, one;\n\t}" ::"r"(d),
        "r"(a_lo), "r"(b_lo), "r"(hi), "r"(idesc), "r"(accumulate), "r"(leader)
        : "memory");
}
// A place in a ring of n barriers and the parity of the phase it is in.
struct RingTurn {
    int at;
    uint32_t phase;
    __device__ inline void advance(int n) {
        if (++at == n) at = 0, phase ^= 1u;
    }
};

__global__ void __launch_bounds__(kGemmThreads, 1)
    logits_gemm_kernel(const GemmArgs a, const __grid_constant__ CUtensorMap xmap, const __grid_constant__ CUtensorMap wmap) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char *smem = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    __shared__ uint64_t full_bar[kMaxStages], empty_bar[kMaxStages], acc_full[2], acc_empty[2], drain_bar;
    __shared__ uint32_t tmem_base_smem;
    __shared__ int abort_flag;

    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const int n_kb = (int)(a.K / kGemmBK), n_rb = (int)((a.N + a.rows - 1) / a.rows), n_tt = (int)((a.M + kTile - 1) / kTile);
    const int64_t n_items = (int64_t)n_rb * n_tt;
    const int plane_bytes = a.rows * kGemmBK * 2, stage_bytes = kXBytes + a.planes * plane_bytes;
    volatile int *abort_v = &abort_flag;

    if (threadIdx.x == 0) {
        for (int s = 0; s < kMaxStages; ++s) mbar_init(&full_bar[s], 1), mbar_init(&empty_bar[s], 1);
        for (int b = 0; b < 2; ++b) mbar_init(&acc_full[b], 1), mbar_init(&acc_empty[b], 4);
        mbar_init(&drain_bar, 1);
        abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_smem)), "r"(kGemmTmemCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = tmem_base_smem;

    auto raise_abort = [&](int64_t item, int role) {
        if (atomicExch(&abort_flag, 1) == 0 && atomicCAS(&a.status[0], 0u, 2u) == 0u) {
            a.status[1] = (uint32_t)item;
            a.status[2] = (uint32_t)role;
        }
    };

    uint32_t issued = 0;  // stages filled by this thread (the copy thread only)
    if (warp == 0) {
        // ===================== copies: one thread, as far ahead as free stages allow =====================
        if (lane == 0) {
            RingTurn turn{0, 1u};  // the phase before the first leaves every stage free
            for (int64_t item = blockIdx.x; item < n_items && !*abort_v; item += gridDim.x) {
                const int tile = (int)(item / n_rb), rb = (int)(item % n_rb);
                for (int kb = 0; kb < n_kb; ++kb, ++issued, turn.advance(a.stages)) {
                    if (!mbar_wait(&empty_bar[turn.at], turn.phase, abort_v, a.wait_limit_ns)) {
                        raise_abort(item, 5);
                        break;
                    }
                    if (blockIdx.x == 0 && (int)issued == a.test_skip_slot) continue;
                    const uint32_t dst = smem_u32(smem + turn.at * stage_bytes);
                    mbar_expect_tx(&full_bar[turn.at], (uint32_t)stage_bytes);
                    tma_load_2d(dst, &xmap, kb * kGemmBK, tile * kTile, &full_bar[turn.at]);
                    for (int p = 0; p < a.planes; ++p)
                        tma_load_2d(dst + kXBytes + p * plane_bytes, &wmap, kb * kGemmBK, (int)(p * a.Npad) + rb * a.rows, &full_bar[turn.at]);
                }
            }
        }
    } else if (warp == 1) {
        // ===================== MMA issue =====================
        const uint32_t leader = elect_one() ? 1u : 0u, idesc = instr_desc_bf16(a.rows);
        const uint64_t desc0 = smem_desc(smem_u32(smem));
        const uint32_t hi = (uint32_t)(desc0 >> 32), plane_lo = (uint32_t)plane_bytes / 16, stage_lo = (uint32_t)stage_bytes / 16;
        uint32_t lo = (uint32_t)desc0, acc_count = 0;
        RingTurn turn{0, 0u};
        bool ok = true;
        for (int64_t item = blockIdx.x; item < n_items && ok; item += gridDim.x, ++acc_count) {
            const uint32_t buf = acc_count & 1u;
            ok = __all_sync(0xffffffffu, mbar_wait(&acc_empty[buf], ((acc_count >> 1) & 1u) ^ 1u, abort_v, a.wait_limit_ns));
            if (!ok) {
                if (leader) raise_abort(item, 2);
                break;
            }
            tc_fence_after();
            const uint32_t d = tmem_base + buf * (uint32_t)kMaxRows;
            bool ready = false;
            for (int kb = 0; kb < n_kb; ++kb) {
                if (!__all_sync(0xffffffffu, ready)) {
                    ok = __all_sync(0xffffffffu, mbar_wait(&full_bar[turn.at], turn.phase, abort_v, a.wait_limit_ns));
                    if (!ok) {
                        if (leader) raise_abort(item, 3);
                        break;
                    }
                }
                tc_fence_after();
                uint64_t *const done = &empty_bar[turn.at];
                const uint32_t b_lo = lo + kXBytes / 16;
                const uint32_t lo_nxt = turn.at + 1 == a.stages ? (uint32_t)desc0 : lo + stage_lo;
                turn.advance(a.stages);
                ready = mbar_test(&full_bar[turn.at], turn.phase);  // asked for under the MMAs
                for (int p = 0; p < a.planes; ++p) tc_kblock_ss(leader, d, lo, b_lo + p * plane_lo, hi, idesc, (kb | p) != 0);
                tc_commit_if(leader, done);  // the stage is free once these MMAs have read it
                lo = lo_nxt;
            }
            if (ok) tc_commit_if(leader, &acc_full[buf]);
        }
        // every MMA of this CTA has completed before tensor memory is released (not given up while aborting)
        tc_commit_if(leader, &drain_bar);
        mbar_wait(&drain_bar, 0u, nullptr, a.wait_limit_ns);
        __syncwarp();
    } else {
        // ===================== epilogue =====================
        // Lane = token: sixteen weight rows at a time go through shared memory, so that a store writes 64 neighbouring bytes of two tokens.
        const int quad = warp & 3;  // the tensor-memory lanes a warp may read: 32 (warp % 4) ..
        float *turned = reinterpret_cast<float *>(smem + a.stages * stage_bytes) + (warp - 2) * 32 * kEpiPitch;
        uint32_t acc_count = 0;
        for (int64_t item = blockIdx.x; item < n_items && !*abort_v; item += gridDim.x, ++acc_count) {
            const int tile = (int)(item / n_rb), rb = (int)(item % n_rb);
            const uint32_t buf = acc_count & 1u;
            if (lane == 0 && !mbar_wait(&acc_full[buf], (acc_count >> 1) & 1u, abort_v, a.wait_limit_ns)) raise_abort(item, 4);
            __syncwarp();
            if (*abort_v) break;
            tc_fence_after();
            const uint32_t taddr = tmem_base + ((uint32_t)(quad * 32) << 16) + buf * (uint32_t)kMaxRows;
            const int64_t t0 = (int64_t)tile * kTile + quad * 32, e0 = (int64_t)rb * a.rows;
            for (int c0 = 0; c0 < a.rows; c0 += kEpiCols) {
                float v[16];
                tc_ld16(taddr + (uint32_t)c0, v);
                if (c0 + kEpiCols == a.rows) {  // the last columns are in registers: the accumulator may be overwritten
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&acc_empty[buf]);
                }
#pragma unroll
                for (int c = 0; c < kEpiCols; ++c) turned[lane * kEpiPitch + c] = v[c];
                __syncwarp();
                const int64_t e = e0 + c0 + (lane & 15);
                const float b = (e < a.N && a.bias) ? a.bias[e] : 0.f;
#pragma unroll
                for (int t = 0; t < 32; t += 2) {
                    const int64_t tok = t0 + t + (lane >> 4);
                    if (e < a.N && tok < a.M) a.logits[tok * a.ld + e] = turned[(t + (lane >> 4)) * kEpiPitch + (lane & 15)] + b;
                }
                __syncwarp();
            }
        }
    }

    // an aborting CTA waits (bounded) for the copies it issued before its shared memory can go to another CTA
    if (*abort_v && issued > 0)
        for (int s = 0; s < a.stages; ++s) {
            if (issued <= (uint32_t)s) continue;
            const uint32_t last = ((issued - 1 - (uint32_t)s) / a.stages) * a.stages + (uint32_t)s;
            if (blockIdx.x == 0 && (int)last == a.test_skip_slot) continue;  // the test hook's fill never comes
            mbar_wait(&full_bar[s], (last / a.stages) & 1u, nullptr, 1000000ull);
        }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kGemmTmemCols) : "memory");
    }
}

// The weight rows of a tile: those for which the launch's estimate is least.  In SM cycles a k-block takes the longest of its copies (50 bytes a
// cycle and SM, measured with every SM at it), its MMAs (66 at least: reading 4 KB of activations from shared memory bounds them) and what one stage
// less than there are hides of a copy's latency; an item, its epilogue.  Few tokens want narrow tiles, so that the k-blocks' chain of MMAs is
// shared by the machine (128 weight rows a tile, the weights on the M side: 10 CTAs at 150 tokens); many want wide ones, for less traffic.
// 513 x 4096 FP32, the sums' order and bits as before: 150 tokens 48 -> 29 us (16 rows), 777 48 -> 30 (32), 1200 48 -> 32 (48), 4096 91 -> 52 (144),
// 16384 230 -> 227.  What bounds it: the MMAs' operand reads, from 4096 tokens on the copies.
struct GemmShape {
    int rows, stages;
};
GemmShape gemm_shape(int64_t M, int64_t N, int64_t n_kb, int planes, int sms) {
    GemmShape best{16, 2};
    double least = 0;
    for (int rows = 16; rows <= kMaxRows && (rows == 16 || rows < N + 16); rows += 16) {
        const int bytes = kXBytes + planes * rows * kGemmBK * 2;
        const int stages = (int)std::min<size_t>(kMaxStages, (kGemmSmem - 1024 - kEpiBytes) / bytes);
        if (stages < 2) break;
        const double copies = bytes / 50.0, mmas = planes * 4 * std::max(66.0, 32 + rows / 4.0), latency = (1500 + mmas) / stages;
        const double items = (double)((M + kTile - 1) / kTile) * (double)((N + rows - 1) / rows);
        const double cost = std::ceil(items / sms) * ((double)n_kb * std::max(copies, std::max(mmas, latency)) + 20.0 * rows + 3000);
        if (least == 0 || cost <= least) least = cost, best = GemmShape{rows, stages};
    }
    return best;
}

// W [N, K] (FP32 or BF16) -> P BF16 planes [P][Npad][K]: plane p holds the BF16 rounding of what the planes before it left
// of the weight; rows N .. Npad - 1 are zero.  With a BF16 weight one plane is the weight itself.
template <typename TW>
__global__ void __launch_bounds__(256) split_planes_kernel(const TW *__restrict__ w, int64_t N, int64_t Npad, int64_t K, int planes,
                                                           uint16_t *__restrict__ out) {
    const int64_t total = Npad * K;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        float r = i / K < N ? load_as_f32(w, i) : 0.f;
        for (int p = 0; p < planes; ++p) {
            const uint16_t b = f32_to_bf16_bits(r);
            out[(int64_t)p * total + i] = b;
            r -= bf16_bits_to_f32(b);  // exact: the difference of an FP32 value and its BF16 rounding fits FP32
        }
    }
}

int64_t pad_rows(int64_t N) { return (N + kTile - 1) / kTile * kTile; }

int check_proj(const char *fn, const void *x, const void *w, const void *y, int64_t M, int64_t N, int64_t K) {
    SXB_CHECK(x != nullptr && w != nullptr && y != nullptr, fn, ": null pointer (x=", x, ", w=", w, ", y=", y, ")");
    SXB_CHECK(M >= 1 && N >= 1 && N <= (1 << 24) && K >= 8 && K % 8 == 0 && K <= (1 << 24), fn, ": M = ", M, ", N = ", N, ", K = ", K,
              " (K a multiple of 8)");
    SXB_CHECK(aligned16(x) && aligned16(w), fn, ": x and w must be 16-byte aligned");
    return SXB_OK;
}

template <typename TOUT>
int launch_stream_logits(const char *fn, const void *x, const void *w, int w_act, const float *bias, int64_t M, int64_t N, int64_t K,
                         TOUT *y, int64_t ld, cudaStream_t st) {
    // Eights of tokens a CTA takes: two while the launch then fits the machine at two CTAs an SM (65 rows, 37 tokens: 3.6 us against 4.6), else eight,
    // for which the weights are loaded and split once (513 rows, 17 / 37 / 127 tokens: 8.0 -> 5.2, 12.1 -> 6.1, 30.6 -> 14).
    const int64_t by_row = (N + kMmaRows - 1) / kMmaRows * kStreamSplit;
    const int NT = M <= kMmaTokens ? 1 : M <= 2 * kMmaTokens || by_row * ((M + 2 * kMmaTokens - 1) / (2 * kMmaTokens)) <= 2 * sm_count() ? 2 : kStreamEights;
    const dim3 grid((unsigned)by_row, (unsigned)std::min<int64_t>((M + NT * kMmaTokens - 1) / (NT * kMmaTokens), 65535));
    auto xb = static_cast<const uint16_t *>(x);
    auto launch = [&](auto kern, auto *wt) { return launch_behind(kern, grid, dim3(32 * kStreamWarps), 0, st, kStreamSplit, xb, wt, bias, M, N, K, y, ld); };
    cudaError_t e;
    if (w_act == SXB_ACT_F32) {
        auto wt = static_cast<const float *>(w);
        e = NT == 1   ? launch(logits_stream_kernel<float, TOUT, 1>, wt)
            : NT == 2 ? launch(logits_stream_kernel<float, TOUT, 2>, wt)
                      : launch(logits_stream_kernel<float, TOUT, kStreamEights>, wt);
    } else {
        auto wt = static_cast<const uint16_t *>(w);
        e = NT == 1   ? launch(logits_stream_kernel<uint16_t, TOUT, 1>, wt)
            : NT == 2 ? launch(logits_stream_kernel<uint16_t, TOUT, 2>, wt)
                      : launch(logits_stream_kernel<uint16_t, TOUT, kStreamEights>, wt);
    }
    SXB_CUDA(e, fn, ": launching M=", M, " N=", N, " K=", K);
    SXB_CHECK_LAUNCH(fn, " M=", M, " N=", N, " K=", K);
    return SXB_OK;
}

}  // namespace
}  // namespace sxb

using namespace sxb;

extern "C" {

int sxb_linear_bf16w(const void *x, const uint16_t *w, void *y, int64_t M, int64_t N, int64_t K, int act, int out_act,
                     sxb_stream_t stream) {
    const char *fn = "linear_bf16w";
    if (int rc = check_proj(fn, x, w, y, M, N, K)) return rc;
    SXB_CHECK(act == SXB_ACT_BF16, fn, ": BF16 activations only, got ", act);
    SXB_CHECK(out_act == SXB_ACT_BF16 || out_act == SXB_ACT_F32, fn, ": output dtype ", out_act, " unsupported (BF16, or F32)");
    SXB_CHECK(apart(x, M * K * 2, y, M * N * act_bytes(out_act)), fn, ": y overlaps x");
    auto st = static_cast<cudaStream_t>(stream);
    return out_act == SXB_ACT_F32 ? launch_stream_logits<float>(fn, x, w, SXB_ACT_BF16, nullptr, M, N, K, (float *)y, N, st)
                                  : launch_stream_logits<uint16_t>(fn, x, w, SXB_ACT_BF16, nullptr, M, N, K, (uint16_t *)y, N, st);
}

int sxb_router_logits(const void *x, const void *w, int w_act, const float *bias, int64_t M, int64_t N, int64_t K, float *logits,
                      int64_t ld, sxb_stream_t stream) {
    const char *fn = "router_logits";
    if (int rc = check_proj(fn, x, w, logits, M, N, K)) return rc;
    SXB_CHECK(w_act == SXB_ACT_F32 || w_act == SXB_ACT_BF16, fn, ": weight dtype ", w_act, " unsupported (F32 or BF16)");
    SXB_CHECK(ld >= N, fn, ": logits row stride ld = ", ld, " < N = ", N);
    SXB_CHECK(apart(x, M * K * 2, logits, M * ld * 4), fn, ": logits overlap x");
    return launch_stream_logits<float>(fn, x, w, w_act, bias, M, N, K, logits, ld, static_cast<cudaStream_t>(stream));
}

size_t sxb_router_planes_bytes(int64_t N, int64_t K, int planes) {
    if (!(N >= 1 && K >= 1 && planes >= 1 && planes <= kMaxPlanes)) {
        fail_check(SXB_FILE_, __LINE__, __func__, "N >= 1 && K >= 1 && 1 <= planes <= 3",
                   cat("router_planes_bytes: N = ", N, ", K = ", K, ", planes = ", planes));
        return 0;
    }
    return (size_t)planes * (size_t)pad_rows(N) * (size_t)K * 2;
}

int sxb_router_prepare(const void *w, int w_act, int64_t N, int64_t K, int planes, void *planes_out, sxb_stream_t stream) {
    const char *fn = "router_prepare";
    SXB_CHECK(w != nullptr && planes_out != nullptr, fn, ": null pointer");
    SXB_CHECK(w_act == SXB_ACT_F32 || w_act == SXB_ACT_BF16, fn, ": weight dtype ", w_act, " unsupported (F32 or BF16)");
    SXB_CHECK(planes >= 1 && planes <= kMaxPlanes, fn, ": planes = ", planes, ", expected 1..", kMaxPlanes);
    SXB_CHECK(N >= 1 && K >= 64 && K % 64 == 0 && K <= (1 << 24), fn, ": N = ", N, ", K = ", K, " (K a multiple of 64)");
    SXB_CHECK(aligned16(planes_out), fn, ": the planes must be 16-byte aligned");
    const int64_t Npad = pad_rows(N);
    const unsigned blocks = (unsigned)std::min<int64_t>((Npad * K + 255) / 256, (int64_t)sm_count() * 8);
    auto st = static_cast<cudaStream_t>(stream);
    if (w_act == SXB_ACT_F32) split_planes_kernel<float><<<blocks, 256, 0, st>>>((const float *)w, N, Npad, K, planes, (uint16_t *)planes_out);
    else split_planes_kernel<uint16_t><<<blocks, 256, 0, st>>>((const uint16_t *)w, N, Npad, K, planes, (uint16_t *)planes_out);
    SXB_CHECK_LAUNCH(fn, " N=", N, " K=", K, " planes=", planes);
    return SXB_OK;
}

int sxb_router_logits_wmma(const void *x, const void *planes_in, int planes, const float *bias, int64_t M, int64_t N, int64_t K,
                           float *logits, int64_t ld, sxb_stream_t stream) {
    const char *fn = "router_logits_wmma";
    if (int rc = check_proj(fn, x, planes_in, logits, M, N, K)) return rc;
    SXB_CHECK(planes >= 1 && planes <= kMaxPlanes, fn, ": planes = ", planes, ", expected 1..", kMaxPlanes);
    SXB_CHECK(K % kGemmBK == 0, fn, ": K = ", K, " must be a multiple of ", kGemmBK);
    SXB_CHECK(M <= (1 << 24), fn, ": M = ", M, " tokens, expected <= 2^24");
    SXB_CHECK(ld >= N, fn, ": logits row stride ld = ", ld, " < N = ", N);
    SXB_CHECK(apart(x, M * K * 2, logits, M * ld * 4), fn, ": logits overlap x");
    GemmArgs a{};
    a.bias = bias, a.logits = logits, a.M = M, a.N = N, a.Npad = pad_rows(N), a.K = K, a.ld = ld, a.planes = planes;
    const GemmShape shape = gemm_shape(M, N, K / kGemmBK, planes, sm_count());
    a.rows = shape.rows, a.stages = shape.stages;
    a.wait_limit_ns = wait_limit_ns(), a.test_skip_slot = test_skip_slot();
    if (int rc = library_status_words(fn, &a.status)) return rc;
    CUtensorMap xmap, wmap;
    if (int rc = tensor_map_2d(fn, x, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (uint64_t)K, (uint64_t)M, (uint64_t)K * 2, kGemmBK, kTile,
                               CU_TENSOR_MAP_SWIZZLE_128B, &xmap))
        return rc;
    // one plane may be the raw BF16 weight [N, K] itself: its rows past N read as zero instead of being stored as zeros
    if (int rc = tensor_map_2d(fn, planes_in, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (uint64_t)K, (uint64_t)(planes == 1 ? N : planes * a.Npad), (uint64_t)K * 2,
                               kGemmBK, (uint32_t)a.rows, CU_TENSOR_MAP_SWIZZLE_128B, &wmap))
        return rc;
    const size_t smem = (size_t)a.stages * (kXBytes + planes * a.rows * kGemmBK * 2) + kEpiBytes + 1024;
    // the function's limit is one for all threads of the process: always the largest, not this call's
    SXB_CUDA(cudaFuncSetAttribute(logits_gemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kGemmSmem), fn, ": reserving shared memory");
    const int64_t items = ((N + a.rows - 1) / a.rows) * ((M + kTile - 1) / kTile);
    const unsigned grid = (unsigned)std::min<int64_t>(items, sm_count());
    logits_gemm_kernel<<<grid, kGemmThreads, smem, static_cast<cudaStream_t>(stream)>>>(a, xmap, wmap);
    SXB_CHECK_LAUNCH(fn, " M=", M, " N=", N, " K=", K, " planes=", planes);
    return SXB_OK;
}

int sxb_residual_add(const void *x, const void *y, int y_act, void *out, int64_t n, sxb_stream_t stream) {
    const char *fn = "residual_add";
    SXB_CHECK(x != nullptr && y != nullptr && out != nullptr, fn, ": null pointer");
    SXB_CHECK(n >= 8 && n % 8 == 0, fn, ": n = ", n, " elements, expected a positive multiple of 8");
    SXB_CHECK(y_act == SXB_ACT_F32 || y_act == SXB_ACT_BF16, fn, ": dtype of y ", y_act, " unsupported (F32 or BF16)");
    SXB_CHECK(aligned16(x) && aligned16(y) && aligned16(out), fn, ": x, y and out must be 16-byte aligned");
    SXB_CHECK(apart(out, n * 2, y, n * act_bytes(y_act)), fn, ": out overlaps y");
    const int64_t chunks = n / 8;
    const unsigned blocks = (unsigned)std::min<int64_t>((chunks + 255) / 256, (int64_t)sm_count() * 8);
    auto st = static_cast<cudaStream_t>(stream);
    if (y_act == SXB_ACT_F32) launch_behind(residual_add_kernel<float>, blocks, 256, 0, st, 1, (const uint4 *)x, (const float *)y, (uint4 *)out, chunks);
    else launch_behind(residual_add_kernel<uint16_t>, blocks, 256, 0, st, 1, (const uint4 *)x, (const uint16_t *)y, (uint4 *)out, chunks);
    SXB_CHECK_LAUNCH(fn, " n=", n);
    return SXB_OK;
}

}  // extern "C"
