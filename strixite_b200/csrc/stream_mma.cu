// Streaming expert kernels, and dense ones of Q4 weights (Q8: dense_mma.cu), for the HBM-bound regime (decode and small ragged batches;
// also the exact-product path at any size).  C ABI twins of the launchers in kernels/linear_q4.hpp, kernels/linear_q8.hpp and of the
// MoeMath::F32 / WmmaBf16 forms of kernels/moe_grouped.hpp.
//
// What the reference does (kernels/linear_q4.hip:175-199): a wave walks one weight row, every lane takes 32 codes per
// 16-byte load and forms s * sum(x*q) + m * sum(x) per chunk with one FMA per weight, then a wave-shuffle reduction.
// On B200 that form is issue-bound long before HBM is: at 6.5 TB/s an SM receives ~46 codes per clock, and one FMA plus
// the nibble -> float conversion per code and per token already exceeds the 128 FP32 lanes.
//
// This kernel keeps the same arithmetic - exact products of BF16 activations with the integer codes, FP32 sums, scale
// and min applied per group in FP32 - but lets the tensor cores form the products:
//   * a warp owns 16 weight rows; lane (g = lane / 4, c = lane % 4) streams rows g and g + 8 with one 16-byte
//     `ld.global.nc` each per step, the four lanes of a quad covering 64 contiguous bytes of a row, which for the
//     served formats (Q4 G = 128, Q8 G = 64) is exactly one quantization group;
//   * codes become F16 pairs in registers: a code n in the low mantissa bits of an F16 whose exponent field is zero IS the
//     subnormal n * 2^-24 (n * 2^-20 four bits further up), so eight nibbles take a shift and four masks of the half-rate
//     integer pipe, four bytes two byte permutes, and a packed multiply by a power of two makes a pair of normal numbers.
//     (With BF16 operands, whose seven mantissa bits hold a nibble in one place only, a pair took a shift and a lop3, and a
//     Q8 code the pairs of its two nibbles.)  The activations come as F16 too, each token's times the power of two that takes
//     its largest magnitude to 2^15 .. 2^16: everything down to 2^-29 of the largest is a normal F16, BF16's eight significant
//     bits exactly.  What is smaller is rounded at 2^-40 of the largest, which shows where the large values meet weights of exactly
//     zero (code and min) and the small ones are the dot.  Q8 keeps those: they are left out of the F16 operand and added to the
//     finished dots in FP32, and a token with more than kLowMax of them takes BF16 operands, codes and all (rows_dot_wide).  Q4
//     has no such form (it costs 1.5 to 3 % of a decode step): it rounds at 2^-40, where its codes as BF16 pairs 16 + n, with 16
//     sum(x) taken off again, lost what lay below 2^-24;
//   * the activations of the tile's <= 8 tokens sit in shared memory already permuted into `mma.m16n8k16` B-fragment
//     order, so a lane fetches its fragments with conflict-free 16-byte loads; k is permuted consistently on both
//     operands, which a dot product does not notice;
//   * per step: D = sum over the quad's codes of q * x on the tensor cores (exact products, FP32 sums), then
//     acc += s * D + m * sum(x) in FP32; the token's power of two comes off the finished dot.
// Work is cut into units of 16 rows x one tile of <= 8 tokens of one expert; CTAs take contiguous ranges of units, and every touched
// expert's weights are read once per tile (once in total when an expert has <= 8 tokens, the decode case).  The routed forms of a
// grouping workspace run as stream_tiles_kernel, the next tile's activations staged under the streaming; the others, and rows too long for its
// two buffers, as stream_kernel, which stages between tiles.

#include "experts.cuh"
#include "skinny_mma.cuh"
#include "tc_ptx.cuh"
#include "unit_runs.cuh"

#include <cuda_bf16.h>
#include <cuda_fp16.h>

namespace sxb {
namespace {

constexpr int kThreads = 256;      // small launches: two CTAs of eight warps an SM
constexpr int kBigThreads = 512;   // launches with work for every SM: one CTA of sixteen warps, units handed out on demand
constexpr int kTileTokens = 8;
constexpr int kPerTokenPasses = 8;  // tiles of eight slots of a token at most (A <= 64)
constexpr int kPrefetch = 4;  // steps of weights in flight per warp beyond the one being consumed
constexpr int64_t kMaxK = 1 << 24;
constexpr int64_t kMaxN = 0x7fffffff;
constexpr size_t kMaxDynSmem = 200 * 1024;
constexpr size_t kCtaExtra = 3 * 1024;  // shared memory of a routed CTA beside the dynamic part: static, and 1 KB of the system's

enum Mode { kGather = 0, kSwiglu = 1, kPartial = 2 };
enum Src { kFromWs = 0, kFromSlots = 1, kDense = 2, kPerToken = 3 };

template <int BITS, int G>
struct Geo {
    static constexpr int kCodesPerLane = (BITS == 4 ? 32 : 16) < G / 4 ? (BITS == 4 ? 32 : 16) : G / 4;
    static constexpr int kLoadBytes = kCodesPerLane * BITS / 8;  // 16, 8 or 4
    static constexpr int kWords = kLoadBytes / 4;
    static constexpr int kStepCodes = 4 * kCodesPerLane;  // codes of one row a quad consumes per step (<= G)
    static constexpr int kUnits = kCodesPerLane / 8;      // 16-byte activation units per lane per step
    static constexpr int kStepsPerGroup = G / kStepCodes;
};

template <int WORDS> __device__ inline void load_codes(uint32_t (&w)[WORDS], const uint8_t *p, bool pred);
template <> __device__ inline void load_codes<4>(uint32_t (&w)[4], const uint8_t *p, bool pred) {
    w[0] = w[1] = w[2] = w[3] = 0u;
    if (pred)
        asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
                     : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3])
                     : "l"(p));
}
template <> __device__ inline void load_codes<2>(uint32_t (&w)[2], const uint8_t *p, bool pred) {
    w[0] = w[1] = 0u;
    if (pred) asm volatile("ld.global.nc.L1::no_allocate.v2.u32 {%0,%1}, [%2];" : "=r"(w[0]), "=r"(w[1]) : "l"(p));
}
template <> __device__ inline void load_codes<1>(uint32_t (&w)[1], const uint8_t *p, bool pred) {
    w[0] = 0u;
    if (pred) asm volatile("ld.global.nc.L1::no_allocate.u32 %0, [%1];" : "=r"(w[0]) : "l"(p));
}

// D = A * B (no accumulator input: the zero operand needs no registers set up).
__device__ inline void mma_f16_first(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
}
__device__ inline void mma_f16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// d (+)= the products of eight codes of weight rows a and b with one staged unit of activations.  Q4: word w0; Q8: words w0,
// w1.  Codes as F16 subnormals (the header of this file): a mask for nibbles 0, 4 and 1, 5 of a word, the same two masks for
// nibbles 2, 6 and 3, 7 eight bits further down; a byte permute for a pair of Q8 codes.  A packed multiply then makes them the
// normal numbers n * 2^-9: with subnormal operands the tensor cores lose the sum some of its low bits (3.4e-5 of the RMS on a
// 64-long dot).
__device__ inline uint32_t times_h2(uint32_t v, uint32_t f) {
    uint32_t r;
    asm("mul.f16x2 %0, %1, %2;" : "=r"(r) : "r"(v), "r"(f));
    return r;
}
template <int BITS, bool FIRST>
__device__ inline void unit_mma(float (&d)[4], uint32_t a_w0, uint32_t a_w1, uint32_t b_w0, uint32_t b_w1, const uint4 &bx) {
    constexpr uint32_t k2p15 = 0x78007800u, k2p11 = 0x68006800u;  // packed 2^15 and 2^11
    uint32_t pa[4], pb[4];
    if (BITS == 4) {
        const uint32_t a8 = a_w0 >> 8, b8 = b_w0 >> 8;
        pa[0] = times_h2(a_w0 & 0x000F000Fu, k2p15), pa[1] = times_h2(a_w0 & 0x00F000F0u, k2p11);
        pa[2] = times_h2(a8 & 0x000F000Fu, k2p15), pa[3] = times_h2(a8 & 0x00F000F0u, k2p11);
        pb[0] = times_h2(b_w0 & 0x000F000Fu, k2p15), pb[1] = times_h2(b_w0 & 0x00F000F0u, k2p11);
        pb[2] = times_h2(b8 & 0x000F000Fu, k2p15), pb[3] = times_h2(b8 & 0x00F000F0u, k2p11);
    } else {
        pa[0] = times_h2(__byte_perm(a_w0, 0u, 0x4140), k2p15), pa[1] = times_h2(__byte_perm(a_w0, 0u, 0x4342), k2p15);
        pa[2] = times_h2(__byte_perm(a_w1, 0u, 0x4140), k2p15), pa[3] = times_h2(__byte_perm(a_w1, 0u, 0x4342), k2p15);
        pb[0] = times_h2(__byte_perm(b_w0, 0u, 0x4140), k2p15), pb[1] = times_h2(__byte_perm(b_w0, 0u, 0x4342), k2p15);
        pb[2] = times_h2(__byte_perm(b_w1, 0u, 0x4140), k2p15), pb[3] = times_h2(__byte_perm(b_w1, 0u, 0x4342), k2p15);
    }
    if (FIRST) mma_f16_first(d, pa[0], pb[0], pa[1], pb[1], bx.x, bx.y);
    else mma_f16(d, pa[0], pb[0], pa[1], pb[1], bx.x, bx.y);
    mma_f16(d, pa[2], pb[2], pa[3], pb[3], bx.z, bx.w);
}

__device__ inline float pow2f(int e) { return __int_as_float((e + 127) << 23); }  // e in -126 .. 127

// What stage_tile finds out about a token of the tile.
template <int BITS> constexpr bool kKeepLow = BITS == 8;  // see the head of this file
constexpr int kLowMax = 4;
struct Low {
    int k;
    float x;
};
struct Token {
    uint32_t top;  // largest magnitude of its activations, BF16 bits
    int low;       // the smallest that is not zero, as a signed 16-bit value with 0x7fff added (0x7fff: all are zero)
    int exp;       // e of the power 2^e that its dots carry beside the codes' 2^-9 (unscaled); 9 = none
    int n_low;     // activations too small for F16 beside the largest; more than kLowMax: the token is staged as BF16
    int n_list[2];  // the first kLowMax of them at most, ascending k, by each of the (one or two) warps that stage the token
    Low list[2][kLowMax];
};
__device__ inline void clear_token(Token &t) { t.top = 0u, t.low = 0x7fff, t.exp = 9, t.n_low = 0, t.n_list[0] = t.n_list[1] = 0; }
__device__ inline bool too_small(float scaled) { return fabsf(scaled) < 0x1p-14f; }

// The exponent e of a token's scale 2^e from the largest magnitude of its activations (BF16 bits without the sign): 2^15 <= max
// * 2^e < 65504, where the clamp to exponents that FP32 can hold allows it.
__device__ inline int token_exponent(uint32_t max_bits) { return min(max(142 - (int)(max_bits >> 7), -112), 126); }
// A dot of the staged operands back to its value: v * 2^(9 - e), in two factors that meet no range limit the result does not.
__device__ inline float unscaled(float v, int e) {
    const int t = 9 - e, h = t >> 1;
    return v * pow2f(h) * pow2f(t - h);
}

struct StreamArgs {
    const uint16_t *x;  // BF16 activations: x [M, K] (gather / dense) or h [M*A, K] (partial)
    const uint8_t *q;
    const uint16_t *scale, *minv;
    int64_t N, K;        // rows per expert, codes per row
    int64_t M, A, E;     // tokens, slots per token, experts in the view
    const int32_t *ws;   // kFromWs
    RouteWords L;
    const int32_t *ids;  // kFromSlots, kPerToken
    const float *coef;   // kPerToken
    void *out;
    uint32_t *err;
    uint32_t *status;    // kFromWs: {2, tile, role} of a wait that ran out, in the workspace's header
    unsigned long long wait_limit_ns;
    int test_skip_slot;  // >= 0: CTA 0's second (even) or third (odd) tile waits for one arrival more than its warps make (tests only)
    int chunks, split;   // see chunk_count: chunks of a contraction; warps that share a unit (1 .. chunks)
};

// Dense projections: a row's contraction is summed in `chunks` chunks of whole blocks, and the chunks' sums are added as a
// binary tree over their order.  Warps that share a unit take a power of two of neighbouring chunks each, i.e. a node of that tree, so a result does
// not depend on how many share it - which follows from the launch's size, and a row must not notice the rest of its batch.
// The routed forms have units enough from the first tokens on, and the chunks would cost them 6 % (150 tokens x 10 experts,
// 4096 x 2048 Q4: 415 -> 441 us).
constexpr int kMaxChunks = 8, kTreeLevels = 3;
inline int chunk_count(int64_t blocks) {
    int n = kMaxChunks;
    while (n > 1 && (blocks % n != 0 || blocks / n < 2)) n /= 2;
    return n;
}
// Node number i joins the tree: v becomes its sum with the left-hand nodes that were waiting for it in this thread's slots, a
// level of them kBigThreads apart.  Returns the slot where it would wait itself (past the last one when the tree is complete).
__device__ inline float4 *tree_join(float4 *level, int i, float (&v)[4]) {
    for (; i & 1; i >>= 1, level += kBigThreads) {
        const float4 l = *level;
        v[0] = l.x + v[0], v[1] = l.y + v[1], v[2] = l.z + v[2], v[3] = l.w + v[3];
    }
    return level;
}
__device__ inline void tree_push(float4 *level, int i, float (&v)[4]) {
    level = tree_join(level, i, v);
    *level = make_float4(v[0], v[1], v[2], v[3]);
}

template <typename T> __device__ inline void store_out(T *p, int64_t i, float v) { store_from_f32(p, i, v); }

// Stages activation row `row` as token n of a tile: F16 in fragment order at xs, times the row's power of two 2^e (token_exponent), and at xsum the
// sums of every step times 2^(e - 9), the factor that the dots with the codes carry.  kKeepLow: activations that would be subnormal are staged as
// zeros and listed in tok, which comes in cleared; *any_low = 1 where there are any.  By `warps` whole warps, of which this is number `share`;
// `meet` is the barrier between the first pass over the row and the second, and is called by every one of them (row == nullptr: no token).
// BATCH loads in flight a lane: under a streaming kernel's load an L2 round trip is thousands of cycles.
template <int BITS, int G, int BATCH, typename Meet>
__device__ __forceinline__ void stage_row(const uint16_t *__restrict__ row, int K, int n, int share, int warps, uint4 *xs, float *xsum, Token &tok,
                                          int *any_low, Meet meet) {
    using geo = Geo<BITS, G>;
    constexpr int UNITS = geo::kUnits, KI = geo::kStepCodes, CPL = geo::kCodesPerLane;
    constexpr int kStepLanes = KI / 8;  // lanes that hold one step of one token: 4, 8 or 16
    constexpr int kBatch = BATCH;
    const int lane = threadIdx.x & 31, stride = 32 * warps;
    const int units = K / 8;
    const uint4 *src = reinterpret_cast<const uint4 *>(row);
    uint4 v[kBatch];
    auto load = [&](int base) {
#pragma unroll
        for (int j = 0; j < kBatch; ++j)
            if (base + j * stride < units) v[j] = src[base + j * stride];
    };
    uint32_t top = 0u, low2 = 0x7fff7fffu;
    if (row != nullptr) {
        // sum(x) of every step: eight values a lane, then a butterfly over the step's lanes
        for (int base = share * 32 + lane; base - lane < units; base += kBatch * stride) {
            load(base);
#pragma unroll
            for (int j = 0; j < kBatch; ++j) {
                const int u = base + j * stride;
                if (u - lane >= units) break;
                float sum = 0.f;
                if (u < units) {
                    const uint32_t w4[4] = {v[j].x, v[j].y, v[j].z, v[j].w};
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        sum += __uint_as_float(w4[i] << 16), sum += __uint_as_float(w4[i] & 0xffff0000u);
                        const uint32_t mag = w4[i] & 0x7fff7fffu;
                        top = __vmaxu2(top, mag);
                        if (kKeepLow<BITS>) low2 = __viaddmin_s16x2(mag, 0x7fff7fffu, low2);
                    }
                }
#pragma unroll
                for (int o = kStepLanes / 2; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
                if (lane % kStepLanes == 0 && u < units) xsum[u / kStepLanes * kTileTokens + n] = sum;
            }
        }
        top = __reduce_max_sync(0xffffffffu, max(top >> 16, top & 0xffffu));
        if (lane == 0) atomicMax(&tok.top, top);
        if (kKeepLow<BITS>) {
            const int low = __reduce_min_sync(0xffffffffu, min((int)low2 >> 16, (int)(int16_t)low2));
            if (lane == 0) atomicMin(&tok.low, low);
        }
    }
    meet();
    // absent tokens' columns keep whatever the memory held: a column of the products depends on its own token only, and theirs
    // are dropped
    if (row == nullptr) return;
    const int e = token_exponent(tok.top), smallest = kKeepLow<BITS> ? tok.low : 0x7fff;
    const float f = pow2f(e);
    const bool low = smallest != 0x7fff && too_small(__uint_as_float((uint32_t)((smallest - 0x7fff) & 0xffff) << 16) * f);
    if (lane == 0 && share == 0) tok.exp = e;
    if (low) {
        int found = 0;
        for (int first = share * 32; first < units; first += stride) {
            const int u = first + lane;
            const uint4 q = u < units ? src[u] : make_uint4(0u, 0u, 0u, 0u);
            const uint32_t w4[4] = {q.x, q.y, q.z, q.w};
            uint32_t mine = 0u;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const float x = __uint_as_float((i & 1) ? w4[i >> 1] & 0xffff0000u : w4[i >> 1] << 16);
                if (x != 0.f && too_small(x * f)) mine |= 1u << i;
            }
            for (uint32_t who = __ballot_sync(0xffffffffu, mine != 0u); who != 0u; who &= who - 1) {
                const int l = __ffs(who) - 1;
                const uint32_t theirs = __shfl_sync(0xffffffffu, mine, l);
                if (lane == l) {
                    int at = found;
#pragma unroll
                    for (int i = 0; i < 8; ++i)
                        if (((mine >> i) & 1u) && at < kLowMax)
                            tok.list[share][at++] = Low{u * 8 + i, __uint_as_float((i & 1) ? w4[i >> 1] & 0xffff0000u : w4[i >> 1] << 16)};
                }
                found += __popc(theirs);
            }
        }
        if (lane == 0 && found > 0) tok.n_list[share] = min(found, kLowMax), atomicAdd(&tok.n_low, found), *any_low = 1;
    }
    // One batch holds a row up to 256 k a load and warp; a longer one is read again.
    const bool held = units <= kBatch * stride;
    for (int base = share * 32 + lane; base < units; base += kBatch * stride) {
        if (!held) load(base);
#pragma unroll
        for (int j = 0; j < kBatch; ++j) {
            const int u = base + j * stride, k = u * 8;
            if (u >= units) break;
            if (u % kStepLanes == 0) xsum[u / kStepLanes * kTileTokens + n] *= f * 0x1p-9f;
            const int step = k / KI, rem = k % KI, cc = rem / CPL, part = (rem % CPL) / 8;
            const uint32_t w4[4] = {v[j].x, v[j].y, v[j].z, v[j].w};
            float lo[4], hi[4];  // elements 2 i and 2 i + 1
#pragma unroll
            for (int i = 0; i < 4; ++i) lo[i] = __uint_as_float(w4[i] << 16) * f, hi[i] = __uint_as_float(w4[i] & 0xffff0000u) * f;
            auto pack = [](float a, float b) { const __half2 h = __floats2half2_rn(a, b); return *reinterpret_cast<const uint32_t *>(&h); };
            if (low) {
#pragma unroll
                for (int i = 0; i < 4; ++i) lo[i] = too_small(lo[i]) ? 0.f : lo[i], hi[i] = too_small(hi[i]) ? 0.f : hi[i];
            }
            uint4 dst;
            if (BITS == 4) {  // [x0 x4 | x1 x5 | x2 x6 | x3 x7]
                dst.x = pack(lo[0], lo[2]), dst.y = pack(hi[0], hi[2]), dst.z = pack(lo[1], lo[3]), dst.w = pack(hi[1], hi[3]);
            } else {  // natural order
                dst.x = pack(lo[0], hi[0]), dst.y = pack(lo[1], hi[1]), dst.z = pack(lo[2], hi[2]), dst.w = pack(lo[3], hi[3]);
            }
            xs[(step * UNITS + part) * 32 + n * 4 + cc] = dst;
        }
    }
}


// Stages up to 8 activation rows (rows[n] < 0 = none), a token by every eighth warp, so that what belongs to the token is the same for a whole
// warp (dealing 16-byte units out over the CTA cost two divisions a unit and an atomic a step: 150 tokens x 10 experts, 4096 x 2048 Q4,
// 415 -> 442 us).  All threads of the CTA; the caller synchronizes before it reads what is staged.
template <int BITS, int G>
__device__ inline void stage_tile(const uint16_t *__restrict__ x, int K, const int64_t *rows, uint4 *xs, float *xsum, Token *tok, int *any_low) {
    const int n = (threadIdx.x >> 5) & (kTileTokens - 1);
    stage_row<BITS, G, 8>(rows[n] >= 0 ? x + rows[n] * K : nullptr, K, n, threadIdx.x >> 8, (int)blockDim.x / (32 * kTileTokens), xs, xsum, tok[n], any_low,
                       [] { __syncthreads(); });
}

// A token with more than kLowMax small activations staged again, as BF16 in natural order, and its sums as they are; by `threads` threads, of
// which this is number t.
template <int BITS, int G>
__device__ __noinline__ void stage_wide(const uint16_t *__restrict__ row, int K, int n, uint4 *xs, float *xsum, Token &tok, int t, int threads) {
    using geo = Geo<BITS, G>;
    constexpr int KI = geo::kStepCodes;
    const uint4 *src = reinterpret_cast<const uint4 *>(row);
    if (t == 0) tok.exp = 9;
    for (int u = t; u < K / 8; u += threads) {
        const int step = u * 8 / KI, rem = u * 8 % KI;
        xs[(step * geo::kUnits + rem % geo::kCodesPerLane / 8) * 32 + n * 4 + rem / geo::kCodesPerLane] = src[u];
    }
    for (int step = t; step < K / KI; step += threads) {
        float sum = 0.f;
        for (int i = 0; i < KI; ++i) sum += bf16_bits_to_f32(row[(int64_t)step * KI + i]);
        xsum[step * kTileTokens + n] = sum;
    }
}
// After stage_tile and a barrier, where some token has small activations.
template <int BITS, int G>
__device__ inline void finish_staging(const uint16_t *__restrict__ x, int K, const int64_t *rows, uint4 *xs, float *xsum, Token *tok) {
    for (int n = 0; n < kTileTokens; ++n)
        if (tok[n].n_low > kLowMax) stage_wide<BITS, G>(x + rows[n] * K, K, n, xs, xsum, tok[n], threadIdx.x, blockDim.x);
    __syncthreads();
}

// What a token's listed activations add to its dot with weight row `row`, in ascending k (the mins' part is in xsum).
template <int BITS, int G>
__device__ __noinline__ float low_dot(const uint8_t *q, const uint16_t *scale, int K, int64_t row, const Token &tok) {
    float sum = 0.f;
    for (int i = 0, j = 0; i < tok.n_list[0] || j < tok.n_list[1];) {
        const bool first = j >= tok.n_list[1] || (i < tok.n_list[0] && tok.list[0][i].k < tok.list[1][j].k);
        const Low l = first ? tok.list[0][i++] : tok.list[1][j++];
        const uint8_t byte = BITS == 4 ? q[row * (K / 2) + l.k / 2] : q[row * K + l.k];
        const int code = BITS == 4 ? (byte >> (4 * (l.k & 1))) & 15 : byte;
        sum = fmaf(bf16_bits_to_f32(scale[row * (K / G) + l.k / G]), (float)code * l.x, sum);
    }
    return sum;
}

// The dots of weight rows rowa / rowb with the tokens that are staged as BF16 (the other tokens' sums are meaningless): codes as BF16
// too, exact products at any distance.  acc as below.  The whole contraction in order, whatever warps share it otherwise; rare, so
// short rather than fast.
template <int BITS, int G>
__device__ __noinline__ float4 rows_dot_wide(const uint8_t *q, const uint16_t *scale, const uint16_t *minv, int K, int64_t rowa, int64_t rowb,
                                             bool va, bool vb, const uint4 *xs, const float *xsum) {
    using geo = Geo<BITS, G>;
    constexpr int W = geo::kWords;
    const int lane = threadIdx.x & 31, c = lane & 3, steps = K / geo::kStepCodes, groups = K / G;
    const int64_t row_bytes = BITS == 4 ? K / 2 : K;
    const uint8_t *pa = q + rowa * row_bytes + c * geo::kLoadBytes, *pb = q + rowb * row_bytes + c * geo::kLoadBytes;
    auto pair = [](uint32_t w0, uint32_t w1, int i) -> uint32_t {  // codes 2 i and 2 i + 1 of eight
        const uint32_t w = BITS == 4 || i < 2 ? w0 : w1;
        const uint32_t lo = BITS == 4 ? (w >> (8 * i)) & 15u : (w >> (16 * (i & 1))) & 255u;
        const uint32_t hi = BITS == 4 ? (w >> (8 * i + 4)) & 15u : (w >> (16 * (i & 1) + 8)) & 255u;
        const __nv_bfloat162 p = __floats2bfloat162_rn((float)lo, (float)hi);  // eight significant bits: exact
        return *reinterpret_cast<const uint32_t *>(&p);
    };
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 1
    for (int step = 0; step < steps; ++step) {
        uint32_t wa[W], wb[W];
        load_codes<W>(wa, pa + (int64_t)step * 4 * geo::kLoadBytes, va);
        load_codes<W>(wb, pb + (int64_t)step * 4 * geo::kLoadBytes, vb);
        const int64_t ga = rowa * groups + step / geo::kStepsPerGroup, gb = rowb * groups + step / geo::kStepsPerGroup;
        const float s_a = va ? bf16_bits_to_f32(__ldg(scale + ga)) : 0.f, m_a = va ? bf16_bits_to_f32(__ldg(minv + ga)) : 0.f;
        const float s_b = vb ? bf16_bits_to_f32(__ldg(scale + gb)) : 0.f, m_b = vb ? bf16_bits_to_f32(__ldg(minv + gb)) : 0.f;
        float d[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int v = 0; v < geo::kUnits; ++v) {
            const uint4 bx = xs[(step * geo::kUnits + v) * 32 + lane];
            const int i0 = BITS == 4 ? v : 2 * v, i1 = BITS == 4 ? v : 2 * v + 1;
            mma_bf16(d, pair(wa[i0], wa[i1], 0), pair(wb[i0], wb[i1], 0), pair(wa[i0], wa[i1], 1), pair(wb[i0], wb[i1], 1), bx.x, bx.y);
            mma_bf16(d, pair(wa[i0], wa[i1], 2), pair(wb[i0], wb[i1], 2), pair(wa[i0], wa[i1], 3), pair(wb[i0], wb[i1], 3), bx.z, bx.w);
        }
        const float2 xs2 = *reinterpret_cast<const float2 *>(xsum + step * kTileTokens + 2 * c);
        acc.x = fmaf(s_a, d[0], fmaf(m_a, xs2.x, acc.x)), acc.y = fmaf(s_a, d[1], fmaf(m_a, xs2.y, acc.y));
        acc.z = fmaf(s_b, d[2], fmaf(m_b, xs2.x, acc.z)), acc.w = fmaf(s_b, d[3], fmaf(m_b, xs2.y, acc.w));
    }
    return acc;
}

// One warp: the dots of weight rows rowa / rowb (lane quad g streams both) with the staged tokens.
// acc[0], acc[1] = row a x tokens 2c, 2c+1;  acc[2], acc[3] = row b x the same tokens.
template <int BITS, int G>
__device__ inline void rows_dot_impl(float (&acc)[4], const StreamArgs &a, int64_t rowa, int64_t rowb, bool va, bool vb,
                                     const uint4 *xs, const float *xsum, int lane) {
    using geo = Geo<BITS, G>;
    constexpr int W = geo::kWords, UNITS = geo::kUnits, KI = geo::kStepCodes;
    const int K = (int)a.K, steps = K / KI, groups = K / G, c = lane & 3;
    const int64_t row_bytes = BITS == 4 ? a.K / 2 : a.K;
    const uint8_t *pa = a.q + rowa * row_bytes + c * geo::kLoadBytes;
    const uint8_t *pb = a.q + rowb * row_bytes + c * geo::kLoadBytes;
    const uint16_t *sa = a.scale + rowa * groups, *ma = a.minv + rowa * groups;
    const uint16_t *sb = a.scale + rowb * groups, *mb = a.minv + rowb * groups;

    uint32_t wa[kPrefetch][W], wb[kPrefetch][W];
    uint16_t qs[kPrefetch][4];  // scale a, min a, scale b, min b
    auto fetch = [&](int slot, int step) {
        const bool in = step < steps;
        load_codes<W>(wa[slot], pa + (int64_t)step * 4 * geo::kLoadBytes, in && va);
        load_codes<W>(wb[slot], pb + (int64_t)step * 4 * geo::kLoadBytes, in && vb);
        const int grp = step / geo::kStepsPerGroup;
        qs[slot][0] = in && va ? __ldg(sa + grp) : (uint16_t)0;
        qs[slot][1] = in && va ? __ldg(ma + grp) : (uint16_t)0;
        qs[slot][2] = in && vb ? __ldg(sb + grp) : (uint16_t)0;
        qs[slot][3] = in && vb ? __ldg(mb + grp) : (uint16_t)0;
    };
#pragma unroll
    for (int p = 0; p < kPrefetch; ++p) fetch(p, p);
    for (int step0 = 0; step0 < steps; step0 += kPrefetch) {
#pragma unroll
        for (int p = 0; p < kPrefetch; ++p) {
            const int step = step0 + p;
            if (step < steps) {
                float d[4] = {0.f, 0.f, 0.f, 0.f};
                const uint4 *xu = xs + (size_t)step * UNITS * 32 + lane;
#pragma unroll
                for (int v = 0; v < UNITS; ++v) {
                    const uint4 bx = xu[v * 32];
                    if (BITS == 4) unit_mma<4, false>(d, wa[p][v], 0u, wb[p][v], 0u, bx);
                    else unit_mma<8, false>(d, wa[p][2 * v], wa[p][2 * v + 1], wb[p][2 * v], wb[p][2 * v + 1], bx);
                }
                const float2 xs2 = *reinterpret_cast<const float2 *>(xsum + step * kTileTokens + 2 * c);
                const float s_a = bf16_bits_to_f32(qs[p][0]), s_b = bf16_bits_to_f32(qs[p][2]);
                const float m_a = bf16_bits_to_f32(qs[p][1]), m_b = bf16_bits_to_f32(qs[p][3]);
                acc[0] = fmaf(s_a, d[0], fmaf(m_a, xs2.x, acc[0]));
                acc[1] = fmaf(s_a, d[1], fmaf(m_a, xs2.y, acc[1]));
                acc[2] = fmaf(s_b, d[2], fmaf(m_b, xs2.x, acc[2]));
                acc[3] = fmaf(s_b, d[3], fmaf(m_b, xs2.y, acc[3]));
            }
            fetch(p, step + kPrefetch);  // refill the slot just consumed
        }
    }
}

// The common shape, kept lean because the kernel saturates the integer pipe before HBM: a step is one group, the row has
// a whole number of four-step blocks, scales and mins come by aligned 8-byte loads.  No per-load predicates (a row past
// the end of the expert is replaced by a row that exists; its sums are dropped by the caller), pointers advance by
// increments, the last block is peeled so nothing is fetched past the end of a row, and a step's first MMA takes a
// zero accumulator operand instead of cleared registers.
// TREE: the contraction in chunks (chunk_count), this warp's part of it only; otherwise one running sum.
template <int BITS, int G, bool TREE>
__device__ inline void rows_dot_fast(float (&acc)[4], const StreamArgs &a, int64_t rowa, int64_t rowb, const uint4 *xs,
                                     const float *xsum, int lane, int part, float4 *tree) {
    using geo = Geo<BITS, G>;
    constexpr int W = geo::kWords, UNITS = geo::kUnits, KI = geo::kStepCodes;
    constexpr int kBlockBytes = kPrefetch * 4 * geo::kLoadBytes;  // bytes of one row consumed per block of four steps
    const int K = (int)a.K, blocks = K / (KI * kPrefetch) / (TREE ? a.split : 1), groups = K / G, c = lane & 3;
    const int first = TREE ? part * blocks : 0, per_chunk = TREE ? K / (KI * kPrefetch) / a.chunks : 0;
    const int64_t row_bytes = BITS == 4 ? a.K / 2 : a.K, at = first * kBlockBytes + c * geo::kLoadBytes;
    const uint8_t *pa = a.q + rowa * row_bytes + at, *pb = a.q + rowb * row_bytes + at;
    const uint2 *sa = reinterpret_cast<const uint2 *>(a.scale + rowa * groups) + first, *ma = reinterpret_cast<const uint2 *>(a.minv + rowa * groups) + first;
    const uint2 *sb = reinterpret_cast<const uint2 *>(a.scale + rowb * groups) + first, *mb = reinterpret_cast<const uint2 *>(a.minv + rowb * groups) + first;
    const uint4 *xu = xs + lane + first * (kPrefetch * UNITS * 32);
    const float *xq = xsum + 2 * c + first * (kPrefetch * kTileTokens);

    uint32_t wa[kPrefetch][W], wb[kPrefetch][W];
    uint2 qv[4], qn[4];  // {scale a, min a, scale b, min b} of the block in use / of the next one
    auto fetch_codes = [&](int p) {  // step p of the block pa / pb point at
        load_codes<W>(wa[p], pa + p * 4 * geo::kLoadBytes, true);
        load_codes<W>(wb[p], pb + p * 4 * geo::kLoadBytes, true);
    };
    auto fetch_scales = [&](uint2 (&dst)[4]) { dst[0] = __ldg(sa), dst[1] = __ldg(ma), dst[2] = __ldg(sb), dst[3] = __ldg(mb); };
    auto consume = [&](int p) {
        float d[4];
#pragma unroll
        for (int v = 0; v < UNITS; ++v) {
            const uint4 bx = xu[(p * UNITS + v) * 32];
            const int i0 = BITS == 4 ? v : 2 * v, i1 = BITS == 4 ? v : 2 * v + 1;
            if (v == 0) unit_mma<BITS, true>(d, wa[p][i0], wa[p][i1], wb[p][i0], wb[p][i1], bx);
            else unit_mma<BITS, false>(d, wa[p][i0], wa[p][i1], wb[p][i0], wb[p][i1], bx);
        }
        const float2 xs2 = *reinterpret_cast<const float2 *>(xq + p * kTileTokens);
        // BF16 bits -> FP32: the upper half of the word as it is, the lower half shifted up
        auto f32_of = [&](const uint2 &q) { const uint32_t w = p < 2 ? q.x : q.y; return __uint_as_float((p & 1) ? (w & 0xffff0000u) : (w << 16)); };
        const float s_a = f32_of(qv[0]), s_b = f32_of(qv[2]);
        const float m_a = f32_of(qv[1]), m_b = f32_of(qv[3]);
        acc[0] = fmaf(s_a, d[0], fmaf(m_a, xs2.x, acc[0]));
        acc[1] = fmaf(s_a, d[1], fmaf(m_a, xs2.y, acc[1]));
        acc[2] = fmaf(s_b, d[2], fmaf(m_b, xs2.x, acc[2]));
        acc[3] = fmaf(s_b, d[3], fmaf(m_b, xs2.y, acc[3]));
    };

    fetch_scales(qv);
#pragma unroll
    for (int p = 0; p < kPrefetch; ++p) fetch_codes(p);
    int chunk = 0, left = per_chunk;
    for (int b = 1; b < blocks; ++b) {  // consume block b - 1, fetching block b into the registers it frees
        pa += kBlockBytes, pb += kBlockBytes, ++sa, ++ma, ++sb, ++mb;
        fetch_scales(qn);
#pragma unroll
        for (int p = 0; p < kPrefetch; ++p) {
            consume(p);
            fetch_codes(p);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) qv[i] = qn[i];
        xu += kPrefetch * UNITS * 32, xq += kPrefetch * kTileTokens;
        if (TREE && --left == 0) {
            tree_push(tree, chunk++, acc);
            acc[0] = acc[1] = acc[2] = acc[3] = 0.f, left = per_chunk;
        }
    }
#pragma unroll
    for (int p = 0; p < kPrefetch; ++p) consume(p);
    if (TREE && chunk > 0) tree_join(tree, chunk, acc);
}

// Whether a row's scales and mins are whole aligned 8-byte loads of four groups.
__host__ __device__ inline bool vector_scales(const StreamArgs &a, int G) {
    return (a.K / G) % 4 == 0 && ((reinterpret_cast<uintptr_t>(a.scale) | reinterpret_cast<uintptr_t>(a.minv)) & 7) == 0;
}

// The dots of this warp's part of the contraction (part 0 of 1: all of it).  tree: the thread's slots, kBigThreads apart.
template <int BITS, int G, bool TREE>
__device__ inline void rows_dot(float (&acc)[4], const StreamArgs &a, int64_t rowa, int64_t rowb, bool va, bool vb,
                                const uint4 *xs, const float *xsum, int lane, int part, float4 *tree) {
    using geo = Geo<BITS, G>;
    if (geo::kStepsPerGroup == 1 && vector_scales(a, G)) {
        // rows past the end of the expert: stream a row that exists instead (the caller drops their sums)
        const int64_t any = va ? rowa : vb ? rowb : 0;
        rows_dot_fast<BITS, G, TREE>(acc, a, va ? rowa : any, vb ? rowb : any, xs, xsum, lane, part, tree);
    } else {
        rows_dot_impl<BITS, G>(acc, a, rowa, rowb, va, vb, xs, xsum, lane);
    }
}

// A unit's dots acc -> results.  Lane (g, c) holds rows ra and rb of the expert for tokens 2c and 2c + 1 of the tile; low: some of its tokens have
// activations too small for F16.
template <int BITS, int G, int MODE, typename TOUT>
__device__ __forceinline__ void finish_unit(const StreamArgs &a, TOUT *out, float (&acc)[4], int bucket, int cnt, int64_t ra, int64_t rb, bool va, bool vb,
                                            const uint4 *xs, const float *xsum, const Token *tok, const int64_t *orows, int low) {
    const int K = (int)a.K, c = threadIdx.x & 3;
    const int64_t I = a.N / 2;
    const bool valid = bucket < a.E;  // bucket E: slots with an id outside [0, E) - their outputs become NaN
    const int64_t row0 = (int64_t)bucket * a.N;
    const bool any_low = kKeepLow<BITS> && valid && low != 0;
    if (any_low) {
        bool wide[2] = {tok[2 * c].n_low > kLowMax, tok[2 * c + 1].n_low > kLowMax};
        if (__any_sync(0xffffffffu, wide[0] || wide[1])) {
            const float4 w = rows_dot_wide<BITS, G>(a.q, a.scale, a.minv, K, row0 + ra, row0 + rb, va, vb, xs, xsum);
            if (wide[0]) acc[0] = w.x, acc[2] = w.z;
            if (wide[1]) acc[1] = w.y, acc[3] = w.w;
        }
    }
#pragma unroll
    for (int t = 0; t < 2; ++t) {
        const int n = 2 * c + t;
        if (n >= cnt) continue;
        const int64_t orow = orows[n];
        const Token &token = tok[n];
        float dot_a = unscaled(acc[t], token.exp), dot_b = unscaled(acc[2 + t], token.exp);
        if (any_low && token.n_low > 0 && token.n_low <= kLowMax) {
            if (va) dot_a += low_dot<BITS, G>(a.q, a.scale, K, row0 + ra, token);
            if (vb) dot_b += low_dot<BITS, G>(a.q, a.scale, K, row0 + rb, token);
        }
        if (MODE == kSwiglu) {
            if (!va) continue;
            // kernels/linear_q4.hip:272-274: g, u as stored, h = stored(stored(silu(g)) * u)
            const float gg = as_stored_bf16(dot_a), uu = as_stored_bf16(dot_b);
            const float hv = as_stored_bf16(silu_f32(gg)) * uu;
            store_out(out, orow * I + ra, valid ? hv : qnan_f32());
        } else {
            if (va) store_out(out, orow * a.N + ra, valid ? dot_a : qnan_f32());
            if (vb) store_out(out, orow * a.N + rb, valid ? dot_b : qnan_f32());
        }
    }
}

template <int BITS, int G, int MODE, int SRC, typename TOUT>
__global__ void __launch_bounds__(kBigThreads, 1) stream_kernel(const StreamArgs a) {
    behind_grid();
    using geo = Geo<BITS, G>;
    const int kWarps = (int)blockDim.x >> 5;
    extern __shared__ __align__(16) unsigned char smem[];
    const int K = (int)a.K, steps = K / geo::kStepCodes;
    const size_t pass_bytes = (size_t)steps * geo::kUnits * 512 + (size_t)steps * kTileTokens * 4;
    __shared__ int64_t s_row[kTileTokens];  // activation row of each token of the tile, -1 = none
    __shared__ int64_t s_out[kTileTokens];  // output row (slot, or token for dense)
    __shared__ Token s_tok[SRC == kPerToken ? kPerTokenPasses : 1][kTileTokens];
    __shared__ int s_low[SRC == kPerToken ? kPerTokenPasses : 1];  // some token of the tile has activations too small for F16
    __shared__ int s_bucket, s_cnt;
    __shared__ int s_next;  // the next unit of the CTA's run that no warp has taken yet
    constexpr bool kTree = SRC == kDense;
    __shared__ float4 s_tree[kTree ? kTreeLevels * kBigThreads : 1];  // tree_push; its last level also hands parts' sums over
    const int split = kTree ? a.split : 1;

    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, c = lane & 3;
    const int64_t I = a.N / 2;
    const int64_t units_per_tile = MODE == kSwiglu ? (I + 7) / 8 : (a.N + 15) / 16;
    const int64_t n_tiles = SRC == kFromWs      ? a.ws[0]
                            : SRC == kFromSlots ? a.M * a.A
                            : SRC == kDense     ? (a.M + kTileTokens - 1) / kTileTokens
                                                : a.M;
    const int64_t total = n_tiles * units_per_tile;
    TOUT *out = static_cast<TOUT *>(a.out);
    // How the units are dealt to the CTAs.  Even split: CTA b takes units [total b / n, total (b + 1) / n) - every CTA busy,
    // but a CTA whose range crosses a tile boundary stages activations twice.  Tile-aligned: every tile's units are cut into
    // `cpt` equal runs and a CTA takes whole runs, one staging each.  The aligned cut is taken when it leaves (almost) no CTA
    // idle; inside a run the warps take units on demand either way.
    const int64_t nb = gridDim.x;
    int64_t cpt = max((int64_t)1, nb / max(n_tiles, (int64_t)1));
    const int n_groups = kWarps / split;  // a group of `split` warps takes a unit at a time
    const int64_t chunk = ((units_per_tile + cpt - 1) / cpt + n_groups - 1) / n_groups * n_groups;
    cpt = (units_per_tile + chunk - 1) / chunk;
    const int64_t n_chunks = n_tiles * cpt;
    const bool aligned = ((n_chunks + nb - 1) / nb) * chunk * 100 <= ((total + nb - 1) / nb) * 115;
    for (int64_t ci = blockIdx.x; ci < (aligned ? n_chunks : nb); ci += nb) {
    int64_t u_begin, u_end;
    if (aligned) {
        u_begin = (ci / cpt) * units_per_tile + (ci % cpt) * chunk;
        u_end = min((ci / cpt + 1) * units_per_tile, u_begin + chunk);
    } else {
        u_begin = total * ci / nb, u_end = total * (ci + 1) / nb;
    }
    for (int64_t tile = u_begin / units_per_tile; tile * units_per_tile < u_end; ++tile) {
        const int64_t lo = max(u_begin, tile * units_per_tile), hi = min(u_end, (tile + 1) * units_per_tile);

        if (SRC == kPerToken) {
            // Per-slot combine (kernels/linear_q4.hip:281-322): the tile is token `tile`; its A slots' h rows are
            // staged eight to a pass, every slot meets its own expert's rows, and y = sum_a coef * dot in slot order.
            const int64_t m = tile;
            const int passes = (int)((a.A + kTileTokens - 1) / kTileTokens);
            __syncthreads();
            if (threadIdx.x == 0) {
                int bad = -1;
                for (int k = 0; k < a.A && bad < 0; ++k)
                    if (a.ids[m * a.A + k] < 0 || a.ids[m * a.A + k] >= a.E) bad = k;
                if (bad >= 0) raise_error(a.err, (uint32_t)a.ids[m * a.A + bad], (uint32_t)(m * a.A + bad));
                s_cnt = bad < 0;
            }
            __syncthreads();
            const bool valid = s_cnt != 0;
            for (int p = 0; valid && p < passes; ++p) {
                __syncthreads();
                if (threadIdx.x < kTileTokens) {
                    const int k = p * kTileTokens + threadIdx.x;
                    s_row[threadIdx.x] = k < a.A ? m * a.A + k : -1;
                    clear_token(s_tok[p][threadIdx.x]);
                    if (threadIdx.x == 0) s_low[p] = 0;
                }
                __syncthreads();
                stage_tile<BITS, G>(a.x, K, s_row, reinterpret_cast<uint4 *>(smem + p * pass_bytes),
                                    reinterpret_cast<float *>(smem + p * pass_bytes + (size_t)steps * geo::kUnits * 512), s_tok[p], &s_low[p]);
                __syncthreads();
                if (kKeepLow<BITS> && s_low[p])
                    finish_staging<BITS, G>(a.x, K, s_row, reinterpret_cast<uint4 *>(smem + p * pass_bytes),
                                            reinterpret_cast<float *>(smem + p * pass_bytes + (size_t)steps * geo::kUnits * 512), s_tok[p]);
            }
            __syncthreads();
            for (int64_t unit = lo + warp; unit < hi; unit += kWarps) {
                const int64_t u = unit - tile * units_per_tile;
                const int64_t ra = u * 16 + g, rb = ra + 8;
                const bool va = ra < a.N, vb = rb < a.N;
                float ta = 0.f, tb = 0.f;
                for (int k = 0; valid && k < a.A; ++k) {
                    const int p = k / kTileTokens, col = k % kTileTokens;
                    const int64_t base = (int64_t)a.ids[m * a.A + k] * a.N;
                    float acc[4] = {0.f, 0.f, 0.f, 0.f};
                    const uint4 *xs = reinterpret_cast<const uint4 *>(smem + p * pass_bytes);
                    const float *xsum = reinterpret_cast<const float *>(smem + p * pass_bytes + (size_t)steps * geo::kUnits * 512);
                    const Token &tok = s_tok[p][col];
                    if (kKeepLow<BITS> && tok.n_low > kLowMax) {
                        const float4 w = rows_dot_wide<BITS, G>(a.q, a.scale, a.minv, K, base + ra, base + rb, va, vb, xs, xsum);
                        acc[0] = w.x, acc[1] = w.y, acc[2] = w.z, acc[3] = w.w;
                    } else {
                        rows_dot<BITS, G, false>(acc, a, base + ra, base + rb, va, vb, xs, xsum, lane, 0, nullptr);
                    }
                    if (c == col / 2) {  // the lane of the quad that holds this slot's column
                        const float cf = a.coef[m * a.A + k];
                        float da = unscaled(col & 1 ? acc[1] : acc[0], tok.exp), db = unscaled(col & 1 ? acc[3] : acc[2], tok.exp);
                        if (kKeepLow<BITS> && tok.n_low > 0 && tok.n_low <= kLowMax) {
                            if (va) da += low_dot<BITS, G>(a.q, a.scale, K, base + ra, tok);
                            if (vb) db += low_dot<BITS, G>(a.q, a.scale, K, base + rb, tok);
                        }
                        ta = fmaf(cf, da, ta);
                        tb = fmaf(cf, db, tb);
                    }
                }
                // the four lanes of a quad hold the partial sums of slots {0,1}, {2,3}, {4,5}, {6,7} (mod 8)
                ta += __shfl_xor_sync(0xffffffffu, ta, 1), tb += __shfl_xor_sync(0xffffffffu, tb, 1);
                ta += __shfl_xor_sync(0xffffffffu, ta, 2), tb += __shfl_xor_sync(0xffffffffu, tb, 2);
                if (c == 0) {
                    if (va) store_out(out, m * a.N + ra, valid ? ta : qnan_f32());
                    if (vb) store_out(out, m * a.N + rb, valid ? tb : qnan_f32());
                }
            }
            continue;
        }

        __syncthreads();  // every warp is done with the previous tile's shared memory
        if (threadIdx.x < kTileTokens) {
            const int n = threadIdx.x;
            int64_t row = -1, orow = -1;
            if (SRC == kFromWs) {
                const int bucket = a.ws[a.L.t8_bucket + tile], start = a.ws[a.L.t8_start + tile];
                const int cnt = min(kTileTokens, a.ws[a.L.offsets + bucket + 1] - start);
                if (n == 0) s_bucket = bucket, s_cnt = cnt;
                if (n < cnt) {
                    orow = a.ws[a.L.slots + start + n];
                    row = MODE == kPartial ? orow : orow / a.A;
                }
            } else if (SRC == kFromSlots) {
                if (n == 0) {
                    const int32_t id = a.ids[tile];
                    const bool ok = id >= 0 && id < a.E;
                    if (!ok) raise_error(a.err, (uint32_t)id, (uint32_t)tile);
                    s_bucket = ok ? id : (int)a.E, s_cnt = 1;
                    orow = tile;
                    row = MODE == kPartial ? tile : tile / a.A;
                }
            } else {
                const int64_t m = tile * kTileTokens + n;
                if (n == 0) s_bucket = 0, s_cnt = (int)min((int64_t)kTileTokens, a.M - tile * kTileTokens);
                if (m < a.M) row = orow = m;
            }
            s_row[n] = row, s_out[n] = orow, clear_token(s_tok[0][n]);
            if (n == 0) s_low[0] = 0;
        }
        __syncthreads();
        const int bucket = s_bucket, cnt = s_cnt;
        const bool valid = bucket < a.E;  // bucket E: slots with an id outside [0, E) - their outputs become NaN
        uint4 *xs = reinterpret_cast<uint4 *>(smem);
        float *xsum = reinterpret_cast<float *>(smem + (size_t)steps * geo::kUnits * 512);
        const int part = warp & (split - 1), group = warp / split;
        // The two weight rows of a unit that this lane streams, as rows inside the expert.
        auto rows_of = [&](int64_t unit, int64_t &ra, int64_t &rb, bool &va, bool &vb) {
            const int64_t u = unit - tile * units_per_tile;
            if (MODE == kSwiglu) {
                ra = u * 8 + g, rb = I + u * 8 + g;
                va = vb = u * 8 + g < I;
            } else {
                ra = u * 16 + g, rb = ra + 8;
                va = ra < a.N, vb = rb < a.N;
            }
        };
        if (kTree && valid && lo + group < hi) {
            // The codes of the warp's first unit are asked for, into L2, before the staging below goes to memory itself.
            int64_t ra, rb;
            bool va, vb;
            rows_of(lo + group, ra, rb, va, vb);
            const int64_t row_bytes = BITS == 4 ? a.K / 2 : a.K;
            const uint8_t *base = a.q + (int64_t)bucket * a.N * row_bytes;
            for (int64_t at = row_bytes * part / split + c * 128; at < row_bytes * (part + 1) / split; at += 512) {
                if (va) asm volatile("prefetch.global.L2 [%0];" ::"l"(base + ra * row_bytes + at));
                if (vb) asm volatile("prefetch.global.L2 [%0];" ::"l"(base + rb * row_bytes + at));
            }
        }
        if (valid) stage_tile<BITS, G>(a.x, K, s_row, xs, xsum, s_tok[0], &s_low[0]);
        if (threadIdx.x == 0) s_next = 0;
        __syncthreads();
        if (kKeepLow<BITS> && s_low[0]) finish_staging<BITS, G>(a.x, K, s_row, xs, xsum, s_tok[0]);

        // split == 1: warps take units on demand.  Two warps of an SM do not stream at the same rate (measured: the units of one
        // of two co-resident CTAs took 2.5 times as long as the other's while both were alive), and a fixed deal leaves the
        // fast ones idle at the end.  A unit's result does not depend on which warp computes it.
        // split > 1 (few units): `split` warps share a unit, each a run of its contraction's chunks, and the first adds the parts.
        int round = 0;
        auto next_unit = [&]() -> int64_t {
            if (kTree && split > 1) return lo + group + (int64_t)round * n_groups;
            int taken = 0;
            if (lane == 0) taken = atomicAdd(&s_next, 1);
            return lo + __shfl_sync(0xffffffffu, taken, 0);
        };
        auto group_sync = [&] { asm volatile("bar.sync %0, %1;" ::"r"(1 + group), "r"(32 * split) : "memory"); };
        for (int64_t unit; (unit = next_unit()) < hi; ++round) {
            int64_t ra, rb;
            bool va, vb;
            rows_of(unit, ra, rb, va, vb);
            float acc[4] = {0.f, 0.f, 0.f, 0.f};
            if (valid) rows_dot<BITS, G, kTree>(acc, a, (int64_t)bucket * a.N + ra, (int64_t)bucket * a.N + rb, va, vb, xs, xsum, lane, part, s_tree + threadIdx.x);
            if (kTree && split > 1) {
                // a warp that shares a unit has at most half its chunks, so the last level of its own tree is free for this
                float4 *parts = s_tree + (kTreeLevels - 1) * kBigThreads + threadIdx.x;
                if (part != 0) *parts = make_float4(acc[0], acc[1], acc[2], acc[3]);
                group_sync();
                if (part == 0) {
                    tree_push(s_tree + threadIdx.x, 0, acc);
                    for (int p = 1; p < split; ++p) {
                        const float4 v = parts[32 * p];
                        acc[0] = v.x, acc[1] = v.y, acc[2] = v.z, acc[3] = v.w;
                        if (p + 1 < split) tree_push(s_tree + threadIdx.x, p, acc);
                        else tree_join(s_tree + threadIdx.x, p, acc);
                    }
                }
                group_sync();
                if (part != 0) continue;
            }
            finish_unit<BITS, G, MODE>(a, out, acc, bucket, cnt, ra, rb, va, vb, xs, xsum, s_tok[0], s_out, s_low[0]);
        }
    }
    }
}

// The routed forms: one CTA of sixteen warps an SM, the tiles' activations in two buffers of shared memory.  The next tile's are staged under the
// streaming, a token by a warp - at once where the buffer is free, else after its next unit - and a warp that finds no unit left goes on to the
// next tile by itself: no barrier of the CTA stands between two tiles.  So a CTA may begin and end inside a tile, and the units are dealt evenly, unless
// whole tiles a group of CTAs suit the launch better (unit_runs.cuh).
// Results as stream_kernel's, bit for bit: a unit's sums do not depend on who forms them.
// What bounds it: HBM while it streams, 22 bytes a cycle and SM, 6.2 TB/s, whatever the tile; launch and first staging (8000 cycles), the last
// units.  With one buffer and a barrier on either side of the staging, tile-aligned runs and, in small launches, CTAs of eight warps two an SM, it
// streamed 76 to 87 % of the time.  4096 x 2048 + 1024 x 4096, 512 experts, top-10, gate/up and down us, before -> now: 16 tokens Q4 130 + 70 -> 121 + 63,
// 37 tokens (Q8 down) 207 + 167 -> 184 + 158, 150 tokens 424 + 234 -> 384 + 211; the layer as a graph, 2 tokens 82 -> 65, 4 107 -> 87, 64 599 -> 523.
// The staging's loads are four at a time and inline: with eight or sixteen in flight, or as a call, the loop over a unit's codes lost registers to
// them (16 tokens 126 + 65; as a call 200 + 89).
// The codes come through L1, some 32 KB of them on their way.  The pack of more than 2048 slots leaves the SMs of its last CTAs with all of their 256 KB
// but 28 as shared memory, which is enough for a CTA of this kernel, and there its warps ran at half their speed: with runs dealt ahead of time the whole launch did.  So
// the launch says how much shared memory it wants (launch_behind_l1): gate/up at 205 tokens 809 -> 405 us (Q8 down 334 -> 227), the layer of 230 tokens 1242 -> 847,
// of 400 tokens 1575 -> 1170; up to 204 tokens the same as before.
// Every wait is bounded; one that runs out is recorded in the grouping workspace's status words and ends the warp.
constexpr int kTileBufs = 2, kBigWarps = kBigThreads / 32;
struct TileBuf {
    int64_t row[kTileTokens], out[kTileTokens];  // activation and output row of each token, -1 = none
    Token tok[kTileTokens];
    int bucket, cnt, next;  // next: the next unit of the CTA's run that no warp has taken yet
};
// A token of the next tile, by one warp.
template <int BITS, int G>
__device__ __forceinline__ void stage_token(const uint16_t *row, int K, int n, uint4 *xs, float *xsum, Token *tok) {
    int any_low = 0;
    stage_row<BITS, G, 4>(row, K, n, 0, 1, xs, xsum, *tok, &any_low, [] { __syncwarp(); });
    __syncwarp();
    if (kKeepLow<BITS> && tok->n_low > kLowMax) stage_wide<BITS, G>(row, K, n, xs, xsum, *tok, threadIdx.x & 31, 32);
}
template <int BITS, int G, int MODE, typename TOUT>
__global__ void __launch_bounds__(kBigThreads, 1) stream_tiles_kernel(const StreamArgs a) {
    behind_grid();
    using geo = Geo<BITS, G>;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ TileBuf bufs[kTileBufs];
    __shared__ int s_low;  // some token of the first tile has activations too small for F16
    __shared__ uint64_t staged[kTileBufs], left[kTileBufs];  // a buffer's tile is staged (a warp a token) / every warp has left it
    const int K = (int)a.K, steps = K / geo::kStepCodes, xs_bytes = steps * geo::kUnits * 512, pass_bytes = xs_bytes + steps * kTileTokens * 4;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2;
    const int I = (int)(a.N / 2), units_per_tile = MODE == kSwiglu ? (I + 7) / 8 : (int)((a.N + 15) / 16);
    TOUT *out = static_cast<TOUT *>(a.out);
    const UnitRun run = unit_run((uint32_t)a.ws[0], (uint32_t)units_per_tile, blockIdx.x, gridDim.x, kBigWarps);
    const int tile0 = run.tile0, tile1 = run.tile1, u0 = run.u0, u1 = run.u1;
    if (tile0 > tile1) return;

    auto xs_of = [&](int b) { return reinterpret_cast<uint4 *>(smem + b * pass_bytes); };
    auto xsum_of = [&](int b) { return reinterpret_cast<float *>(smem + b * pass_bytes + xs_bytes); };
    // Token n of tile `tile`; n == 0 also describes the tile.
    auto describe = [&](TileBuf &t, int tile, int n) {
        const int bucket = a.ws[a.L.t8_bucket + tile], start = a.ws[a.L.t8_start + tile];
        const int cnt = min(kTileTokens, a.ws[a.L.offsets + bucket + 1] - start);
        int64_t row = -1, orow = -1;
        if (n < cnt) orow = a.ws[a.L.slots + start + n], row = MODE == kPartial ? orow : orow / a.A;
        t.row[n] = bucket < a.E ? row : -1, t.out[n] = orow, clear_token(t.tok[n]);
        if (n == 0) t.bucket = bucket, t.cnt = cnt, t.next = tile == tile0 ? u0 : 0;
    };
    if (threadIdx.x < kTileTokens) describe(bufs[0], tile0, threadIdx.x);
    if (threadIdx.x == 0) {
        for (int b = 0; b < kTileBufs; ++b) mbar_init(&staged[b], kTileTokens + (blockIdx.x == 0 && a.test_skip_slot >= 0 && b != (a.test_skip_slot & 1))), mbar_init(&left[b], kBigWarps);
        s_low = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    stage_tile<BITS, G>(a.x, K, bufs[0].row, xs_of(0), xsum_of(0), bufs[0].tok, &s_low);
    __syncthreads();
    if (kKeepLow<BITS> && s_low) finish_staging<BITS, G>(a.x, K, bufs[0].row, xs_of(0), xsum_of(0), bufs[0].tok);

    auto wait = [&](uint64_t *bar, uint32_t parity, int tile, int role) {
        const bool ok = __all_sync(0xffffffffu, mbar_wait(bar, parity, nullptr, a.wait_limit_ns));
        if (!ok && lane == 0 && atomicCAS(&a.status[0], 0u, 2u) == 0u) a.status[1] = (uint32_t)tile, a.status[2] = (uint32_t)role;
        return ok;
    };
    for (int tile = tile0; tile <= tile1; ++tile) {
        const int j = tile - tile0, b = j & 1;
        const uint32_t turn = (uint32_t)((j - 1) >> 1) & 1u;  // of this tile's `staged` and of the last one's `left`
        TileBuf &t = bufs[b];
        if (j > 0 && !wait(&staged[b], turn, tile, kRoleStaged)) return;
        const int low = kKeepLow<BITS> && __any_sync(0xffffffffu, t.tok[lane & (kTileTokens - 1)].n_low != 0);
        const int hi = tile == tile1 ? u1 : units_per_tile;
        bool to_stage = tile < tile1 && warp < kTileTokens;
        for (bool again = false;; again = true) {
            if (to_stage && (again || j == 0 || __all_sync(0xffffffffu, mbar_test(&left[b ^ 1], turn)))) {
                to_stage = false;
                TileBuf &n = bufs[b ^ 1];
                if (j > 0 && !wait(&left[b ^ 1], turn, tile, kRoleLeft)) return;
                if (lane == 0) describe(n, tile + 1, warp);
                __syncwarp();
                if (n.row[warp] >= 0) stage_token<BITS, G>(a.x + n.row[warp] * K, K, warp, xs_of(b ^ 1), xsum_of(b ^ 1), &n.tok[warp]);
                __syncwarp();
                if (lane == 0) mbar_arrive(&staged[b ^ 1]);
            }
            int u = 0;
            if (lane == 0) u = atomicAdd(&t.next, 1);
            u = __shfl_sync(0xffffffffu, u, 0);
            if (u < hi) {
                const int bucket = t.bucket, ra = MODE == kSwiglu ? u * 8 + g : u * 16 + g, rb = MODE == kSwiglu ? I + ra : ra + 8;
                const bool va = MODE == kSwiglu ? ra < I : ra < (int)a.N, vb = MODE == kSwiglu ? va : ra < (int)a.N - 8;
                float acc[4] = {0.f, 0.f, 0.f, 0.f};
                if (bucket < a.E)
                    rows_dot<BITS, G, false>(acc, a, (int64_t)bucket * a.N + ra, (int64_t)bucket * a.N + rb, va, vb, xs_of(b), xsum_of(b), lane, 0, nullptr);
                finish_unit<BITS, G, MODE>(a, out, acc, bucket, t.cnt, ra, rb, va, vb, xs_of(b), xsum_of(b), t.tok, t.out, low);
            }
            if (u >= hi && !to_stage) break;
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&left[b]);
    }
}

// v = four columns of token m, from n on: sum_a fma(coef[m, a], partial[m*A + a, n]) in slot order; NaN for a token with an id
// outside [0, E_total).  Slots of experts outside [e_lo, e_lo + E_local) - other ranks' in expert-parallel runs - are skipped.
// PBF16: the per-slot dots are BF16 bits, N * 2 bytes a slot (kernels/moe_grouped.hip:47-57), read from the same buffer.
// Memory-bound: five slots' loads are issued before the first is added (one slot at a time, its load
// behind its id's: 159 -> 146 us at 4096 tokens x 10 slots x 4096, 509 -> 477 at 16384).
template <bool PBF16>
__device__ inline void combine_slots(float (&v)[4], const float *__restrict__ partial, const int32_t *__restrict__ ids,
                                     const float *__restrict__ coef, int64_t m, int64_t n, int64_t A, int64_t E_total, int64_t e_lo,
                                     int64_t E_local, int64_t N) {
    constexpr int kAhead = 5;
    bool ok = true;
    v[0] = v[1] = v[2] = v[3] = 0.f;
    for (int64_t k0 = 0; k0 < A; k0 += kAhead) {
        float4 p[kAhead];
        float cf[kAhead];
        bool use[kAhead];
#pragma unroll
        for (int u = 0; u < kAhead; ++u) {
            const int64_t slot = m * A + k0 + u;
            const bool in = k0 + u < A;
            const int32_t id = in ? __ldg(ids + slot) : 0;
            ok = ok && (!in || (id >= 0 && id < E_total));
            use[u] = in && id >= e_lo && id < e_lo + E_local;
            cf[u] = use[u] ? __ldg(coef + slot) : 0.f;
            if (!use[u]) continue;
            if constexpr (PBF16) {
                const uint2 b = __ldg(reinterpret_cast<const uint2 *>(reinterpret_cast<const uint16_t *>(partial) + slot * N + n));
                p[u].x = __uint_as_float(b.x << 16), p[u].y = __uint_as_float(b.x & 0xffff0000u);
                p[u].z = __uint_as_float(b.y << 16), p[u].w = __uint_as_float(b.y & 0xffff0000u);
            } else {
                p[u] = __ldg(reinterpret_cast<const float4 *>(partial + slot * N + n));
            }
        }
#pragma unroll
        for (int u = 0; u < kAhead; ++u) {
            if (!use[u]) continue;
            v[0] = fmaf(cf[u], p[u].x, v[0]), v[1] = fmaf(cf[u], p[u].y, v[1]);
            v[2] = fmaf(cf[u], p[u].z, v[2]), v[3] = fmaf(cf[u], p[u].w, v[3]);
        }
    }
    if (!ok) v[0] = v[1] = v[2] = v[3] = qnan_f32();
}

// y[m, n] = sum_a fma(coef[m, a], partial[m*A + a, n]) in slot order, one rounding (kernels/moe_grouped.hip:948-984).
// Four columns a thread.  A token with an id outside [0, E_total) gets a NaN row.  Slots of experts outside
// [e_lo, e_lo + E_local) - other ranks' in expert-parallel runs - are skipped.  SH folds the shared expert's gated add:
// y = stored(sum) + sigmoid(gate) * s, the arithmetic of moe_shared_add on the stored y.
// PBF16: the per-slot dots are BF16 bits, N * 2 bytes a slot (kernels/moe_grouped.hip:47-57), read from the same buffer.
template <typename TOUT, typename TS, bool SH, bool PBF16>
__global__ void __launch_bounds__(256)
    combine_reduce_kernel(const float *__restrict__ partial, const int32_t *__restrict__ ids, const float *__restrict__ coef,
                          int64_t M, int64_t A, int64_t E_total, int64_t e_lo, int64_t E_local, int64_t N,
                          TOUT *__restrict__ y, const TS *__restrict__ s, const float *__restrict__ gate_logit,
                          int64_t gate_ld, uint32_t gate_index, uint32_t *err) {
    behind_grid();
    const int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) * 4;
    if (i >= M * N) return;
    const int64_t m = i / N, n = i % N;  // N % 4 == 0: the four columns lie in one row
    float v[4];
    combine_slots<PBF16>(v, partial, ids, coef, m, n, A, E_total, e_lo, E_local, N);
    if constexpr (SH) {
        const float gl = gate_logit[m * gate_ld];
        const bool gok = isfinite(gl);
        if (!gok && n == 0) raise_error(err, (uint32_t)m, gate_index);
        const float gt = gok ? 1.f / (1.f + expf(-gl)) : qnan_f32();
#pragma unroll
        for (int j = 0; j < 4; ++j) v[j] = fmaf(gt, load_as_f32(s, i + j), as_stored<TOUT>(v[j]));
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) store_from_f32(y, i + j, v[j]);
}

// The same reduce for an expert-parallel rank whose rows go to their owners: no shared add, FP32 sums; the four columns
// are stored, as this rank's piece, into the owner's receive buffer through its peer mapping (16 or 8 bytes a store).
template <bool PBF16, bool OUT_F16>
__global__ void __launch_bounds__(256)
    combine_reduce_peer_kernel(const float *__restrict__ partial, const int32_t *__restrict__ ids, const float *__restrict__ coef,
                               int64_t M, int64_t A, int64_t E_total, int64_t e_lo, int64_t E_local, int64_t N, const PeerOut peer) {
    const int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) * 4;
    if (i >= M * N) return;
    const int64_t m = i / N, n = i % N;
    float v[4];
    combine_slots<PBF16>(v, partial, ids, coef, m, n, A, E_total, e_lo, E_local, N);
    const int owner = (int)(m / peer.t);
    const int64_t at = (((int64_t)peer.rank * peer.t + m % peer.t) * N + n);
    if constexpr (OUT_F16) {
        // F16, not BF16: eleven significant bits keep the sum of a row's pieces inside the layer's tolerance (BF16 pieces
        // measured 3.4e-2 of the RMS); a piece beyond F16's range (|v| > 65504) would become infinite
        const __half2 lo = __floats2half2_rn(v[0], v[1]), hi = __floats2half2_rn(v[2], v[3]);
        uint2 o;
        o.x = *reinterpret_cast<const uint32_t *>(&lo), o.y = *reinterpret_cast<const uint32_t *>(&hi);
        *reinterpret_cast<uint2 *>(static_cast<uint16_t *>(peer.base[owner]) + at) = o;
    } else {
        *reinterpret_cast<float4 *>(static_cast<float *>(peer.base[owner]) + at) = make_float4(v[0], v[1], v[2], v[3]);
    }
    // no fence here: the stores have been performed when the kernel has completed, and the rank signals its peers only by
    // work enqueued behind this kernel on the same stream
}

int check_view(const char *fn, const SxbQView *w) {
    SXB_CHECK(w != nullptr, fn, ": null weight view");
    SXB_CHECK(w->q != nullptr && w->scale != nullptr && w->minv != nullptr, fn, ": null weight pointer (q=",
              (const void *)w->q, ", scale=", (const void *)w->scale, ", min=", (const void *)w->minv, ")");
    SXB_CHECK(w->G == 32 || w->G == 64 || w->G == 128, fn, ": group size ", w->G, " unsupported (32, 64 or 128)");
    SXB_CHECK(w->N >= 1 && w->N <= kMaxN, fn, ": N = ", w->N, ", expected 1..", kMaxN);
    SXB_CHECK(w->K >= w->G && w->K <= kMaxK && w->K % w->G == 0, fn, ": K = ", w->K,
              " must be a positive multiple of group size ", w->G, " and <= ", kMaxK);
    SXB_CHECK(aligned16(w->q), fn, ": code array ", (const void *)w->q, " must be 16-byte aligned for vector loads");
    SXB_CHECK(reinterpret_cast<uintptr_t>(w->scale) % 2 == 0 && reinterpret_cast<uintptr_t>(w->minv) % 2 == 0, fn,
              ": scale / min arrays must be 2-byte aligned");
    return SXB_OK;
}

template <int BITS, int G, int MODE, int SRC, typename TOUT>
int launch_stream(const char *fn, const StreamArgs &a, int64_t est_units, cudaStream_t st) {
    using geo = Geo<BITS, G>;
    const int64_t steps = a.K / geo::kStepCodes;
    const int64_t passes = SRC == kPerToken ? (a.A + kTileTokens - 1) / kTileTokens : 1;
    const size_t smem = (size_t)passes * ((size_t)steps * geo::kUnits * 512 + (size_t)steps * kTileTokens * 4);
    SXB_CHECK(smem <= kMaxDynSmem, fn, ": K = ", a.K, SRC == kPerToken ? " x A = " : "", SRC == kPerToken ? a.A : 0, " needs ", smem,
              " bytes of shared memory for one tile's activations, more than ", kMaxDynSmem,
              " (K * 16 * ceil(A / 8) bytes for the per-slot combine, K * 16 otherwise; use the grouped form)");
    StreamArgs args = a;
    // the function's limit is one for all threads of the process: always the largest, not this call's, which would take it from another thread's
    auto reserve = [&](auto k) -> int {
        SXB_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMaxDynSmem), fn, ": reserving shared memory");
        return SXB_OK;
    };
    // Routed tiles of a grouping workspace; rows too long for two buffers go on below.
    if constexpr (SRC == kFromWs) {
        if (kTileBufs * smem <= kMaxDynSmem) {
            auto tiles = stream_tiles_kernel<BITS, G, MODE, TOUT>;
            if (int rc = reserve(tiles)) return rc;
            args.status = reinterpret_cast<uint32_t *>(const_cast<int32_t *>(a.ws)) + 5, args.wait_limit_ns = stream_wait_limit_ns(), args.test_skip_slot = test_skip_slot();
            args.chunks = args.split = 1;
            launch_behind_l1(tiles, (unsigned)sm_count(), kBigThreads, kTileBufs * smem, st, kTileBufs * smem + kCtaExtra, args);
            return SXB_OK;
        }
    }
    auto kern = stream_kernel<BITS, G, MODE, SRC, TOUT>;
    if (int rc = reserve(kern)) return rc;
    // A dense projection of few units for the machine's warps: up to eight warps share one, as long as that gives a warp at most two and a half
    // parts in turn.  A warp alone walks K / (4 * kStepCodes) blocks one after another, each a round trip to memory (2048 x 4096
    // Q4, one token: 16.4 us with 128 warps at work, 9.1 with eight warps a unit).
    const int64_t machine_warps = (int64_t)sm_count() * (kBigThreads / 32);
    args.chunks = SRC == kDense && geo::kStepsPerGroup == 1 && vector_scales(a, G) ? chunk_count(steps / kPrefetch) : 1, args.split = 1;
    if (SRC == kDense)
        while (args.split * 2 <= args.chunks && est_units * args.split * 4 <= machine_warps * 5) args.split *= 2;
    if (args.split > 1) {
        launch_behind(kern, (unsigned)std::min<int64_t>(sm_count(), est_units), kBigThreads, smem, st, 1, args);
        return SXB_OK;
    }
    // One CTA of sixteen warps an SM when there are several units for every warp of the machine; otherwise CTAs of eight
    // warps, two an SM where their shared memory allows, and never more CTAs than one per unit and warp.
    const bool big = est_units >= machine_warps * 2;
    const int threads = big ? kBigThreads : kThreads, warps = threads / 32;
    // Two fit an SM's 228 KB with 1 KB of the system's and their static shared memory each, 25 KB in the dense form (with 100 KB as
    // the line there too, 100 x 4096 x 6144 Q4 ran as two waves of one CTA an SM: 84 us, now 50).
    const int per_sm = big || smem > (SRC == kDense ? 88 : 100) * 1024 ? 1 : 2;
    int64_t grid = (int64_t)sm_count() * per_sm;
    grid = std::max<int64_t>(1, std::min<int64_t>(grid, (est_units + warps - 1) / warps));
    if (SRC == kFromWs) launch_behind_l1(kern, (unsigned)grid, threads, smem, st, per_sm * (smem + kCtaExtra), args);
    else launch_behind(kern, (unsigned)grid, threads, smem, st, 1, args);
    return SXB_OK;
}

template <int BITS, int MODE, int SRC, typename TOUT>
int launch_by_group(const char *fn, const StreamArgs &a, int64_t G, int64_t est_units, cudaStream_t st) {
    switch (G) {
        case 32: return launch_stream<BITS, 32, MODE, SRC, TOUT>(fn, a, est_units, st);
        case 64: return launch_stream<BITS, 64, MODE, SRC, TOUT>(fn, a, est_units, st);
        default: return launch_stream<BITS, 128, MODE, SRC, TOUT>(fn, a, est_units, st);
    }
}

int need_bf16(const char *fn, int act) {
    SXB_CHECK(act_ok(act), fn, ": unsupported activation dtype ", act);
    SXB_CHECK(act == SXB_ACT_BF16, fn,
              ": FP32 activations are not implemented by the sm_100a expert kernels (BF16 activations only)");
    return SXB_OK;
}

// Dense y = x W^T.
template <int BITS>
int linear_impl(const char *fn, const void *x, const SxbQView *w, void *y, int64_t M, int act, int out_act,
                sxb_stream_t stream) {
    SXB_CHECK(x != nullptr && y != nullptr, fn, ": null pointer (x=", x, ", y=", y, ")");
    if (int rc = check_view(fn, w)) return rc;
    SXB_CHECK(M >= 1 && M <= 65535ll * 8, fn, ": M (rows of x) = ", M, ", expected 1..", 65535ll * 8);
    SXB_CHECK(aligned16(x), fn, ": x ", x, " must be 16-byte aligned for vector loads");
    SXB_CHECK(act_ok(act) && (out_act == act || out_act == SXB_ACT_F32), fn, ": output dtype ", act_name(out_act), " with input ",
              act_name(act), " unsupported (same dtype, or BF16 -> F32)");
    if (act == SXB_ACT_F32) {
        SXB_CHECK(apart(x, M * w->K * 4, y, M * w->N * 4), fn, ": output y overlaps input x");
        return f32_gather<BITS>(fn, x, w, 1, nullptr, nullptr, M, 1, y, false, 1, nullptr, stream);
    }
    if (int rc = need_bf16(fn, act)) return rc;
    SXB_CHECK(apart(x, M * w->K * 2, y, M * w->N * act_bytes(out_act)), fn, ": output y [", y, ", +",
              M * w->N * act_bytes(out_act), " B) overlaps input x [", x, ", +", M * w->K * 2, " B)");
    if constexpr (BITS == 8) {
        // The longest row is part of the interface, the same as in the routed forms of the projection, whose tile of eight tokens it comes from;
        // this kernel itself would take a longer one.
        const int64_t tile_bytes = w->K * 16 + w->K / std::min<int64_t>(64, w->G) * kTileTokens * 4;
        SXB_CHECK(tile_bytes <= (int64_t)kMaxDynSmem, fn, ": K = ", w->K, " is longer than the exact-product projections take (G = ", w->G,
                  ": at most ", (int64_t)kMaxDynSmem / (w->G == 32 ? 34 : 33) * 2 / w->G * w->G, ")");
        return dense_q8(fn, x, w, y, M, out_act, static_cast<cudaStream_t>(stream));
    } else {
        StreamArgs a{};
        a.x = static_cast<const uint16_t *>(x), a.q = w->q, a.scale = w->scale, a.minv = w->minv;
        a.N = w->N, a.K = w->K, a.M = M, a.A = 1, a.E = 1, a.out = y;
        const int64_t units = ((M + 7) / 8) * ((w->N + 15) / 16);
        auto st = static_cast<cudaStream_t>(stream);
        int rc = out_act == SXB_ACT_F32 ? launch_by_group<BITS, kGather, kDense, float>(fn, a, w->G, units, st)
                                        : launch_by_group<BITS, kGather, kDense, uint16_t>(fn, a, w->G, units, st);
        if (rc) return rc;
        SXB_CHECK_LAUNCH(fn, " ", act_name(act), "->", act_name(out_act), " M=", M, " N=", w->N, " K=", w->K, " G=", w->G);
        return SXB_OK;
    }
}

int check_experts(const char *fn, const void *x, const SxbQView *w, int64_t E, int64_t M, int64_t A, const void *y) {
    SXB_CHECK(x != nullptr && y != nullptr, fn, ": null pointer (x=", x, ", y=", y, ")");
    if (int rc = check_view(fn, w)) return rc;
    SXB_CHECK(E >= 1 && w->N % E == 0, fn, ": weight has ", w->N, " rows, not a multiple of E = ", E, " experts");
    SXB_CHECK(A >= 1 && A <= 64 && A <= E, fn, ": A (active experts per token) = ", A, ", expected 1..min(64, E=", E, ")");
    SXB_CHECK(aligned16(x), fn, ": input ", x, " must be 16-byte aligned");
    return SXB_OK;
}

// Per-slot gather (optionally with SwiGLU): kernels/linear_q4.hip:420-453.
template <int BITS>
int experts_slots_impl(const char *fn, const void *x, const SxbQView *w, int64_t E, const int32_t *ids, int64_t M,
                       int64_t A, void *y, int act, uint32_t *err, sxb_stream_t stream, bool swiglu) {
    if (int rc = check_experts(fn, x, w, E, M, A, y)) return rc;
    SXB_CHECK(ids != nullptr && err != nullptr, fn, ": null pointer (ids=", (const void *)ids, ", err=", (const void *)err, ")");
    SXB_CHECK(M >= 1 && M <= 65535, fn, ": M (tokens) = ", M, ", expected 1..65535");
    if (act == SXB_ACT_F32) {
        SXB_CHECK(apart(x, M * w->K * 4, y, M * A * (swiglu ? w->N / E / 2 : w->N / E) * 4), fn, ": output overlaps input");
        return f32_gather<BITS>(fn, x, w, E, ids, nullptr, M, A, y, swiglu, (int)A, err, stream);
    }
    if (int rc = need_bf16(fn, act)) return rc;
    const int64_t N = w->N / E;
    SXB_CHECK(!swiglu || N % 2 == 0, fn, ": SwiGLU gather needs an even row count per expert ([gate | up]), got ", N);
    SXB_CHECK(apart(x, M * w->K * 2, y, M * A * (swiglu ? N / 2 : N) * 2), fn, ": output overlaps input");
    StreamArgs a{};
    a.x = static_cast<const uint16_t *>(x), a.q = w->q, a.scale = w->scale, a.minv = w->minv;
    a.N = N, a.K = w->K, a.M = M, a.A = A, a.E = E, a.ids = ids, a.out = y, a.err = err;
    auto st = static_cast<cudaStream_t>(stream);
    const int64_t units = M * A * (swiglu ? (N / 2 + 7) / 8 : (N + 15) / 16);
    int rc = swiglu ? launch_by_group<BITS, kSwiglu, kFromSlots, uint16_t>(fn, a, w->G, units, st)
                    : launch_by_group<BITS, kGather, kFromSlots, uint16_t>(fn, a, w->G, units, st);
    if (rc) return rc;
    SXB_CHECK_LAUNCH(fn, " ", act_name(act), " M=", M, " A=", A, " E=", E, " N=", N, " K=", w->K, " G=", w->G,
                     swiglu ? " swiglu" : "");
    return SXB_OK;
}

int check_grouped(const char *fn, const void *x, const SxbQView *w, int64_t E, int64_t M, int64_t A, const void *ws,
                  size_t ws_bytes, const void *y) {
    if (int rc = check_experts(fn, x, w, E, M, A, y)) return rc;
    SXB_CHECK(ws != nullptr, fn, ": null workspace");
    SXB_CHECK(E <= kMoeMaxExperts && M * A <= kMoeMaxSlots, fn, ": M = ", M, " tokens x A = ", A, " slots over E = ", E,
              " experts (E <= ", kMoeMaxExperts, ", M*A <= ", kMoeMaxSlots, ")");
    SXB_CHECK(ws_bytes >= (size_t)route_words(M, A, E).total * 4, fn, ": workspace of ", ws_bytes, " bytes, needs ",
              route_words(M, A, E).total * 4, " for M = ", M, ", A = ", A, ", E = ", E);
    return SXB_OK;
}

}  // namespace

// The exact-product grouped forms (MoeMath::F32 / WmmaBf16), shared with grouped.cu's dispatch.
template <int BITS>
int stream_gather_grouped(const char *fn, const void *x, const SxbQView *w, int64_t E, const void *ws, size_t ws_bytes,
                          int64_t M, int64_t A, void *y, int act, bool swiglu, sxb_stream_t stream) {
    if (int rc = check_grouped(fn, x, w, E, M, A, ws, ws_bytes, y)) return rc;
    if (act == SXB_ACT_F32) {
        SXB_CHECK(apart(x, M * w->K * 4, y, M * A * (swiglu ? w->N / E / 2 : w->N / E) * 4), fn, ": output overlaps input x");
        return f32_gather<BITS>(fn, x, w, E, nullptr, ws, M, A, y, swiglu, (int)A, nullptr, stream);
    }
    if (int rc = need_bf16(fn, act)) return rc;
    const int64_t N = w->N / E;
    SXB_CHECK(!swiglu || N % 2 == 0, fn, ": gate_up has ", N, " rows an expert, expected an even count (gate rows then up rows)");
    SXB_CHECK(apart(x, M * w->K * 2, y, M * A * (swiglu ? N / 2 : N) * 2), fn, ": output overlaps input x");
    StreamArgs a{};
    a.x = static_cast<const uint16_t *>(x), a.q = w->q, a.scale = w->scale, a.minv = w->minv;
    a.N = N, a.K = w->K, a.M = M, a.A = A, a.E = E, a.ws = static_cast<const int32_t *>(ws), a.L = route_words(M, A, E);
    a.out = y;
    auto st = static_cast<cudaStream_t>(stream);
    const int64_t units = (M * A / 8 + std::min<int64_t>(E, M * A)) * (swiglu ? (N / 2 + 7) / 8 : (N + 15) / 16);
    int rc = swiglu ? launch_by_group<BITS, kSwiglu, kFromWs, uint16_t>(fn, a, w->G, units, st)
                    : launch_by_group<BITS, kGather, kFromWs, uint16_t>(fn, a, w->G, units, st);
    if (rc) return rc;
    SXB_CHECK_LAUNCH(fn, " ", act_name(act), " M=", M, " A=", A, " E=", E, " N=", N, " K=", w->K, " G=", w->G);
    return SXB_OK;
}

template <int BITS>
int stream_partial_grouped(const char *fn, const void *h, const SxbQView *w, int64_t E, const void *ws, size_t ws_bytes,
                           int64_t M, int64_t A, float *partial, int act, sxb_stream_t stream) {
    if (int rc = check_grouped(fn, h, w, E, M, A, ws, ws_bytes, partial)) return rc;
    if (act == SXB_ACT_F32) return f32_gather<BITS>(fn, h, w, E, nullptr, ws, M, A, partial, false, 1, nullptr, stream);
    if (int rc = need_bf16(fn, act)) return rc;
    const int64_t N = w->N / E;
    StreamArgs a{};
    a.x = static_cast<const uint16_t *>(h), a.q = w->q, a.scale = w->scale, a.minv = w->minv;
    a.N = N, a.K = w->K, a.M = M, a.A = A, a.E = E, a.ws = static_cast<const int32_t *>(ws), a.L = route_words(M, A, E);
    a.out = partial;
    auto st = static_cast<cudaStream_t>(stream);
    const int64_t units = (M * A / 8 + std::min<int64_t>(E, M * A)) * ((N + 15) / 16);
    if (int rc = launch_by_group<BITS, kPartial, kFromWs, float>(fn, a, w->G, units, st)) return rc;
    SXB_CHECK_LAUNCH(fn, " partial M=", M, " A=", A, " E=", E, " N=", N, " K=", w->K, " G=", w->G);
    return SXB_OK;
}

// Per-slot combine without scratch (kernels/linear_q4.hpp:44-46).
template <int BITS>
int stream_combine_slots(const char *fn, const void *h, const SxbQView *w, int64_t E, const int32_t *ids,
                         const float *coef, int64_t M, int64_t A, void *y, int act, int out_act, uint32_t *err,
                         sxb_stream_t stream) {
    SXB_CHECK(coef != nullptr, fn, ": null coef");
    if (int rc = check_experts(fn, h, w, E, M, A, y)) return rc;
    SXB_CHECK(ids != nullptr && err != nullptr, fn, ": null pointer (ids=", (const void *)ids, ", err=", (const void *)err, ")");
    SXB_CHECK(M >= 1 && M <= 65535, fn, ": M (tokens) = ", M, ", expected 1..65535");
    SXB_CHECK(act_ok(act) && (out_act == act || out_act == SXB_ACT_F32), fn, ": output dtype ", act_name(out_act), " with activations ",
              act_name(act), " unsupported (same dtype, or F32)");
    if (act == SXB_ACT_F32) {
        SXB_CHECK(apart(h, M * A * w->K * 4, y, M * (w->N / E) * 4), fn, ": output y overlaps input h");
        return f32_combine<BITS>(fn, h, w, E, ids, coef, M, A, y, err, stream);
    }
    if (int rc = need_bf16(fn, act)) return rc;
    const int64_t N = w->N / E;
    SXB_CHECK(apart(h, M * A * w->K * 2, y, M * N * act_bytes(out_act)), fn, ": output y overlaps input h");
    StreamArgs a{};
    a.x = static_cast<const uint16_t *>(h), a.q = w->q, a.scale = w->scale, a.minv = w->minv;
    a.N = N, a.K = w->K, a.M = M, a.A = A, a.E = E, a.ids = ids, a.coef = coef, a.out = y, a.err = err;
    auto st = static_cast<cudaStream_t>(stream);
    const int64_t units = M * ((N + 15) / 16);
    int rc = out_act == SXB_ACT_F32 ? launch_by_group<BITS, kGather, kPerToken, float>(fn, a, w->G, units, st)
                                    : launch_by_group<BITS, kGather, kPerToken, uint16_t>(fn, a, w->G, units, st);
    if (rc) return rc;
    SXB_CHECK_LAUNCH(fn, " ", act_name(act), " M=", M, " A=", A, " E=", E, " N=", N, " K=", w->K, " G=", w->G);
    return SXB_OK;
}

template int stream_combine_slots<4>(const char *, const void *, const SxbQView *, int64_t, const int32_t *, const float *,
                                     int64_t, int64_t, void *, int, int, uint32_t *, sxb_stream_t);
template int stream_combine_slots<8>(const char *, const void *, const SxbQView *, int64_t, const int32_t *, const float *,
                                     int64_t, int64_t, void *, int, int, uint32_t *, sxb_stream_t);

template int stream_gather_grouped<4>(const char *, const void *, const SxbQView *, int64_t, const void *, size_t, int64_t,
                                      int64_t, void *, int, bool, sxb_stream_t);
template int stream_gather_grouped<8>(const char *, const void *, const SxbQView *, int64_t, const void *, size_t, int64_t,
                                      int64_t, void *, int, bool, sxb_stream_t);
template int stream_partial_grouped<4>(const char *, const void *, const SxbQView *, int64_t, const void *, size_t, int64_t,
                                       int64_t, float *, int, sxb_stream_t);
template int stream_partial_grouped<8>(const char *, const void *, const SxbQView *, int64_t, const void *, size_t, int64_t,
                                       int64_t, float *, int, sxb_stream_t);

int combine_reduce(const char *fn, const float *partial, const int32_t *ids, const float *coef, int64_t M, int64_t A,
                   int64_t E_total, int64_t e_lo, int64_t E_local, int64_t N, void *y, int out_act,
                   const SxbMoeSharedAdd *shared, int s_act, bool partial_bf16, sxb_stream_t stream, const PeerOut *peer) {
    if (peer != nullptr) {
        SXB_CHECK(partial != nullptr && ids != nullptr && coef != nullptr, fn, ": null pointer");
        SXB_CHECK(shared == nullptr && N % 4 == 0 && aligned16(partial), fn, ": peer output takes no shared add; N = ", N);
        SXB_CHECK(peer->world >= 1 && peer->world <= 8 && peer->t >= 1 && M == peer->t * peer->world, fn, ": ", M, " rows over ",
                  peer->world, " ranks of ", peer->t);
        const unsigned blocks = (unsigned)((M * N / 4 + 255) / 256);
        auto st = static_cast<cudaStream_t>(stream);
#define SXB_PEER(PB, OB) combine_reduce_peer_kernel<PB, OB><<<blocks, 256, 0, st>>>(partial, ids, coef, M, A, E_total, e_lo, E_local, N, *peer)
        if (partial_bf16) {
            if (peer->f16) SXB_PEER(true, true);
            else SXB_PEER(true, false);
        } else {
            if (peer->f16) SXB_PEER(false, true);
            else SXB_PEER(false, false);
        }
#undef SXB_PEER
        SXB_CHECK_LAUNCH(fn, " reduce to peers M=", M, " A=", A, " N=", N);
        return SXB_OK;
    }
    SXB_CHECK(partial != nullptr && ids != nullptr && coef != nullptr && y != nullptr, fn, ": null pointer (partial=",
              (const void *)partial, ", ids=", (const void *)ids, ", coef=", (const void *)coef, ", y=", y, ")");
    SXB_CHECK(N % 4 == 0 && aligned16(partial), fn, ": N = ", N, " must be a multiple of 4 and partial 16-byte aligned");
    SXB_CHECK(act_ok(out_act), fn, ": unsupported output dtype ", out_act);
    if (shared != nullptr) {
        SXB_CHECK(shared->s != nullptr && shared->gate_logit != nullptr && shared->err != nullptr, fn,
                  ": shared add with a null pointer (s=", shared->s, ", gate_logit=", (const void *)shared->gate_logit,
                  ", err=", (const void *)shared->err, ")");
        SXB_CHECK(shared->gate_ld >= 1, fn, ": shared add gate_ld = ", shared->gate_ld, ", expected >= 1");
        SXB_CHECK(apart(y, M * N * act_bytes(out_act), shared->s, M * N * act_bytes(s_act)), fn, ": y overlaps shared s");
    }
    SXB_CHECK(apart(y, M * N * act_bytes(out_act), partial, M * A * N * 4), fn, ": y overlaps partial");
    const unsigned blocks = (unsigned)((M * N / 4 + 255) / 256);
    auto st = static_cast<cudaStream_t>(stream);
    const float *gl = shared ? shared->gate_logit : nullptr;
    const int64_t gld = shared ? shared->gate_ld : 0;
    const uint32_t gi = shared ? shared->gate_index : 0;
    uint32_t *err = shared ? shared->err : nullptr;
#define SXB_REDUCE_P(TOUT, TS, SH, PB)                                                                                  \
    combine_reduce_kernel<TOUT, TS, SH, PB><<<blocks, 256, 0, st>>>(partial, ids, coef, M, A, E_total, e_lo, E_local, N, \
                                                                    static_cast<TOUT *>(y),                              \
                                                                    static_cast<const TS *>(shared ? shared->s : nullptr), \
                                                                    gl, gld, gi, err)
#define SXB_REDUCE(TOUT, TS, SH)                          \
    do {                                                  \
        if (partial_bf16) SXB_REDUCE_P(TOUT, TS, SH, true); \
        else SXB_REDUCE_P(TOUT, TS, SH, false);            \
    } while (0)
    if (out_act == SXB_ACT_F32) {
        if (!shared) SXB_REDUCE(float, float, false);
        else if (s_act == SXB_ACT_F32) SXB_REDUCE(float, float, true);
        else SXB_REDUCE(float, uint16_t, true);
    } else {
        if (!shared) SXB_REDUCE(uint16_t, uint16_t, false);
        else if (s_act == SXB_ACT_F32) SXB_REDUCE(uint16_t, float, true);
        else SXB_REDUCE(uint16_t, uint16_t, true);
    }
#undef SXB_REDUCE
#undef SXB_REDUCE_P
    SXB_CHECK_LAUNCH(fn, " reduce M=", M, " A=", A, " N=", N, shared ? " +shared" : "");
    return SXB_OK;
}

}  // namespace sxb

using namespace sxb;

extern "C" {

int sxb_linear_q4(const void *x, const SxbQView *w, void *y, int64_t M, int act, int out_act, sxb_stream_t stream) {
    return linear_impl<4>("linear_q4", x, w, y, M, act, out_act, stream);
}
int sxb_linear_q8(const void *x, const SxbQView *w, void *y, int64_t M, int act, int out_act, sxb_stream_t stream) {
    return linear_impl<8>("linear_q8", x, w, y, M, act, out_act, stream);
}

int sxb_linear_q4_experts_gather(const void *x, const SxbQView *w, int64_t E, const int32_t *ids, int64_t M, int64_t A,
                                 void *y, int act, uint32_t *err, sxb_stream_t stream) {
    return experts_slots_impl<4>("linear_q4_experts_gather", x, w, E, ids, M, A, y, act, err, stream, false);
}
int sxb_linear_q4_experts_gather_swiglu(const void *x, const SxbQView *w, int64_t E, const int32_t *ids, int64_t M,
                                        int64_t A, void *h, int act, uint32_t *err, sxb_stream_t stream) {
    return experts_slots_impl<4>("linear_q4_experts_gather_swiglu", x, w, E, ids, M, A, h, act, err, stream, true);
}
int sxb_linear_q8_experts_gather(const void *x, const SxbQView *w, int64_t E, const int32_t *ids, int64_t M, int64_t A,
                                 void *y, int act, uint32_t *err, sxb_stream_t stream) {
    return experts_slots_impl<8>("linear_q8_experts_gather", x, w, E, ids, M, A, y, act, err, stream, false);
}
int sxb_linear_q8_experts_gather_swiglu(const void *x, const SxbQView *w, int64_t E, const int32_t *ids, int64_t M,
                                        int64_t A, void *h, int act, uint32_t *err, sxb_stream_t stream) {
    return experts_slots_impl<8>("linear_q8_experts_gather_swiglu", x, w, E, ids, M, A, h, act, err, stream, true);
}

}  // extern "C"
