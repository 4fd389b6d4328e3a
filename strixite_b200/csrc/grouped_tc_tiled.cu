// The tcgen05 expert GEMM for tile-blocked activations (sxb_stage_f16_tiles, or the h that the SwiGLU form of these
// kernels writes): the MoeMath::WmmaF16 forms of linear_q*_experts_gather_grouped[_swiglu] / _combine_grouped
// (kernels/moe_grouped.hpp:58-91) and the dense linear_q*_wmma projections (kernels/linear_wmma.hpp:23-26) when their
// activations arrive in that form.  Numerics as in grouped_tc.cu (kernels/moe_grouped.hpp:29-38,
// kernels/wmma_gemm.hpp:116-129): F16 operands, weights code * scale + min with one rounding, FP32 accumulation.
//
// Work item: 128 weight rows (a row per tensor-memory lane) x up to 128 tokens of one expert.  k advances in steps of 128.
//
// What bounds it (B200, SM cycles per step, the pieces measured alone): the MMAs take max(305, 4 n) for n tokens (below 76
// tokens reading the A operand bounds them); dequantizing 128 x 128 codes and storing them to tensor memory takes the sixteen
// producer warps 202; the HBM time of the codes is 340 (Q4) or 680 (Q8).  All of it together runs at some 520 a step for 15 tokens
// and 700 for 80 (the times below at 1.9 GHz): every role shares the four schedulers' issue slots and instruction caches, so what counts is
// instructions (584 a step of them the dequantization).  Launches in a row run at the card's power limit, at 15 tokens an expert as at 300: then it is energy.
//   * One lane's MMAs and commits count, but its whole warp runs the loop, under control flow that the compiler can see to be uniform:
//     addresses and descriptors then live in uniform registers.  Run by one lane of a diverged warp the MMAs took no longer to issue, but
//     the loop around them 490 cycles a step (the wait 140, commit and the way back 350): 650 a step at 15 tokens with the stamps
//     that showed it, which bounded every shape.  The scales of the step's own groups and this loop: gate/up 563 -> 540 us at 777
//     tokens, 789 -> 728 at 4096, dense 1001 x 8192 x 4096 64.7 -> 57.1, 4000 tokens Q8 232 -> 216.
//   * Steps of 128 k, eight MMAs a commit: with the loop of one lane a commit and the next stage's wait cost ~250 cycles whatever lay between.
//   * Dequantization is a mask and a multiply-add (dequant_q4_scaled): 146 instructions a warp and step.  The rest of the producers' loop counts as much (with
//     neither copies nor MMAs it took 464 of then 548 us at 777 tokens): arrivals are predicated, not branched to; without SS scales come through pointers that
//     advance, the next item's first ones asked for at the item's start: 410 alone, gate/up 548 -> 506 us.  Asking for barriers a phase ahead or a
//     second quarter dequantized before the stage is free: no faster (+0 to +1 %).
//   * A wait suspends its warp instead of polling; item descriptions come through shared memory (the item ring); the
//     epilogue's pass is 16 tokens, not 32 (shorter code: gate/up 2593 -> 2477 us at 16384 tokens).
//   * Where contractions are short the item counts: eight steps of down against 4500 instructions of epilogue at 80 tokens, 230 a warp and pass, which
//     made it the bound (it worked 6700 of an item's 7300 cycles), and the producers waited for it in an item ring of two.  Output rows through the item
//     ring, shared memory in place of a shuffle a token, gate and up in one thread: down 1900 instructions an item fewer; scan loops that do not unroll: 72 KB of
//     code, now 50.  Under load, us: down with its combine 654 -> 600 at 4096 tokens, 2449 -> 2281 at 16384 (Q8), 353 at 777 either way; gate/up 847 -> 838,
//     2669 -> 2620 and 598 -> 586.  The next item's scales asked into L2 ahead of the scan: gate/up 2 % slower, down no faster.
//   * Scales and mins lie in shared memory where two items' fit, up to 32 groups a row (SS): the item warp reads them anyway.  Producers that each ask for their
//     own row's groups (what is left for longer rows) fetch two bytes from each of 32 sectors a load, as many bytes from L2 as the codes are, and
//     carry pointers and the next item's rows along: 1330 instructions a step against 1140 (gate/up, 15 tokens an expert), for twelve ring slots of Q4 codes
//     against eight.  Under load, us: gate/up 609 -> 582 at 777 tokens, 881 -> 847 at 4096, 2650 -> 2566 at 16384; down with its combine 363 -> 345, 627 -> 613,
//     2348 -> 2309 (Q8); dense 1001 x 8192 x 4096 Q4 61.5 -> 59.0, 4096 x 4096 x 1024 Q8 43.4 -> 38.6.
//   * In down the item warp is the longest chain, 4500 cycles an item: so it asks for the next item's scales, in HBM, before it has published this one (down 361 ->
//     345 at 777 tokens).  A second item warp leaves 72 registers a thread: down 350 -> 336, gate/up 550 -> 562.
// Why 128 tokens: that leaves tensor memory for two accumulators (an item's epilogue runs under the next item's mainloop) and four 64-column
// stages of A.  An expert of more tokens has its rows dequantized again for every 128 of them; a wider tile, which would share that at the price of an
// accumulator or of stages, has not been built.
// Measured, 512 experts, d = 4096, I = 1024, Q4, a few launches at a time: gate/up + SwiGLU 495 us at 777 tokens (15 an expert), 670 at
// 4096 (80 an expert); down 275 and 425 (gathering row-major activations the same products took 1052, 1132, 820 and 861).
//
// SwiGLU: gate row j and up row j are rows of the same accumulator, so they cannot share a lane.  An item holds 64
// gate rows and their 64 up rows; inside every tensor-memory lane quadrant lanes 0-15 are gate rows and lanes 16-31 the up
// rows of the same h columns, and the epilogue reads both in the sixteen-lane form of tcgen05.ld, which gives a thread a gate value
// and its up value.
//
// Operands as in grouped_tc.cu: A (weights) dequantized in registers and stored to tensor memory by the producer warps
// (the [tmem] form of tcgen05.mma), B (activations) two cp.async.bulk per step (one per 64-k sub-tile) into
// 128-byte-swizzled K-major tiles, packed codes by tensor copies (128 codes x 128 rows a box and ring slot).
//
// One persistent CTA per SM.  Warps: the epilogue first (one per lane quadrant; two in the hyper-connection up mix, whose
// epilogue carries the arithmetic of the stream combine - see TcHcUp), then MMA issue, activation copies, the ring of weight
// codes and the item ring, then four sets of four weight producers (a lane quadrant's warps take every fourth step each).  All lanes
// of a producer warp wait on its barriers themselves: a poll by one lane and a reconvergence after it cost more than 32
// lanes reading the same word.  Every wait is bounded: past the limit the CTA raises its abort flag, records
// {2, item, role} in the status words, drains the tensor pipe and frees its tensor memory before returning.  The tensor
// copies read this GPU's own weight array only, each into the shared memory of the one CTA that issues it.

#include "grouped_tc.cuh"

#include <cmath>
#include <type_traits>

namespace sxb {
namespace {

constexpr int kTile = 128;           // tokens per item at most = columns of an accumulator
constexpr int kSubK = 64;            // k of one 128-byte swizzle line of F16
constexpr int kBK = 2 * kSubK;       // k per stage
constexpr int kRows = 128;           // weight rows per item = tensor-memory lanes
constexpr int kSubBytes = kTile * 128;      // activation tile of 64 k
constexpr int kStageBytes = 2 * kSubBytes;  // of a stage
constexpr int kAStageCols = kBK / 2; // 128 F16 of one weight row per lane
constexpr int kAccs = 2;
constexpr int kTmemCols = 512;

constexpr int kScaleGroups = 32;  // SS: groups of a row at most
// ... items whose scales lie in shared memory, as a power of two
__host__ __device__ constexpr int scale_bufs_log(int groups) { return groups <= kScaleGroups / 2 ? 2 : 1; }
constexpr int kScaleBufs = 4;
// kTcHcUp: one buffer of an epilogue warp - a pass's 128 (token, stream) segments of X, 32 bytes each at most, then inv
constexpr int kHcUpBufBytes = 128 * 32 + 32 * 16;
constexpr int kSharedBytes = 227 * 1024;  // of a CTA
constexpr int kStaticBytes = 3 * 1024;    // barriers, item ring and the like at most: the dynamic part starts on the next 1024 bytes behind them

// HC: the hyper-connection up mix (kTcHcUp), whose contraction is short and whose epilogue needs registers and shared memory:
// half the producers, stages and ring slots.
// SS: the scales of the items at hand lie in shared memory.
// A set of four producer warps (one per lane quadrant) owns one stage, and its own ring slots: it meets every barrier it
// waits on again only after it has seen that barrier's previous phase end, so watching the parity is enough.
template <int BITS, bool HC, bool SS>
struct Shape {
    static constexpr int kWays = HC ? 2 : 4;  // producer sets
    static constexpr int kStages = kWays;
    static constexpr int kSlotBytes = kRows * kBK * BITS / 8;  // a ring slot: the packed codes of a step, 8 or 16 KB
    // What shared memory holds beside the stages and the scales.  Without SS Q4 has room for twelve slots (583 -> 572 us at 777 tokens against eight, before SS took
    // that case to eight slots and 548).
    static constexpr int kWSlots = kWays * (HC ? (BITS == 4 ? 4 : 2) : BITS == 8 ? 1 : SS ? 2 : 3);
    // Items that the ring holds.  The epilogue keeps an item's place until it is done with it.  Without SS three, us under load with two / three / four: dense
    // 4096 x 8192 x 4096 Q8 315 / 263 / 272; gate/up of 64 experts, d = 7168, I = 2048, Q4, 4000 tokens 2047 / 1735 / 1768; down of 128 experts,
    // 2560 x 768 Q4, 4000 tokens - / 204 / 196.  A deeper one lets the item warp's look at a later item's scales push those that the producers want out of L1,
    // where rows are long.
    static constexpr int kItemRing = SS ? 4 : 3;
    static constexpr int kEpiSets = HC ? 2 : 1;  // epilogue warps per lane quadrant
    static constexpr int kEpiWarps = 4 * kEpiSets, kMmaWarp = kEpiWarps, kBCopyWarp = kEpiWarps + 1, kWCopyWarp = kEpiWarps + 2,
                         kItemWarp = kEpiWarps + 3, kFirstAWarp = kEpiWarps + 4;
    static constexpr int kThreads = 32 * (kFirstAWarp + 4 * kWays);
    static constexpr int kItemReaders = kEpiWarps + 3 + 4 * kWays;  // warps that read every item from the item ring
    // The dynamic part: stages, ring slots, scales of a launch's longest rows, the up mix's buffers.  With scales of 32 groups the CTA's shared memory is full to
    // the byte, and one more static word past kStaticBytes would have every launch of those forms refused.
    static constexpr int kBufferBytes = kStages * kStageBytes + kWSlots * kSlotBytes + (HC ? kEpiWarps * 2 * kHcUpBufBytes : 0);
    static constexpr int kMostDynamic = kBufferBytes + (SS ? 2 * kScaleGroups * kRows * 4 : 0);
    static_assert(kMostDynamic + kStaticBytes <= kSharedBytes, "shared memory");
    static_assert(kAccs * kTile + kStages * kAStageCols <= kTmemCols, "tensor memory");
    static_assert((kWays & (kWays - 1)) == 0 && kWSlots % kWays == 0, "sets");
};

// The power of two that undoes a row's scale 2^k on its accumulators, 2^(24 - k).  Rows at natural magnitude: scale = -2^24.  The item
// ring holds a scale's biased exponent, 0 for kNatural.
constexpr float kNatural = -0x1p24f;
__host__ __device__ constexpr uint32_t unscale_bits(uint32_t scale_bits) { return ((127u + 24u + 127u) << 23) - scale_bits; }  // past int
static_assert(unscale_bits((127u + 24u) << 23) == 127u << 23 && unscale_bits((127u - 1u) << 23) == (127u + 25u) << 23, "2^(24 - k)");
__device__ inline float scale_of(uint8_t exponent) { return exponent != 0 ? __uint_as_float((uint32_t)exponent << 23) : kNatural; }
__device__ inline float unscale(float scale) { return __uint_as_float(unscale_bits(__float_as_uint(fabsf(scale)))); }

struct Item {
    int bucket, start, cnt;  // expert (bucket E = invalid ids, -1 = no more items), first position in slots[], tokens of the item
    int rb;                  // row block
};

// A role's place in a ring of N barriers and the parity of the phase it is in; steps of at most a turn.
template <int N>
struct Turn {
    int at;
    uint32_t phase;
    __device__ inline void advance(int by) {
        at += by;
        if (at >= N) at -= N, phase ^= 1u;
    }
};

// A row's common power of two is set by its largest group, and weights far below that one's lose bits (dequant_q4_scaled).  With e
// the largest exponent among a row's groups (of the scale, or of the min less 8) and every other group's at most kScaleSpread
// below, nothing is lost: a code's step is a BF16 of eight bits and at least 2^-16, so its last bit is at least 2^-23, above the
// last place of an F16 subnormal, 2^-24.  A quadrant of an item with a row spread wider - columns that a quantizer scaled up on
// purpose - takes its weights at their natural magnitude (dequant_q4_word), unless the common power makes them no smaller than that
// (scales below 2^-9).  Error of the small columns' dots against 64 bits, Q4, groups 2^7 / 2^10 / 2^12 apart: 5.6e-4 / 9.2e-3 /
// 3.4e-2 with the common power of two, 2e-5 at any distance without.
constexpr int kScaleSpread = 6;

template <int MODE>
__device__ inline int row_blocks(const TcArgs &a) {
    return MODE == kTcSwiglu ? (int)((a.N / 2 + kRows / 2 - 1) / (kRows / 2)) : (int)((a.N + kRows - 1) / kRows);
}
// Scales and mins of N groups of a row as the item warp leaves them in shared memory: a word a group, the min above.
template <int N>
struct ScaleWords {
    uint32_t w[N];
    __device__ inline float scale(int g) const { return __uint_as_float(value(g) << 16); }
    __device__ inline float min(int g) const { return __uint_as_float(value(g) & 0xffff0000u); }
    __device__ inline uint32_t value(int g) const {
        uint32_t v = w[0];
#pragma unroll
        for (int i = 1; i < N; ++i) v = g == i ? w[i] : v;
        return v;
    }
};

// Scales and mins (BF16 bits) of N consecutive groups of a row.
template <int N>
struct Scales {
    static constexpr int kWords = (N + 1) / 2;
    uint32_t s[kWords], m[kWords];
    __device__ inline float scale(int g) const { return value(s, g); }
    __device__ inline float min(int g) const { return value(m, g); }
    static __device__ inline float value(const uint32_t (&v)[kWords], int g) {
        uint32_t w = v[0];
#pragma unroll
        for (int i = 1; i < kWords; ++i) w = (g >> 1) == i ? v[i] : w;
        return __uint_as_float((g & 1) ? (w & 0xffff0000u) : (w << 16));
    }
};
template <int N>
__device__ inline void load_groups(uint32_t (&v)[Scales<N>::kWords], const uint16_t *p) {
    if constexpr (N == 1) {
        v[0] = __ldg(p);
    } else if constexpr (N == 2) {
        v[0] = __ldg(reinterpret_cast<const uint32_t *>(p));
    } else {
        const uint2 u = __ldg(reinterpret_cast<const uint2 *>(p));
        v[0] = u.x, v[1] = u.y;
    }
}
// The same one by one: arrays that do not start on a vector's boundary.
template <int N>
__device__ __noinline__ Scales<N> load_scales_each(const uint16_t *sp, const uint16_t *mp) {
    Scales<N> c{};
#pragma unroll
    for (int i = 0; i < N; ++i) c.s[i >> 1] |= (uint32_t)__ldg(sp + i) << (16 * (i & 1)), c.m[i >> 1] |= (uint32_t)__ldg(mp + i) << (16 * (i & 1));
    return c;
}

// A producer lane's step of a quadrant at natural magnitude (kScaleSpread): its row's codes, 16-byte chunk c at `src` ^ 16 c of shared
// memory, with its groups sc -> tensor memory.  Rare, so it is short rather than fast: a quarter at a time,
// read again from shared memory (as a call, or unrolled, it cost the common step registers: 2000 x 8192 x 4096 Q8 133 us, not 129).
template <int BITS, int G, typename SCALES>
__device__ __forceinline__ void natural_step(uint32_t src, uint32_t a_addr, const SCALES &sc) {
    constexpr int kChunkCodes = BITS == 4 ? 32 : 16, kChunks = 32 / kChunkCodes;
#pragma unroll 1
    for (int hc = 0; hc < 4; ++hc) {
        uint4 d[4];
#pragma unroll
        for (int c = 0; c < kChunks; ++c) {
            const uint4 v = ld_shared_v4(src ^ ((uint32_t)(hc * kChunks + c) * 16u));
            const int g = hc * 32 / G;  // 32 codes lie in one group
            const __half2 s2 = __float2half2_rn(sc.scale(g)), m2 = __float2half2_rn(sc.min(g));
            if (BITS == 4) {
                d[0] = dequant_q4_word(v.x, s2, m2), d[1] = dequant_q4_word(v.y, s2, m2);
                d[2] = dequant_q4_word(v.z, s2, m2), d[3] = dequant_q4_word(v.w, s2, m2);
            } else {
                d[2 * c] = dequant_q8_words(v.x, v.y, s2, m2), d[2 * c + 1] = dequant_q8_words(v.z, v.w, s2, m2);
            }
        }
        tc_st16(a_addr + hc * 16, d);
    }
    __syncwarp();
}

template <int BITS, int G, int MODE, bool SS>
__global__ void __launch_bounds__((Shape<BITS, MODE == kTcHcUp, SS>::kThreads), 1)
    tiled_tc_kernel(const TcArgs a, const __grid_constant__ CUtensorMap wmap) {
    using S = Shape<BITS, MODE == kTcHcUp, SS>;
    constexpr int kStages = S::kStages, kWSlots = S::kWSlots, kSlotBytes = S::kSlotBytes, kWays = S::kWays, kEpiSets = S::kEpiSets,
                  kEpiWarps = S::kEpiWarps, kMmaWarp = S::kMmaWarp, kBCopyWarp = S::kBCopyWarp, kWCopyWarp = S::kWCopyWarp,
                  kItemWarp = S::kItemWarp, kFirstAWarp = S::kFirstAWarp, kItemRing = S::kItemRing;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char *const smem = smem_raw;  // 1024-byte aligned, as the operand tiles want it (the swizzle pattern repeats every 1024 bytes)
    __shared__ uint64_t full_bar[kStages], empty_bar[kStages], acc_full[kAccs], acc_empty[kAccs], drain_bar;
    __shared__ uint64_t w_full[kWSlots], w_empty[kWSlots];
    __shared__ uint64_t item_full[kItemRing], item_empty[kItemRing], scales_empty[kScaleBufs];
    __shared__ __align__(16) Item item_ring[kItemRing];
    __shared__ uint8_t row_scale[kItemRing][kRows];
    __shared__ __align__(16) uint32_t out_row[kItemRing][kTile];  // where a token's output row starts, in 16-byte units
    __shared__ uint32_t tmem_base_smem;
    __shared__ int abort_flag;

    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const int n_steps = (int)a.K / kBK, groups = (int)a.K / G, sb_log = scale_bufs_log(groups), sb_mask = (1 << sb_log) - 1;
    const int rbs = row_blocks<MODE>(a);
    const int n_items = (a.dense_M > 0 ? (int)((a.dense_M + a.dense_tile - 1) / a.dense_tile) : a.ws[3]) * rbs;
    // slot (row of the output / of h) at position pos of the slot order; a dense projection's rows are in their own order
    auto slot_at = [&](int pos) -> int { return a.dense_M > 0 ? pos : a.ws[a.L.slots + pos]; };
    volatile int *abort_v = &abort_flag;

    if (threadIdx.x == 0) {
        for (int s = 0; s < kStages; ++s) mbar_init(&full_bar[s], 4 + 1), mbar_init(&empty_bar[s], 1);
        for (int h = 0; h < kAccs; ++h) mbar_init(&acc_full[h], 1), mbar_init(&acc_empty[h], kEpiWarps);
        mbar_init(&drain_bar, 1);
        for (int s = 0; s < kWSlots; ++s) mbar_init(&w_full[s], 1), mbar_init(&w_empty[s], 4);
        for (int s = 0; s < kItemRing; ++s) mbar_init(&item_full[s], 1), mbar_init(&item_empty[s], S::kItemReaders);
        for (int s = 0; s < kScaleBufs; ++s) mbar_init(&scales_empty[s], 4 * kWays);
        abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == kMmaWarp) {  // one warp allocates the CTA's tensor memory (all 512 columns: one CTA per SM)
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_smem)), "r"(kTmemCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();

    auto raise_abort = [&](int item, int role) {
        if (atomicExch(&abort_flag, 1) == 0 && atomicCAS(&a.status[0], 0u, 2u) == 0u) {
            a.status[1] = (uint32_t)item;
            a.status[2] = (uint32_t)role;
        }
    };
    // All 512 columns are this CTA's, so they start at column 0, and the code below says so with constants.
    const bool run = tmem_base_smem == 0 && (smem_u32(smem) & 1023u) == 0;
    if (!run && threadIdx.x == 0) raise_abort(0, 0);
    __syncthreads();

    const uint32_t b_base = smem_u32(smem), w_base = b_base + (uint32_t)(kStages * kStageBytes), s_base = w_base + (uint32_t)(kWSlots * kSlotBytes);
    uint32_t issued = 0;  // ring slots issued by this thread (the ring's only)

    // Item number i of this CTA, from the item ring.  read_item: a whole warp; read_item_one: a single thread.
    const Item no_item{-1, 0, 0, 0};
    auto read_item_one = [&](int i) -> Item {
        if (!mbar_wait(&item_full[i % kItemRing], (uint32_t)(i / kItemRing) & 1u, abort_v, a.wait_limit_ns)) {
            raise_abort(blockIdx.x + i * gridDim.x, 8);
            return no_item;
        }
        const Item it = item_ring[i % kItemRing];
        mbar_arrive(&item_empty[i % kItemRing]);
        return it;
    };
    auto read_item = [&](int i, int p, float &scale) -> Item {  // scale: the power of two of tensor-memory lane p (row_scale)
        const bool ok = mbar_wait(&item_full[i % kItemRing], (uint32_t)(i / kItemRing) & 1u, abort_v, a.wait_limit_ns);
        if (!__all_sync(0xffffffffu, ok)) {
            if (lane == 0) raise_abort(blockIdx.x + i * gridDim.x, 8);
            return no_item;
        }
        const Item it = item_ring[i % kItemRing];
        scale = scale_of(row_scale[i % kItemRing][p]);
        __syncwarp();
        if (lane == 0) mbar_arrive(&item_empty[i % kItemRing]);
        return it;
    };

    // The row of the stacked weight in tensor-memory lane p of an item, -1 past the end of the expert.
    auto row_of = [&](const Item &it, int p) -> int64_t {
        if (MODE == kTcSwiglu) {
            const int64_t I = a.N / 2, j = (int64_t)it.rb * (kRows / 2) + (p >> 5) * 16 + (p & 15);
            return j < I ? (int64_t)it.bucket * a.N + ((p & 16) ? I + j : j) : -1;
        }
        const int64_t rr = (int64_t)it.rb * kRows + p;
        return rr < a.N ? (int64_t)it.bucket * a.N + rr : -1;
    };

    if (!run) {
    } else if (warp >= kFirstAWarp) {
        // ===================== A producers: weights =====================
        // A thread writes one weight row into its own tensor-memory lane; a warp may only touch the lane quadrant
        // warp % 4.  Step number cnt of the CTA, counted across its items, belongs to set cnt % kWays, which works in stage
        // number `set`; the sets are out of step with one another, so that while one waits for a barrier or for its stores
        // the others have the arithmetic pipes.
        const int set = (warp - kFirstAWarp) >> 2, a_quad = warp & 3;
        const int p0 = a_quad * 32 + lane;  // tensor-memory lane = row of the item
        // row of the ring slot that holds this lane's codes: the SwiGLU form's slot is [64 gate rows | 64 up rows]
        const int srow = MODE == kTcSwiglu ? (lane >> 4) * (kRows / 2) + a_quad * 16 + (lane & 15) : p0;
        constexpr int kGroups = kBK / G;             // of a step
        constexpr int kRowBytes = kBK * BITS / 8;    // of a row of a ring slot: 64 or 128
        constexpr int kCodeRegs = kBK * BITS / 128;  // 16-byte chunks of codes per row and step
        constexpr int kWordsPerChunk = BITS == 4 ? 4 : 2;  // runs of eight codes in one of them
        // K is a multiple of 128 and so a row's groups of a step's: where the arrays start decides
        const bool vec_scales = kGroups == 1 || ((reinterpret_cast<uintptr_t>(a.scale) | reinterpret_cast<uintptr_t>(a.minv)) & (2 * kGroups - 1)) == 0;
        // this thread's row inside the first slot; its chunks are swizzled (128-byte mode, 64-byte for rows of 64 bytes), so that chunk c
        // lies at my_w ^ 16 c
        const uint32_t my_w = w_base + (uint32_t)(srow * kRowBytes) + (uint32_t)(kRowBytes == 64 ? (srow >> 1) & 3 : srow & 7) * 16u;
        const uint32_t a_addr = ((uint32_t)(a_quad * 32) << 16) + (uint32_t)(kAccs * kTile + set * kAStageCols);
        const uint32_t signals = lane == 0 ? 1u : 0u;

        // Not SS: scales and mins of a step's groups, fetched one step of the set ahead of use (fetched eight groups at a time, of which a set used a
        // quarter or half, and picked out by selects, they were 5 % of the Q8 forms).  A row past the end of the expert gets zeros: its
        // operand row is then zero whatever codes its lane reads.
        auto load_scales = [&](const uint16_t *sp, const uint16_t *mp) {
            Scales<kGroups> c{};
            if (vec_scales) load_groups<kGroups>(c.s, sp), load_groups<kGroups>(c.m, mp);
            else c = load_scales_each<kGroups>(sp, mp);
            return c;
        };
        auto scales_at = [&](int wrow, int step) {
            const int64_t at = (int64_t)wrow * groups + step * kGroups;
            return wrow < 0 ? Scales<kGroups>{} : load_scales(a.scale + at, a.minv + at);
        };
        auto wait = [&](uint64_t *bar, uint32_t parity, int i, int role) {
            if (mbar_wait(bar, parity, abort_v, a.wait_limit_ns)) return true;
            raise_abort(blockIdx.x + i * gridDim.x, role);
            return false;
        };
        uint32_t free_phase = 1u;  // parity of the phase that leaves the stage to the set's next step: there is none before the first
        Turn<kWSlots> slot{set, 0u};
        int st = set;  // the set's next step, relative to the item at hand
        bool live = true;
        // The step whose codes come into slot.at next, of item number i: sc its groups, scale and scale_min the row's power of two.
        auto fill_stage = [&](const auto &sc, float scale, float scale_min, bool natural, int i) {
            bool ok = wait(&w_full[slot.at], slot.phase, i, 7);
            const uint32_t src = my_w + slot.at * (uint32_t)kSlotBytes;
            uint4 code[kCodeRegs];
#pragma unroll
            for (int c = 0; c < kCodeRegs; ++c) code[c] = ld_shared_v4(src ^ ((uint32_t)c << 4));
            __half2 s2[kGroups], s16[kGroups], m2[kGroups];
#pragma unroll
            for (int gi = 0; gi < kGroups; ++gi) {
                s2[gi] = __float2half2_rn(sc.scale(gi) * scale), m2[gi] = __float2half2_rn(sc.min(gi) * scale_min);
                s16[gi] = __hmul2(s2[gi], __float2half2_rn(0.0625f));
            }
            // 32 codes of the row -> 32 F16 = 16 tensor-memory columns of this lane
            auto quarter = [&](int hc, uint4 (&d)[4]) {
#pragma unroll
                for (int cc = 0; cc < 4; ++cc) {
                    const int gi = ((hc * 4 + cc) * 8) / G;
                    const uint4 v = code[(hc * 4 + cc) / kWordsPerChunk];
                    if (BITS == 4) d[cc] = dequant_q4_scaled(cc == 0 ? v.x : cc == 1 ? v.y : cc == 2 ? v.z : v.w, s2[gi], s16[gi], m2[gi]);
                    else d[cc] = (cc & 1) ? dequant_q8_scaled(v.z, v.w, s2[gi], m2[gi]) : dequant_q8_scaled(v.x, v.y, s2[gi], m2[gi]);
                }
            };
            uint4 d[4];
            quarter(0, d);
            ok = wait(&empty_bar[set], free_phase, i, 1) && ok;
            // reconverges the warp; a wait that gave up in any lane ends the warp's work
            if (!__all_sync(0xffffffffu, ok)) {
                live = false;
                return;
            }
            tc_fence_after();  // the stores below come after the MMAs that freed the stage
            if (!natural) {
                mbar_arrive_if(signals, &w_empty[slot.at]);  // the codes are in registers: the slot may be refilled
                tc_st16(a_addr, d);
#pragma unroll
                for (int hc = 1; hc < 4; ++hc) {
                    quarter(hc, d);
                    tc_st16(a_addr + hc * 16, d);
                }
            } else {
                natural_step<BITS, G>(src, a_addr, sc);
                mbar_arrive_if(signals, &w_empty[slot.at]);
            }
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            tc_fence_before();  // orders the stores before the MMAs that read them across the barrier
            __syncwarp();
            mbar_arrive_if(signals, &full_bar[set]);
            free_phase ^= 1u;
        };
        if constexpr (SS) {
            // A row's scales come from shared memory; rows past the end of the expert have some other row's: their sums are dropped.
            for (int i = 0; live; ++i) {
                float scale = 1.f;
                const Item it = read_item(i, p0, scale);
                if (it.bucket < 0) break;
                if (it.bucket < a.E) {
                    const float scale_min = scale * 0x1p-24f;
                    const bool natural = __any_sync(0xffffffffu, scale < 0.f);  // the quadrant's rows share it
                    uint32_t at = s_base + (uint32_t)(((i & sb_mask) * groups + st * kGroups) * kRows + p0) * 4u;
                    for (; st < n_steps && live; st += kWays, slot.advance(kWays), at += kWays * kGroups * kRows * 4) {
                        ScaleWords<kGroups> sc;
#pragma unroll
                        for (int g = 0; g < kGroups; ++g) sc.w[g] = ld_shared_u32(at + g * kRows * 4);
                        fill_stage(sc, scale, scale_min, natural, i);
                    }
                    st -= n_steps;
                }
                __syncwarp();
                mbar_arrive_if(signals, &scales_empty[i & sb_mask]);
            }
        } else {
            float nxt_scale = 1.f;
            Item nxt = read_item(0, p0, nxt_scale);
            int row = nxt.bucket >= 0 && nxt.bucket < a.E ? (int)row_of(nxt, p0) : -1;
            Scales<kGroups> sc_nxt = scales_at(st < n_steps ? row : -1, st);  // of the set's next step
            for (int i = 0; nxt.bucket >= 0 && live; ++i) {
                const Item it = nxt;
                const float scale = nxt_scale, scale_min = scale * 0x1p-24f;
                nxt = read_item(i + 1, p0, nxt_scale);
                const int nxt_row = nxt.bucket >= 0 && nxt.bucket < a.E ? (int)row_of(nxt, p0) : -1;
                if (it.bucket >= a.E) {
                    row = nxt_row, sc_nxt = scales_at(st < n_steps ? row : -1, st);
                    continue;
                }
                const bool natural = __any_sync(0xffffffffu, scale < 0.f);  // the quadrant's rows share it
                // The set's first step of the next item, if it has one there: its scales are asked for at this item's start, but for four groups (registers)
                // and for gate/up of Q8, which HBM bounds: 512 experts x 4096 x 2048, 256 tokens 929 us so and 889 at the end, 500 940 and 899.
                constexpr bool kEarly = kGroups < 4 && !(BITS == 8 && MODE == kTcSwiglu);
                const int after = st + (max(n_steps - st, 0) + kWays - 1) / kWays * kWays - n_steps;
                Scales<kGroups> sc_item{};
                if (kEarly) sc_item = scales_at(after < n_steps ? nxt_row : -1, after);
                const uint16_t *sp = a.scale + (int64_t)max(row, 0) * groups + (st + kWays) * kGroups, *mp = a.minv + (sp - a.scale);
                for (; st < n_steps; st += kWays, slot.advance(kWays), sp += kWays * kGroups, mp += kWays * kGroups) {
                    const Scales<kGroups> sc = sc_nxt;
                    if (row >= 0 && st + kWays < n_steps) sc_nxt = load_scales(sp, mp);
                    fill_stage(sc, scale, scale_min, natural, i);
                    if (!live) break;
                }
                if (!kEarly) sc_item = scales_at(after < n_steps ? nxt_row : -1, after);
                st -= n_steps, row = nxt_row, sc_nxt = sc_item;
            }
        }
    } else if (warp == kItemWarp) {
        // ===================== the item ring =====================
        // One warp looks the CTA's items up ahead of everyone else: the other roles read an item's description from shared
        // memory instead of each walking two dependent loads of the grouping workspace per item.  It also finds each
        // row's power of two (dequant_q4_scaled) from the row's scales and mins, four rows a lane, and whether one suits the rows of
        // a tensor-memory quadrant at all (kScaleSpread); the scales go to shared memory on the way (SS), or are in L2 when the producers want
        // them.  Where contractions are short this is the longest chain of an item: its instructions count.
        const bool vec_scales = groups % 8 == 0 && ((reinterpret_cast<uintptr_t>(a.scale) | reinterpret_cast<uintptr_t>(a.minv)) & 15) == 0;
        const bool pair_scales = groups % 2 == 0 && ((reinterpret_cast<uintptr_t>(a.scale) | reinterpret_cast<uintptr_t>(a.minv)) & 3) == 0;
        // What it needs to know of an item takes two loads, the second from where the first says: the first one for the next item is under way while
        // this one's scales are looked at.
        const int tiles_by = (int)gridDim.x / rbs, rbs_by = (int)gridDim.x % rbs;
        int tile = (int)blockIdx.x / rbs, rb = (int)blockIdx.x % rbs;
        auto look_up = [&](Item &x) {
            x.rb = rb;
            if (a.dense_M > 0) x.bucket = 0, x.start = tile * a.dense_tile;  // dense projection: tile t holds rows dense_tile * t .. of the one group
            else x.bucket = a.ws[a.L.t128_bucket + tile], x.start = a.ws[a.L.t128_start + tile];
            tile += tiles_by, rb += rbs_by;
            if (rb >= rbs) rb -= rbs, ++tile;
        };
        auto count_of = [&](const Item &x) {
            return a.dense_M > 0 ? (int)min((int64_t)a.dense_tile, a.dense_M - x.start) : min(kTile, a.ws[a.L.offsets + x.bucket + 1] - x.start);
        };
        const int64_t row_bytes = MODE == kTcSwiglu ? a.N : a.N * (MODE == kTcPartial ? 4 : 2);  // of the output
        const bool rows_wanted = MODE != kTcHcUp && !(MODE == kTcSwiglu && a.out_f16 >= 3);  // the tile-blocked h follows from the positions
        // SwiGLU without SS: its four registers of slots are asked for behind the scan of the scales.  Held across it they made ptxas spill (Q8, groups of 64: 108
        // bytes a thread), and local memory then took the L1 lines that the producers find their scales in: gate/up of 512 experts, d = 4096, I = 1024, Q8,
        // 300 tokens 1004-1062 us under load, 839-916 so (853-917 before slots were looked up here); 4096 x 8192 x 4096 Q8 + SwiGLU 274 -> 261 (257).
        constexpr bool kSlotsLate = !SS && MODE == kTcSwiglu;
        // The scans without SS stand in front of a launch's first step: two loads of eight groups, two of two or four of one are under way for each of four rows.  A few
        // launches at a time, us, one load -> so:
        // by twos dense 1500 x 2048 x 2816 Q4 24.7 -> 23.8, by ones 64 x 4096 x 1408 Q8 12.4 -> 11.6, 300 x 4096 x 1920 Q4 13.6 -> 12.5; by eights the down half of
        // the hyper-connection mix, 77 tokens, d = 4096, rank 320, 32.8 -> 30.8, dense 4096 x 8192 x 4096 Q8 under load 283 -> 272.
        // Waits until the producers are done with the item that had item i's place for scales.  Once an item, whether it needs the place or not: only then is
        // watching the parity enough.
        auto scales_free = [&](int i) {
            const bool ok = i <= sb_mask || mbar_wait(&scales_empty[i & sb_mask], ((uint32_t)(i >> sb_log) & 1u) ^ 1u, abort_v, a.wait_limit_ns);
            if (__all_sync(0xffffffffu, ok)) return true;
            if (lane == 0) raise_abort(blockIdx.x + i * gridDim.x, 9);
            return false;
        };
        int64_t at[4];  // of an item's rows r * 32 + lane: where their scales start; lanes past the expert's end look at a row that exists
        uint4 sv[4], mv[4];
        auto find_rows = [&](const Item &x) {
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const int64_t wrow = row_of(x, r * 32 + lane);
                at[r] = (wrow < 0 ? row_of(x, 0) : wrow) * groups;
            }
        };
        auto ask = [&](int g) {
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                sv[r] = __ldg(reinterpret_cast<const uint4 *>(a.scale + at[r] + g));
                mv[r] = __ldg(reinterpret_cast<const uint4 *>(a.minv + at[r] + g));
            }
        };
        Item nxt = no_item;
        if ((int)blockIdx.x < n_items) look_up(nxt), nxt.cnt = count_of(nxt);
        if (SS && nxt.bucket >= 0 && nxt.bucket < a.E) find_rows(nxt), ask(0);
        for (int i = 0;; ++i) {
            const Item it = nxt;
            const int item = blockIdx.x + i * gridDim.x;
            const bool more = item + (int)gridDim.x < n_items;
            nxt = no_item;
            if (more) look_up(nxt);
            int slot[4] = {0, 0, 0, 0};
            auto find_slots = [&] {
                if (!rows_wanted || it.bucket < 0) return;
#pragma unroll
                for (int r = 0; r < 4; ++r) slot[r] = r * 32 + lane < it.cnt ? slot_at(it.start + r * 32 + lane) : 0;
            };
            if (!kSlotsLate) find_slots();
            // Of every group v = max(|scale| * 2^8, |min|) as BF16 bits, 0x400 = an empty group; two 16-bit maxima of v, and signed
            // minima of v + 0x7bff, in which an empty group's is the largest.  Five instructions for two groups.
            uint32_t top[4] = {0u, 0u, 0u, 0u}, low[4] = {0x7fff7fffu, 0x7fff7fffu, 0x7fff7fffu, 0x7fff7fffu};
            auto take = [&](int r, uint32_t s, uint32_t m) {
                const uint32_t v = __viaddmax_u16x2(s & 0x7fff7fffu, 0x04000400u, m & 0x7fff7fffu);
                top[r] = __vmaxu2(top[r], v), low[r] = __viaddmin_s16x2(v, 0x7bff7bffu, low[r]);
            };
            if (it.bucket >= 0 && it.bucket < a.E) {
                if (!SS) find_rows(it);
                if (SS) {
                    if (!scales_free(i)) break;
                    uint32_t to = s_base + (uint32_t)((i & sb_mask) * groups * kRows + lane) * 4u;
#pragma unroll 1
                    for (int g = 0;; to += 8 * kRows * 4) {
#pragma unroll
                        for (int r = 0; r < 4; ++r) {
                            auto two = [&](int k, uint32_t s, uint32_t m) {
                                take(r, s, m);
                                st_shared_u32(to + (2 * k * kRows + r * 32) * 4, __byte_perm(s, m, 0x5410));
                                st_shared_u32(to + ((2 * k + 1) * kRows + r * 32) * 4, __byte_perm(s, m, 0x7632));
                            };
                            two(0, sv[r].x, mv[r].x), two(1, sv[r].y, mv[r].y), two(2, sv[r].z, mv[r].z), two(3, sv[r].w, mv[r].w);
                        }
                        if ((g += 8) >= groups) break;
                        ask(g);
                    }
                } else if (vec_scales) {
#pragma unroll 2
                    for (int g = 0; g < groups; g += 8) {
                        ask(g);
#pragma unroll
                        for (int r = 0; r < 4; ++r)
                            take(r, sv[r].x, mv[r].x), take(r, sv[r].y, mv[r].y), take(r, sv[r].z, mv[r].z), take(r, sv[r].w, mv[r].w);
                    }
                } else if (pair_scales) {
#pragma unroll 2
                    for (int g = 0; g < groups; g += 2)
#pragma unroll
                        for (int r = 0; r < 4; ++r)
                            take(r, __ldg(reinterpret_cast<const uint32_t *>(a.scale + at[r] + g)), __ldg(reinterpret_cast<const uint32_t *>(a.minv + at[r] + g)));
                } else {
#pragma unroll 4
                    for (int g = 0; g < groups; ++g)
#pragma unroll
                        for (int r = 0; r < 4; ++r) take(r, __ldg(a.scale + at[r] + g), __ldg(a.minv + at[r] + g));
                }
            } else if (SS && it.bucket >= 0) {
                if (!scales_free(i)) break;
            }
            if (kSlotsLate) find_slots();
            if (more) nxt.cnt = count_of(nxt);
            if (SS && nxt.bucket >= 0 && nxt.bucket < a.E) find_rows(nxt), ask(0);  // from HBM, under what is left to do here
            if (i >= kItemRing) {
                const bool ok = mbar_wait(&item_empty[i % kItemRing], ((uint32_t)(i / kItemRing) & 1u) ^ 1u, abort_v, a.wait_limit_ns);
                if (!__all_sync(0xffffffffu, ok)) {
                    if (lane == 0) raise_abort(item, 9);
                    break;
                }
            }
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                // e: the exponent of the row's largest scale (or min less 8), kept where 2^(14 - e) is a float; that power takes every
                // scale below 2^15 and every min, after its further 2^-24, below 1/2.  e_low: the smallest group's.
                const int hi = (int)max(top[r] >> 16, top[r] & 0xffffu), lo = min((int)low[r] >> 16, (int)(int16_t)low[r]);
                const int e = min(max((hi >> 7) - 8, 127 - 24), 127 + 15), e_low = (((lo - 0x7bff) & 0xffff) >> 7) - 8;
                const bool spread = __any_sync(0xffffffffu, e > 127 - 10 && lo != 0x7fff && e_low < e - kScaleSpread);
                row_scale[i % kItemRing][r * 32 + lane] = spread ? 0 : (uint8_t)(127 + 14 + 127 - e);
                if (rows_wanted) out_row[i % kItemRing][r * 32 + lane] = (uint32_t)(((int64_t)slot[r] * row_bytes) >> 4);
            }
            if (lane == 0) item_ring[i % kItemRing] = it;
            __syncwarp();
            if (lane == 0) mbar_arrive(&item_full[i % kItemRing]);
            if (it.bucket < 0) break;
        }
    } else if (warp == kWCopyWarp) {
        // ===================== the ring of weight codes =====================
        // The ring is kept as far ahead as free slots allow, a box of codes a slot: 128 consecutive rows (the SwiGLU form: 64 gate rows and
        // their 64 up rows).  Q4, whose steps are short: a whole warp's loop with one lane's copies, as the MMA warp's, and the next slot asked for under
        // this one's copy.  One thread's loop took 400 of a step's 540 cycles; us under load, that -> this: gate/up 548 -> 532 at 777 tokens, 468 -> 450
        // at 300, down with its combine 325 -> 320 and 265 -> 259.  Q8's step has twice the time, and its down went 442 -> 448: one thread.
        // test hook: CTA 0 leaves one slot unfilled (neither the byte count nor the copy), so that its consumers' wait runs out at the launch's
        // limit and the abort path is exercised without anything faulting
        if constexpr (BITS == 4) {
            const uint32_t leader = elect_one() ? 1u : 0u;
            Turn<kWSlots> turn{0, 0u};
            bool ok = true, ready = false;
            for (int i = 0; ok; ++i) {
                float unused;
                const Item it = read_item(i, lane, unused);
                if (__any_sync(0xffffffffu, it.bucket < 0)) break;
                if (__any_sync(0xffffffffu, it.bucket >= a.E)) continue;
                const int y = (int)__reduce_max_sync(0xffffffffu, (uint32_t)(MODE == kTcSwiglu ? it.rb * (kRows / 2) : (int)(it.bucket * a.N + (int64_t)it.rb * kRows)));
                const int z = MODE == kTcSwiglu ? (int)__reduce_max_sync(0xffffffffu, (uint32_t)(2 * it.bucket)) : 0;
                for (int step = 0; step < n_steps; ++step) {
                    if (!__all_sync(0xffffffffu, ready)) {
                        ok = __all_sync(0xffffffffu, mbar_wait(&w_empty[turn.at], turn.phase ^ 1u, abort_v, a.wait_limit_ns));
                        if (!ok) {
                            if (leader) raise_abort(blockIdx.x + i * gridDim.x, 6);
                            break;
                        }
                    }
                    uint64_t *full = &w_full[turn.at];
                    const uint32_t dst = w_base + (uint32_t)(turn.at * kSlotBytes);
                    turn.advance(1);
                    ready = mbar_test(&w_empty[turn.at], turn.phase ^ 1u);
                    if (!(blockIdx.x == 0 && (int)issued == a.test_skip_slot)) {
                        mbar_expect_tx_if(leader, full, (uint32_t)kSlotBytes);
                        if (MODE == kTcSwiglu) tma_load_3d_if(leader, dst, &wmap, step * (kBK * BITS / 8), y, z, full);
                        else tma_load_2d_if(leader, dst, &wmap, step * (kBK * BITS / 8), y, full);
                    }
                    ++issued;
                }
            }
        } else {
            if (elect_one()) {
                bool ok = true;
                Turn<kWSlots> turn{0, 0u};
                for (int i = 0; ok; ++i) {
                    const Item it = read_item_one(i);
                    if (it.bucket < 0) break;
                    if (it.bucket >= a.E) continue;
                    const int y = MODE == kTcSwiglu ? it.rb * (kRows / 2) : (int)(it.bucket * a.N + (int64_t)it.rb * kRows);
                    for (int step = 0; step < n_steps; ++step) {
                        const int slot = turn.at;
                        if (!mbar_wait(&w_empty[slot], turn.phase ^ 1u, abort_v, a.wait_limit_ns)) {
                            raise_abort(blockIdx.x + i * gridDim.x, 6);
                            ok = false;
                            break;
                        }
                        const uint32_t dst = w_base + (uint32_t)(slot * kSlotBytes);
                        if (!(blockIdx.x == 0 && (int)issued == a.test_skip_slot)) {
                            mbar_expect_tx(&w_full[slot], (uint32_t)kSlotBytes);
                            if (MODE == kTcSwiglu) tma_load_3d(dst, &wmap, step * (kBK * BITS / 8), y, 2 * it.bucket, &w_full[slot]);
                            else tma_load_2d(dst, &wmap, step * (kBK * BITS / 8), y, &w_full[slot]);
                        }
                        ++issued, turn.advance(1);
                    }
                }
            }
            __syncwarp();
        }
    } else if (warp == kBCopyWarp) {
        // ===================== activations =====================
        // One thread, two bulk copies per step: the tile of (item, 64 k) is one contiguous run of cnt * 128 bytes;
        // completion is counted in bytes on the stage's barrier, and every free stage is refilled at once.
        if (elect_one()) {
            uint32_t count = 0;
            bool ok = true;
            const int64_t line = a.L.S * 128;  // bytes from one 64-k sub-tile to the next
            for (int i = 0; ok; ++i) {
                const Item it = read_item_one(i);
                if (it.bucket < 0) break;
                if (it.bucket >= a.E) continue;
                const uint32_t bytes = (uint32_t)it.cnt * 128u;
                const unsigned char *src = reinterpret_cast<const unsigned char *>(a.x) + (int64_t)it.start * 128;
                for (int st = 0; st < n_steps; ++st, ++count, src += 2 * line) {
                    const uint32_t stage = count % kStages;
                    if (!mbar_wait(&empty_bar[stage], ((count / kStages) & 1u) ^ 1u, abort_v, a.wait_limit_ns)) {
                        raise_abort(blockIdx.x + i * gridDim.x, 5);
                        ok = false;
                        break;
                    }
                    const uint32_t dst = b_base + stage * (uint32_t)kStageBytes;
                    mbar_expect_tx(&full_bar[stage], 2 * bytes);
                    bulk_g2s(dst, src, bytes, &full_bar[stage]);
                    bulk_g2s(dst + kSubBytes, src + line, bytes, &full_bar[stage]);
                }
            }
        }
        __syncwarp();
    } else if (warp == kMmaWarp) {
        // ===================== MMA issue =====================
        // The whole warp runs the loop under control flow that is known to be uniform (votes and a reduction of what came through shared
        // memory), so that addresses and descriptors stay in uniform registers; one lane's MMAs and commits count.  Whether the next
        // step's operands are there is asked before this step's MMAs are issued: the answer comes under them.
        const uint32_t leader = elect_one() ? 1u : 0u;
        const uint64_t desc0 = smem_desc(b_base);
        const uint32_t b_lo0 = (uint32_t)desc0, b_hi = (uint32_t)(desc0 >> 32), at0 = (uint32_t)(kAccs * kTile);
        uint32_t b_lo = b_lo0, at = at0;
        Turn<kStages> turn{0, 0u};
        int done = 0;  // the stage of the step at hand
        uint32_t acc_count = 0;
        bool ok = true;
        for (int i = 0; ok; ++i) {
            float unused;
            const Item it = read_item(i, lane, unused);
            if (__any_sync(0xffffffffu, it.bucket < 0)) break;
            if (__any_sync(0xffffffffu, it.bucket >= a.E)) continue;
            const uint32_t idesc = __reduce_max_sync(0xffffffffu, instr_desc((it.cnt + 15) & ~15));
            const uint32_t half = acc_count & 1u;  // the accumulators take turns
            ok = __all_sync(0xffffffffu, mbar_wait(&acc_empty[half], ((acc_count >> 1) & 1u) ^ 1u, abort_v, a.wait_limit_ns));
            if (!ok) {
                if (leader) raise_abort(blockIdx.x + i * gridDim.x, 2);
                break;
            }
            ++acc_count;
            tc_fence_after();
            const uint32_t d = half * (uint32_t)kTile;
            bool ready = false;
            for (int st = 0; st < n_steps; ++st) {
                if (!__all_sync(0xffffffffu, ready)) {
                    ok = __all_sync(0xffffffffu, mbar_wait(&full_bar[turn.at], turn.phase, abort_v, a.wait_limit_ns));
                    if (!ok) {
                        if (leader) raise_abort(blockIdx.x + i * gridDim.x, 3);
                        break;
                    }
                }
                tc_fence_after();
                turn.advance(1);
                ready = mbar_test(&full_bar[turn.at], turn.phase);
                tc_step_ts<kSubBytes>(leader, d, at, b_lo, b_hi, idesc, st != 0);
                tc_commit_if(leader, &empty_bar[done]);  // the stage is free when these MMAs have read it
                done = (done + 1) % kStages;
                at += kAStageCols, b_lo += kStageBytes / 16;
                if (turn.at == 0) at = at0, b_lo = b_lo0;
            }
            if (ok) tc_commit_if(leader, &acc_full[half]);
        }
        // Drain: every MMA issued by this CTA has completed before tensor memory is released.
        // (this wait does not give up when the CTA is aborting: tensor memory must not be released under an MMA)
        tc_commit_if(leader, &drain_bar);
        mbar_wait(&drain_bar, 0u, nullptr, a.wait_limit_ns);
        __syncwarp();
    } else if (MODE == kTcHcUp && warp < kEpiWarps) {
        // ===================== epilogue of the hyper-connection up mix =====================
        // Lane = (stream s = lane & 3, output column j): per token it needs one activation X[t, s d + j] and inv[t, s].
        // Loads into registers would stall the in-order issue once per token, so a pass's 32 tokens x 4 streams x 8 columns
        // of X and 32 x 4 of inv come through shared memory by 16-byte asynchronous copies (no registers held), issued one
        // pass ahead - across items too - into the warp's own double buffer.  Same hand-overs with the MMA warp as below.
        if constexpr (MODE == kTcHcUp) {
            // The activation dtype is a compile-time constant of the loops (one instantiation each): a run-time choice
            // between two loads per token would put a branch between the tokens, and their chains would not overlap.
            auto run = [&](auto f32_tag) {
                constexpr bool kF32 = decltype(f32_tag)::value;
                constexpr int es = kF32 ? 4 : 2, seg = 8 * es;  // bytes of a (token, stream) segment: this quadrant's 8 columns
                constexpr int kPieces = (128 * seg / 16) / 32;   // 16-byte copies per lane and pass
                using TX = typename std::conditional<kF32, float, uint16_t>::type;
                const TcHcUp &hc = a.hc;
                uint32_t acc_count = 0, pass_count = 0;
                const int quad = warp & 3, s = lane & 3, jj = lane >> 2;
                const int col_lo = (warp >> 2) * (kTile / kEpiSets);
                const uint32_t lane_addr = (uint32_t)(quad * 32) << 16;
                const int64_t row_bytes = 4 * hc.d * es;  // a token's four streams
                unsigned char *my_buf = smem + kStages * kStageBytes + kWSlots * kSlotBytes + warp * (2 * kHcUpBufBytes);
                // Copy number k of a pass: piece p = 32 k + lane of the pass's [token][stream][part] order, i.e. token
                // k * (8 / parts) + tok_l, stream str_l, part part_l with parts = seg / 16.
                constexpr int kParts = seg / 16, kTokStep = 8 / kParts;
                const int part_l = lane % kParts, str_l = (lane / kParts) & 3, tok_l = lane / (4 * kParts);
                auto issue = [&](const Item &it, int c0, int col_hi, unsigned char *buf) {
                    const unsigned char *src = static_cast<const unsigned char *>(hc.x) + ((int64_t)it.rb * 32 + quad * 8 + (int64_t)str_l * hc.d) * es +
                                               part_l * 16 + (int64_t)(it.start + c0 + tok_l) * row_bytes;
                    const uint32_t dst = smem_u32(buf) + (uint32_t)lane * 16u;
#pragma unroll
                    for (int k = 0; k < kPieces; ++k)
                        if (c0 + k * kTokStep + tok_l < col_hi) cp_async16(dst + (uint32_t)k * 512u, src + (int64_t)(k * kTokStep) * row_bytes);
                    if (c0 + lane < col_hi) cp_async16(smem_u32(buf) + 128 * 32 + (uint32_t)lane * 16u, hc.inv + (int64_t)(it.start + c0 + lane) * 4);
                    cp_async_commit();
                };
                auto col_hi_of = [&](const Item &it) { return min(it.cnt, col_lo + kTile / kEpiSets); };
                float itn_scale = 1.f;
                Item itn = read_item(0, quad * 32 + lane, itn_scale);
                if (itn.bucket >= 0) issue(itn, col_lo, col_hi_of(itn), my_buf);
                for (int i = 0; itn.bucket >= 0; ++i) {
                    const Item it = itn;
                    // sigmoid(z) = 1 / (1 + 2^(-z log2 e)), with the row's power of two taken out of z on the way
                    const float nz = -1.44269504f * unscale(itn_scale);
                    itn = read_item(i + 1, quad * 32 + lane, itn_scale);
                    const int item = blockIdx.x + i * gridDim.x;
                    const int64_t j = (int64_t)it.rb * 32 + quad * 8 + jj;
                    const float nwp = 1.0f + __ldg(hc.norm_w + (int64_t)s * hc.d + j);
                    const int col_hi = col_hi_of(it);
                    const uint32_t half = acc_count % kAccs, acc_phase = (acc_count / kAccs) & 1u;
                    ++acc_count;
                    if (lane == 0 && !mbar_wait(&acc_full[half], acc_phase, abort_v, a.wait_limit_ns)) raise_abort(item, 4);
                    __syncwarp();
                    if (*abort_v) break;
                    tc_fence_after();
                    if (col_lo >= col_hi && lane == 0) mbar_arrive(&acc_empty[half]);
                    // a pass is issued even when this set has no tokens in the item, so that every item consumes one buffer at least
                    for (int c0 = col_lo; c0 < col_hi || c0 == col_lo; c0 += 32) {
                        unsigned char *buf = my_buf + (pass_count & 1u) * kHcUpBufBytes, *nxt = my_buf + ((pass_count + 1) & 1u) * kHcUpBufBytes;
                        ++pass_count;
                        __syncwarp();  // every lane has finished reading the buffer that the next copies overwrite
                        if (c0 + 32 < col_hi) {
                            issue(it, c0 + 32, col_hi, nxt);
                        } else if (itn.bucket >= 0) {
                            issue(itn, col_lo, col_hi_of(itn), nxt);
                        } else {
                            cp_async_commit();
                        }
                        if (c0 >= col_hi) {  // nothing to finish: only the buffer rotation above
                            cp_async_wait<1>();
                            break;
                        }
                        float va[16], vb[16];
                        const uint32_t tcol = lane_addr + half * (uint32_t)kTile + (uint32_t)c0;
                        tc_ld16x2(tcol, tcol + 16u, va, vb);
                        if (c0 + 32 >= col_hi) {
                            tc_fence_before();
                            __syncwarp();
                            if (lane == 0) mbar_arrive(&acc_empty[half]);
                        }
                        cp_async_wait<1>();  // this pass's copies have landed (the next pass's may still be in flight)
                        __syncwarp();
                        const int live = col_hi - c0;
                        const TX *xs_ = reinterpret_cast<const TX *>(buf + s * seg) + jj;  // token tt: + tt * 32 elements
                        const float *ivs = reinterpret_cast<const float *>(buf + 128 * 32) + s;
                        // First every token's term of this lane's stream, in place of its accumulator (shared-memory reads and
                        // arithmetic only: a store to u in between would fence the next token's reads behind it, both being
                        // generic addresses).  Then the four streams of a column - lanes l, l ^ 1, l ^ 2, l ^ 3 - are added
                        // four tokens at a time by a reduce-scatter: three shuffles instead of the eight of four butterflies,
                        // and it leaves each of the four lanes with the sum of one token, which that lane stores.
#pragma unroll
                        for (int t = 0; t < 16; ++t) {
#pragma unroll
                            for (int hf = 0; hf < 2; ++hf) {
                                const int tt = t + 16 * hf;
                                const float z = hf ? vb[t] : va[t];
                                const float c = __fdividef(load_as_f32(xs_, tt * 32) * ivs[tt * 4] * nwp, 1.0f + exp2_fast(z * nz));
                                if (hf) vb[t] = c;
                                else va[t] = c;
                            }
                        }
                        const bool b0 = (lane & 1) != 0, b1 = (lane & 2) != 0;
                        const int mine = (b0 ? 2 : 0) + (b1 ? 1 : 0);  // which of a group's four tokens this lane ends up with
                        TX *up = static_cast<TX *>(hc.u) + (int64_t)(it.start + c0 + mine) * hc.d + j;
#pragma unroll
                        for (int i = 0; i < 8; ++i) {
                            const float ta = i < 4 ? va[4 * i] : vb[4 * i - 16], tb = i < 4 ? va[4 * i + 1] : vb[4 * i - 15];
                            const float tc = i < 4 ? va[4 * i + 2] : vb[4 * i - 14], td = i < 4 ? va[4 * i + 3] : vb[4 * i - 13];
                            // lanes with bit 0 clear keep tokens a, b and send c, d; the others the reverse
                            const float k0 = (b0 ? tc : ta) + __shfl_xor_sync(0xffffffffu, b0 ? ta : tc, 1);
                            const float k1 = (b0 ? td : tb) + __shfl_xor_sync(0xffffffffu, b0 ? tb : td, 1);
                            // lanes with bit 1 clear keep the first of the two and send the second; the others the reverse
                            const float sum = (b1 ? k1 : k0) + __shfl_xor_sync(0xffffffffu, b1 ? k0 : k1, 2);
                            if (4 * i + mine < live) store_from_f32(up, (int64_t)(4 * i) * hc.d, sum * 0.25f);
                        }
                    }
                }
                cp_async_wait<0>();
            };
            if (a.hc.f32) run(std::true_type{});
            else run(std::false_type{});
        }
    } else if (warp < kEpiWarps) {
        // ===================== epilogue =====================
        // 16 tokens at a time from tensor memory into registers, stored straight to global memory: for a fixed token a warp's rows are
        // contiguous bytes.  Tensor memory goes back to the MMA warp as soon as the item's last columns are in registers.  Where a token's
        // output row starts comes through the item ring; a line of the tile-blocked h follows from the token's position.  A pass runs as
        // straight code that the warp has to itself, at about eight cycles an instruction beside the producers: instructions count.
        uint32_t acc_count = 0;
        const int64_t I = a.N / 2;
        const uint32_t lane_addr = (uint32_t)(warp * 32) << 16;  // warp = the lane quadrant it may read
        for (int i = 0;; ++i) {
            const int ring = i % kItemRing;
            {
                const bool ok = mbar_wait(&item_full[ring], (uint32_t)(i / kItemRing) & 1u, abort_v, a.wait_limit_ns);
                if (!__all_sync(0xffffffffu, ok)) {
                    if (lane == 0) raise_abort(blockIdx.x + i * gridDim.x, 8);
                    break;
                }
            }
            const Item it = item_ring[ring];
            if (it.bucket < 0) break;
            const bool valid = it.bucket < a.E;
            const uint32_t half = acc_count & 1u, acc = lane_addr + half * (uint32_t)kTile;
            if (valid) {
                const uint32_t acc_phase = (acc_count >> 1) & 1u;
                ++acc_count;
                const bool ok = mbar_wait(&acc_full[half], acc_phase, abort_v, a.wait_limit_ns);
                if (!__all_sync(0xffffffffu, ok)) {
                    if (lane == 0) raise_abort(blockIdx.x + i * gridDim.x, 4);
                    break;
                }
                tc_fence_after();
            }
            // What undoes a row's power of two.  Slots with an id outside [0, E) have no products: their rows become NaN.
            auto back_of = [&](int p) { return valid ? unscale(scale_of(row_scale[ring][warp * 32 + p])) : qnan_f32(); };
            auto columns_read = [&](int c0) {  // the last columns are out: this warp's share of the accumulator is free
                if (valid && c0 + 16 >= it.cnt) {
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&acc_empty[half]);
                }
            };
            if constexpr (MODE == kTcSwiglu) {
                // Gate rows are the quadrant's lanes 0-15, the up rows of the same h columns its lanes 16-31.  Read in the form of sixteen
                // lanes by eight columns, both give a thread the same places: h columns r0 and r0 + 8 of tokens t and t + 1, and of
                // t + 8 and t + 9.  From the FP32 accumulators, rounded once (kernels/moe_grouped.hip:508-524).
                const int r0 = lane >> 2, t0 = (lane & 3) * 2;
                const float g0 = back_of(r0), g1 = back_of(r0 + 8), u0 = back_of(r0 + 16), u1 = back_of(r0 + 24);
                const bool h_as_f16 = a.out_f16 != 0, q4_order = a.out_f16 == 2 || a.out_f16 == 3, tiled_out = a.out_f16 >= 3;
                const int64_t j0 = (int64_t)it.rb * (kRows / 2) + warp * 16 + r0;  // h column; j0 + 8 is the other
                const bool ok0 = j0 < I, ok1 = j0 + 8 < I;
                const int pos = q4_order ? (((r0 & 3) << 1) | (r0 >> 2)) : r0;  // [0 4 1 5 2 6 3 7]
                // tile-blocked h: the token's line, its 16-byte chunks swizzled by the token; token t + 1 is the odd one of the pair
                const uint32_t in0 = (uint32_t)(t0 * 128 + (((2 * warp) ^ t0) << 4) + pos * 2), in1 = in0 ^ 16u;
                unsigned char *const out = static_cast<unsigned char *>(a.out) +
                                           (tiled_out ? ((int64_t)it.rb * a.L.S + it.start) * 128 : ((j0 & ~(int64_t)7) + pos) * 2);
                for (int c0 = 0; c0 < it.cnt; c0 += 16) {
                    float g[8] = {}, u[8] = {};
                    if (valid) tc_ld16lanes_x2(acc + (uint32_t)c0, acc + (16u << 16) + (uint32_t)c0, g, u);
                    columns_read(c0);
                    uint16_t h[8];
#pragma unroll
                    for (int t = 0; t < 8; ++t) {
                        const float gv = g[t] * ((t & 2) ? g1 : g0), uv = u[t] * ((t & 2) ? u1 : u0);
                        const uint16_t b = __bfloat16_as_ushort(__float2bfloat16_rn(silu_fast(gv) * uv));
                        h[t] = h_as_f16 ? __half_as_ushort(__float2half_rn(bf16_bits_to_f32(b))) : b;
                    }
                    const int live = it.cnt - c0 - t0;  // of this thread's tokens: 0, 1, 8, 9 from t0 on
                    auto put = [&](unsigned char *p, int t, int token, bool ok) { st_global_if(ok && token < live, p, h[t]); };
                    if (tiled_out) {
                        unsigned char *const p0 = out + (int64_t)c0 * 128 + in0, *const p1 = out + (int64_t)c0 * 128 + in1;
                        put(p0, 0, 0, ok0), put(p1, 2, 0, ok1), put(p1 + 128, 1, 1, ok0), put(p0 + 128, 3, 1, ok1);
                        put(p0 + 1024, 4, 8, ok0), put(p1 + 1024, 6, 8, ok1), put(p1 + 1152, 5, 9, ok0), put(p0 + 1152, 7, 9, ok1);
                    } else {
                        const uint2 a_b = *reinterpret_cast<const uint2 *>(&out_row[ring][c0 + t0]), c_d = *reinterpret_cast<const uint2 *>(&out_row[ring][c0 + t0 + 8]);
                        unsigned char *const pa = out + (uint64_t)a_b.x * 16, *const pb = out + (uint64_t)a_b.y * 16, *const pc = out + (uint64_t)c_d.x * 16,
                                             *const pd = out + (uint64_t)c_d.y * 16;
                        put(pa, 0, 0, ok0), put(pa + 16, 2, 0, ok1), put(pb, 1, 1, ok0), put(pb + 16, 3, 1, ok1);
                        put(pc, 4, 8, ok0), put(pc + 16, 6, 8, ok1), put(pd, 5, 9, ok0), put(pd + 16, 7, 9, ok1);
                    }
                }
            } else {
                // Lane = weight row; FP32 rows, or BF16 rows: the plain gather's y, or the per-slot dots as kernels/moe_grouped.hip:47-57 stores them.
                const float back = back_of(lane);
                const int64_t r = (int64_t)it.rb * kRows + warp * 32 + lane;
                const int rows_live = r < a.N ? it.cnt : 0;
                unsigned char *const out = static_cast<unsigned char *>(a.out) + r * (MODE == kTcPartial ? 4 : 2);
                for (int c0 = 0; c0 < it.cnt; c0 += 16) {
                    float v[16] = {};
                    if (valid) tc_ld16(acc + (uint32_t)c0, v);
                    columns_read(c0);
#pragma unroll
                    for (int t = 0; t < 16; ++t) v[t] *= back;
                    const int live = rows_live - c0;  // tokens of this pass; the columns past them are computed and dropped
#pragma unroll
                    for (int t = 0; t < 16; t += 4) {
                        const uint4 row = *reinterpret_cast<const uint4 *>(&out_row[ring][c0 + t]);
                        auto put = [&](uint32_t at, int k) {
                            unsigned char *const p = out + (uint64_t)at * 16;
                            if (MODE == kTcPartial) st_global_if(k < live, p, v[k]);
                            else st_global_if(k < live, p, __bfloat16_as_ushort(__float2bfloat16_rn(v[k])));
                        };
                        put(row.x, t), put(row.y, t + 1), put(row.z, t + 2), put(row.w, t + 3);
                    }
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&item_empty[ring]);
        }
    }

    // An aborting CTA must not return under copies it issued into its own shared memory (which may go to the next CTA):
    // the thread that ran the ring of weight codes waits, bounded, for the last fill of every slot; the activation copies
    // complete on barriers that also count thread arrivals, so their issuer lets a generous time pass instead.
    if (*abort_v) {
#pragma unroll 1
        for (int sl = 0; sl < kWSlots && issued > 0; ++sl) {
            if (issued <= (uint32_t)sl) continue;
            const uint32_t last = ((issued - 1 - (uint32_t)sl) / kWSlots) * kWSlots + (uint32_t)sl;
            if (blockIdx.x == 0 && (int)last == a.test_skip_slot) continue;  // the test hook's slot was never filled
            mbar_wait(&w_full[sl], (last / kWSlots) & 1u, nullptr, 1000000ull);
        }
        if (warp == kBCopyWarp)
            for (const unsigned long long t0 = global_ns(); global_ns() - t0 < 50000ull;) {}
    }
    tc_fence_before();
    __syncthreads();
    if (warp == kMmaWarp) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base_smem), "r"(kTmemCols) : "memory");
    }
}

}  // namespace

// Rows a tile of a dense projection has: 128 unless fewer fill the last wave of items better.  A step of 128 k takes about 450 + 3 n SM cycles for n
// rows with Q4 codes and 650 + 3 n with Q8.  Tiles of 128 -> as chosen, us: 300 x 2048 x 4096 Q8 + SwiGLU 26.2 -> 22.6 (80 rows), 200 x 2560 x 4096 Q4
// 20.5 -> 16.5 (64), 150 x 4096 x 4096 19.7 -> 17.9 (64), 777 x 4096 x 1024 Q8 18.5 -> 16.5 (96), 1001 x 8192 x 4096 Q4 53.4 -> 52.3 (112).
int dense_tile_rows(int64_t M, int64_t row_blocks, int64_t steps, int bits, int sms) {
    int best = kTile;
    double least = 0;
    for (int n = kTile; n >= 64; n -= 16) {
        const double items = (double)((M + n - 1) / n) * (double)row_blocks, cost = std::ceil(items / sms) * (steps * ((bits == 4 ? 450 : 650) + 3.0 * n) + 1000);
        if (least == 0 || cost < least) least = cost, best = n;
    }
    return best;
}

// One box of 128 codes x 128 rows (the SwiGLU form: of 64 rows of two matrices) fills a ring slot; 16-byte chunks swizzled in the mode of the box's row length so that the
// producers' 16-byte reads of consecutive rows hit every bank once.
template <int BITS, int MODE>
int launch_tiled_tc(const char *fn, TcArgs a, int64_t G, cudaStream_t st) {
    SXB_CHECK(a.x_kind == 3, fn, ": the tiled tcgen05 kernel takes tile-blocked activations only");
    a.dense_tile = kTile;
    if (a.dense_M > 0 && MODE != kTcHcUp)
        a.dense_tile = dense_tile_rows(a.dense_M, MODE == kTcSwiglu ? (a.N / 2 + kRows / 2 - 1) / (kRows / 2) : (a.N + kRows - 1) / kRows, a.K / kBK, BITS, sm_count());
    const uint64_t row_bytes = (uint64_t)(BITS == 4 ? a.K / 2 : a.K);
    CUtensorMap wmap;
    constexpr uint32_t box = kBK * BITS / 8;
    constexpr CUtensorMapSwizzle swizzle = BITS == 4 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B;
    const uint64_t rows = (uint64_t)(a.E * a.N), I = (uint64_t)a.N / 2;
    if (int rc = MODE == kTcSwiglu ? tensor_map_3d_bytes(fn, a.q, row_bytes, I, rows / I, row_bytes, I * row_bytes, box, (uint32_t)(kRows / 2), 2u, swizzle, &wmap)
                                   : tensor_map_2d(fn, a.q, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, row_bytes, rows, row_bytes, box, (uint32_t)kRows, swizzle, &wmap))
        return rc;
    auto go = [&](auto kern, auto shape, int64_t scale_bytes) -> int {
        using S = decltype(shape);
        SXB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, S::kMostDynamic), fn, ": reserving shared memory");
        kern<<<(unsigned)sm_count(), S::kThreads, (size_t)(S::kBufferBytes + scale_bytes), st>>>(a, wmap);
        return SXB_OK;
    };
    if constexpr (MODE != kTcHcUp) {
        // The scales of two items fit beside the rings up to 32 groups a row, of four up to 16.  The item warp reads them by eights, so rows of 6, 12, 20 or 28 groups, which
        // would fit too, are left to the producers' own loads, as longer rows and arrays that start elsewhere are.  With / without SS: see the head of this file.
        const int64_t groups = a.K / G;
        if (groups <= kScaleGroups && groups % 8 == 0 && ((reinterpret_cast<uintptr_t>(a.scale) | reinterpret_cast<uintptr_t>(a.minv)) & 15) == 0) {
            const int64_t bytes = ((int64_t)groups << scale_bufs_log((int)groups)) * kRows * 4;
            using S = Shape<BITS, false, true>;
            switch (G) {
                case 32: return go(tiled_tc_kernel<BITS, 32, MODE, true>, S{}, bytes);
                case 64: return go(tiled_tc_kernel<BITS, 64, MODE, true>, S{}, bytes);
                default: return go(tiled_tc_kernel<BITS, 128, MODE, true>, S{}, bytes);
            }
        }
    }
    using S = Shape<BITS, MODE == kTcHcUp, false>;
    switch (G) {
        case 32: return go(tiled_tc_kernel<BITS, 32, MODE, false>, S{}, 0);
        case 64: return go(tiled_tc_kernel<BITS, 64, MODE, false>, S{}, 0);
        default: return go(tiled_tc_kernel<BITS, 128, MODE, false>, S{}, 0);
    }
}

template int launch_tiled_tc<4, kTcGather>(const char *, TcArgs, int64_t, cudaStream_t);
template int launch_tiled_tc<4, kTcSwiglu>(const char *, TcArgs, int64_t, cudaStream_t);
template int launch_tiled_tc<4, kTcPartial>(const char *, TcArgs, int64_t, cudaStream_t);
template int launch_tiled_tc<4, kTcPartialBf16>(const char *, TcArgs, int64_t, cudaStream_t);
template int launch_tiled_tc<8, kTcGather>(const char *, TcArgs, int64_t, cudaStream_t);
template int launch_tiled_tc<8, kTcSwiglu>(const char *, TcArgs, int64_t, cudaStream_t);
template int launch_tiled_tc<8, kTcPartial>(const char *, TcArgs, int64_t, cudaStream_t);
template int launch_tiled_tc<8, kTcPartialBf16>(const char *, TcArgs, int64_t, cudaStream_t);
template int launch_tiled_tc<4, kTcHcUp>(const char *, TcArgs, int64_t, cudaStream_t);
template int launch_tiled_tc<8, kTcHcUp>(const char *, TcArgs, int64_t, cudaStream_t);

}  // namespace sxb
