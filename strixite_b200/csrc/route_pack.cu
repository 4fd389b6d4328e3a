// Pack: groups the S = M*A routed slots by expert (a counting sort) and cuts every expert's run of slots into the
// tiles the expert kernels iterate over.  C ABI twin of moe_group_routes / moe_route_workspace_bytes
// (kernels/moe_grouped.hpp:48-54; the reference's kernel is kernels/moe_grouped.hip:136-188, one 1024-thread block
// whose order inside a bucket is whatever its LDS atomics give).
//
// Here the sort is stable - inside a bucket, slots ascend - so the whole workspace is a pure function of ids and can
// be compared word for word with a CPU counting sort.  Ranks inside a bucket come from `match.any` warp votes, never
// from the arrival order of atomics.
//   S <= kSmallSlots: one CTA does everything, eight of its warps a run of slots each.
//   larger S: three launches - histograms of segments, a CTA each, one CTA that scans them into bucket offsets and per-segment
//   bases, and a scatter in which a CTA places its segment in order, a run of it a warp, and the CTAs share the tile lists.

#include "route_pack.cuh"

#include <algorithm>
#include "router_token.cuh"

namespace sxb {
namespace {

constexpr int kPackThreads = 1024;
constexpr int kSmallSlots = 2048;
constexpr int kSegWarps = 8, kSegRounds = kSegSlots / (32 * kSegWarps);  // of the CTA that takes a segment in the histogram / scatter launches

__device__ inline int bucket_of(int32_t id, int e_lo, int E_local) {
    const int b = id - e_lo;
    return (b < 0 || b >= E_local) ? E_local : b;
}

// Exclusive scan of v over the CTA's kPackThreads threads; *total = the sum.  buf: 33 words of shared memory.
__device__ inline uint64_t cta_exclusive_scan(uint64_t v, uint64_t *buf, uint64_t *total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint64_t incl = v;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const uint64_t t = __shfl_up_sync(0xffffffffu, incl, off);
        if (lane >= off) incl += t;
    }
    if (lane == 31) buf[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        const uint64_t w = buf[lane];
        uint64_t wi = w;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const uint64_t t = __shfl_up_sync(0xffffffffu, wi, off);
            if (lane >= off) wi += t;
        }
        buf[lane] = wi - w;
        if (lane == 31) buf[32] = wi;
    }
    __syncthreads();
    *total = buf[32];
    return incl - v + buf[warp];
}

// Where every bucket's slots and tiles begin.  first[i]: the bucket's first tile in list i; entry E + 1 = the total.
constexpr int kTileLists = 2;
__device__ constexpr int kTileRows[kTileLists] = {8, 128};
struct Layout {
    int start[kMoeMaxExperts + 1];
    int first[kTileLists][kMoeMaxExperts + 2];
    uint64_t scan[33];
};

// Per-bucket counts (thread b owns bucket b) -> sm, and offsets and header of the workspace.  Ends with a barrier.
// One scan for the three sums, each in 21 bits (at most 2^20 slots): slots, 8-slot and 128-slot tiles.
__device__ void scan_layout(int count, const RouteWords &L, int32_t *ws, Layout &sm, bool ep) {
    const int b = threadIdx.x, E = (int)L.E;
    // Tiles are cut for buckets 0..E-1, and for the overflow bucket E only outside expert-parallel mode (there its
    // slots are invalid ids whose outputs must become NaN; in EP mode they belong to other ranks and are skipped).
    const bool tiled = b < E || (b == E && !ep);
    if (b > E) count = 0;
    auto tiles = [&](int rows) { return (uint64_t)(tiled ? (count + rows - 1) / rows : 0); };
    uint64_t total;
    const uint64_t sum = cta_exclusive_scan((uint64_t)count | (tiles(8) << 21) | (tiles(128) << 42), sm.scan, &total);
    const int mask = (1 << 21) - 1;
    auto store = [&](int at, uint64_t s) { sm.first[0][at] = (int)(s >> 21) & mask, sm.first[1][at] = (int)(s >> 42); };
    if (b <= E) {
        sm.start[b] = (int)sum & mask;
        ws[L.offsets + b] = (int)sum & mask;
        store(b, sum);
    }
    if (b == 0) {
        store(E + 1, total);
        ws[L.offsets + E + 1] = (int)total & mask;
        ws[0] = (int)(total >> 21) & mask, ws[1] = (int32_t)L.S, ws[2] = E, ws[3] = (int)(total >> 42), ws[4] = ep ? 1 : 0;
        ws[5] = 0, ws[6] = 0, ws[7] = 0;
    }
    __syncthreads();
}

// Tiles t0, t0 + stride, ... of every list: a tile belongs to the last bucket whose first tile is not past it (empty buckets
// never win).
__device__ void emit_tiles(const RouteWords &L, int32_t *ws, const Layout &sm, int t0, int stride) {
    const int E = (int)L.E;
    const int64_t bucket_at[kTileLists] = {L.t8_bucket, L.t128_bucket};
    const int64_t start_at[kTileLists] = {L.t8_start, L.t128_start};
#pragma unroll
    for (int list = 0; list < kTileLists; ++list) {
        const int *first = sm.first[list];
        for (int t = t0; t < first[E + 1]; t += stride) {
            int lo = 0, hi = E + 1;  // invariant: first[lo] <= t < first[hi]
            while (hi - lo > 1) {
                const int mid = (lo + hi) >> 1;
                if (first[mid] <= t) lo = mid;
                else hi = mid;
            }
            ws[bucket_at[list] + t] = lo;
            ws[start_at[list] + t] = sm.start[lo] + (t - first[lo]) * kTileRows[list];
        }
    }
}

// Ranks of a warp's slots s0 + 32 r + lane (ids id[r], below S) among its slots of the same bucket: match.any in a round, the warp's own
// counts (zero at first) across rounds.  bucket < 0: past the end.
template <int ROUNDS>
__device__ inline void rank_slots(const int32_t (&id)[ROUNDS], int s0, int S, int e_lo, int E, uint16_t *counts, int (&bucket)[ROUNDS], int (&rank)[ROUNDS]) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int r = 0; r < ROUNDS; ++r) {
        const bool live = s0 + r * 32 + lane < S;
        bucket[r] = live ? bucket_of(id[r], e_lo, E) : -1 - lane;  // dead lanes match nobody
        if (s0 + r * 32 >= S) continue;
        const unsigned peers = __match_any_sync(0xffffffffu, bucket[r]);
        const int before = live ? counts[bucket[r]] : 0, mine = __popc(peers & ((1u << lane) - 1u));
        rank[r] = before + mine;
        __syncwarp();  // of the whole warp: one per group of peers ran them one after another
        if (live && mine == 0) counts[bucket[r]] = (uint16_t)(before + __popc(peers));
        __syncwarp();
    }
}

// The whole pack of a small batch by one CTA of kPackThreads threads.  Eight warps take a run of slots each, in slot order; a
// slot's rank among its warp's slots of the same bucket comes from match.any and the warp's own counts, and a bucket's base for
// each warp from a prefix over the warps' counts: no warp waits for another (one warp placing 1500 slots, 32 a round, was most
// of an 87 us launch).
constexpr int kPlaceWarps = 8, kPlaceRounds = kSmallSlots / (32 * kPlaceWarps);
__device__ void pack_small_body(const int32_t *__restrict__ ids, const RouteWords &L, int E_total, int e_lo, bool ep, int32_t *ws,
                                uint32_t *err) {
    __shared__ Layout sm;
    __shared__ uint16_t counts[kPlaceWarps][kPackThreads];
    __shared__ int first_bad;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5, S = (int)L.S, E = (int)L.E;
    for (int i = t; i < kPlaceWarps * kPackThreads / 2; i += kPackThreads) reinterpret_cast<uint32_t *>(counts)[i] = 0u;
    if (t == 0) first_bad = 0x7fffffff;
    __syncthreads();
    const int rounds = (S + 32 * kPlaceWarps - 1) / (32 * kPlaceWarps);  // of each warp: 1 .. kPlaceRounds
    int bucket[kPlaceRounds], rank[kPlaceRounds];
    if (warp < kPlaceWarps) {
        int32_t id[kPlaceRounds];
#pragma unroll
        for (int r = 0; r < kPlaceRounds; ++r) {
            const int s = (warp * rounds + r) * 32 + lane;
            id[r] = r < rounds && s < S ? ids[s] : 0;
        }
#pragma unroll
        for (int r = 0; r < kPlaceRounds; ++r) {
            const int s = (warp * rounds + r) * 32 + lane;
            if (r < rounds && s < S && (id[r] < 0 || id[r] >= E_total)) atomicMin(&first_bad, s);
        }
        rank_slots<kPlaceRounds>(id, warp * rounds * 32, min(S, (warp + 1) * rounds * 32), e_lo, E, counts[warp], bucket, rank);
    }
    __syncthreads();
    if (t == 0 && first_bad != 0x7fffffff) raise_error(err, (uint32_t)ids[first_bad], (uint32_t)first_bad);
    int count = 0;
    if (t <= E) {
#pragma unroll
        for (int w = 0; w < kPlaceWarps; ++w) {
            const int c = counts[w][t];
            counts[w][t] = (uint16_t)count;  // the warp's base inside the bucket
            count += c;
        }
    }
    scan_layout(count, L, ws, sm, ep);
    if (warp < kPlaceWarps) {
#pragma unroll
        for (int r = 0; r < kPlaceRounds; ++r)
            if (bucket[r] >= 0) ws[L.slots + sm.start[bucket[r]] + counts[warp][bucket[r]] + rank[r]] = (warp * rounds + r) * 32 + lane;
    }
    emit_tiles(L, ws, sm, t, kPackThreads);
}

__global__ void __launch_bounds__(kPackThreads)
    pack_small_kernel(const int32_t *__restrict__ ids, RouteWords L, int E_total, int e_lo, bool ep, int32_t *ws,
                      uint32_t *err, bool let_in) {
    behind_grid(let_in);
    pack_small_body(ids, L, E_total, e_lo, ep, ws, err);
}

// Router and pack of a small batch (decode: a few dozen tokens) as ONE launch of one CTA: every warp routes tokens
// (route_token), the CTA then packs the slots it has just written.  Same words out as moe_router + moe_group_routes.
template <int NV>
__global__ void __launch_bounds__(kPackThreads)
    route_small_kernel(const float *__restrict__ logits, int64_t ld, int M, int E_total, int k, int32_t *__restrict__ ids,
                       float *__restrict__ coef, RouteWords L, int e_lo, bool ep, int32_t *ws, uint32_t *router_err,
                       uint32_t *expert_err, bool let_in) {
    behind_grid(let_in);
    __shared__ unsigned long long cand[kPackThreads / 32][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int m = warp; m < M; m += kPackThreads / 32)
        route_token<float, NV>(logits + (int64_t)m * ld, lane, m, E_total, k, nullptr, 1, 0, ids + (int64_t)m * k,
                               coef + (int64_t)m * k, k, router_err, cand[warp]);
    __threadfence_block();
    __syncthreads();  // the ids written above are read by other threads of this CTA below
    pack_small_body(ids, L, E_total, e_lo, ep, ws, expert_err);
}

// Large S, launch 1: histogram of every 1024-slot segment (one CTA each) into scratch [nseg][E + 1], and the
// segment's first invalid slot into segbad [nseg].
__global__ void __launch_bounds__(32 * kSegWarps)
    pack_hist_kernel(const int32_t *__restrict__ ids, RouteWords L, int E_total, int e_lo, int32_t *ws) {
    behind_grid();
    __shared__ int hist[kMoeMaxExperts + 1], first_bad;
    const int t = threadIdx.x, E = (int)L.E, S = (int)L.S, s0 = (int)blockIdx.x * kSegSlots;
    int32_t id[kSegRounds];
#pragma unroll
    for (int r = 0; r < kSegRounds; ++r) id[r] = s0 + r * 32 * kSegWarps + t < S ? ids[s0 + r * 32 * kSegWarps + t] : 0;
    for (int b = t; b <= E; b += 32 * kSegWarps) hist[b] = 0;
    if (t == 0) first_bad = 0x7fffffff;
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kSegRounds; ++r) {
        const int s = s0 + r * 32 * kSegWarps + t;
        if (s >= S) break;
        atomicAdd(&hist[bucket_of(id[r], e_lo, E)], 1);
        if (id[r] < 0 || id[r] >= E_total) atomicMin(&first_bad, s);
    }
    __syncthreads();
    int32_t *out = ws + L.scratch + (int64_t)blockIdx.x * (E + 1);
    for (int b = t; b <= E; b += 32 * kSegWarps) out[b] = hist[b];
    if (t == 0) ws[L.segbad + blockIdx.x] = first_bad;
}

// Launch 2 (one CTA): per bucket, turn the segments' counts into their exclusive prefix (the segment's base inside
// the bucket); totals -> offsets, header, tile lists; the first invalid slot -> err.
__global__ void __launch_bounds__(kPackThreads)
    pack_scan_kernel(const int32_t *__restrict__ ids, RouteWords L, bool ep, int32_t *ws, uint32_t *err) {
    behind_grid();
    __shared__ Layout sm;
    const int b = threadIdx.x, E = (int)L.E;
    int total = 0;
    if (b <= E) {
        // sixteen segments at a time: the loads of a chunk are independent of one another (a chain of dependent
        // read-modify-writes over 160 segments was most of this launch)
        int32_t *col = ws + L.scratch + b;
        const int64_t stride = E + 1;
        int c[16], nxt[16];
        auto fetch = [&](int seg0) {
#pragma unroll
            for (int i = 0; i < 16; ++i) nxt[i] = seg0 + i < L.nseg ? col[(int64_t)(seg0 + i) * stride] : 0;
        };
        fetch(0);
        for (int seg0 = 0; seg0 < L.nseg; seg0 += 16) {
#pragma unroll
            for (int i = 0; i < 16; ++i) c[i] = nxt[i];
            fetch(seg0 + 16);  // the next chunk's loads before this chunk's stores, which they do not depend on
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                if (seg0 + i < L.nseg) col[(int64_t)(seg0 + i) * stride] = total;
                total += c[i];
            }
        }
    }
    int bad = 0x7fffffff;
    for (int seg = b; seg < L.nseg; seg += kPackThreads) bad = min(bad, ws[L.segbad + seg]);
    bad = __reduce_min_sync(0xffffffffu, bad);
    __shared__ int bad_w[32];
    if ((b & 31) == 0) bad_w[b >> 5] = bad;
    __syncthreads();
    if (b == 0) {
        for (int w = 1; w < 32; ++w) bad = min(bad, bad_w[w]);
        if (bad != 0x7fffffff) raise_error(err, (uint32_t)ids[bad], (uint32_t)bad);
    }
    scan_layout(total, L, ws, sm, ep);
    // the tile lists are the last launch's work, whose CTAs share it
    for (int i = b; i < kTileLists * (E + 2); i += kPackThreads) ws[L.first + i] = sm.first[i / (E + 2)][i % (E + 2)];
}

// Launch 3: a CTA places its segment, each bucket from offsets[b] + the segment's base on; the CTAs then share the tile lists, whose
// length grows with the slots (written by the one CTA of launch 2 they were most of its 39 us at 16384 tokens).  The segment's warps
// take 128 slots each, as in the small pack: no warp waits for another (a warp a segment, 32 rounds one after another, was most of the
// launch: 15.5 us at 777 to 16384 tokens x 10 slots).
__global__ void __launch_bounds__(32 * kSegWarps)
    pack_scatter_kernel(const int32_t *__restrict__ ids, RouteWords L, int e_lo, int32_t *ws, bool let_in) {
    behind_grid(let_in);
    __shared__ __align__(4) uint16_t counts[kSegWarps][kMoeMaxExperts + 1];
    __shared__ Layout sm;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5, E = (int)L.E, S = (int)L.S, s0 = (int)blockIdx.x * kSegSlots + warp * kSegRounds * 32;
    int32_t id[kSegRounds];
#pragma unroll
    for (int r = 0; r < kSegRounds; ++r) id[r] = s0 + r * 32 + lane < S ? ids[s0 + r * 32 + lane] : 0;
    const int32_t *base = ws + L.scratch + (int64_t)blockIdx.x * (E + 1);
    for (int i = t; i < kSegWarps * (kMoeMaxExperts + 1) / 2; i += 32 * kSegWarps) reinterpret_cast<uint32_t *>(counts)[i] = 0u;
    for (int i = t; i < kTileLists * (E + 2); i += 32 * kSegWarps) sm.first[i / (E + 2)][i % (E + 2)] = ws[L.first + i];
    for (int b = t; b <= E; b += 32 * kSegWarps) sm.start[b] = ws[L.offsets + b];
    __syncthreads();
    int bucket[kSegRounds], rank[kSegRounds];
    rank_slots<kSegRounds>(id, s0, S, e_lo, E, counts[warp], bucket, rank);
    __syncthreads();
    for (int b = t; b <= E; b += 32 * kSegWarps) {
        int at = 0;
#pragma unroll
        for (int w = 0; w < kSegWarps; ++w) {
            const int c = counts[w][b];
            counts[w][b] = (uint16_t)at;  // the warp's base inside the segment's run of the bucket
            at += c;
        }
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kSegRounds; ++r)
        if (bucket[r] >= 0) ws[L.slots + sm.start[bucket[r]] + base[bucket[r]] + counts[warp][bucket[r]] + rank[r]] = s0 + r * 32 + lane;
    emit_tiles(L, ws, sm, blockIdx.x * 32 * kSegWarps + t, gridDim.x * 32 * kSegWarps);
}

}  // namespace

RouteWords route_words(int64_t M, int64_t A, int64_t E) {
    RouteWords L;
    L.S = M * A, L.E = E;
    L.T8max = L.S / 8 + E + 2, L.T128max = L.S / 128 + E + 2;
    L.nseg = L.S <= kSmallSlots ? 0 : (L.S + kSegSlots - 1) / kSegSlots;
    L.offsets = 8;
    L.slots = L.offsets + E + 2;
    L.t8_bucket = L.slots + L.S;
    L.t8_start = L.t8_bucket + L.T8max;
    L.t128_bucket = L.t8_start + L.T8max;
    L.t128_start = L.t128_bucket + L.T128max;
    L.segbad = L.t128_start + L.T128max;
    L.scratch = L.segbad + L.nseg;
    L.first = L.scratch + L.nseg * (E + 1);
    L.total = L.first + (L.nseg ? kTileLists * (E + 2) : 0);
    return L;
}

int group_routes(const char *fn, const int32_t *ids, int64_t M, int64_t A, int64_t E_total, int64_t e_lo,
                 int64_t E_local, bool ep, void *ws, size_t ws_bytes, uint32_t *err, bool let_in, sxb_stream_t stream) {
    SXB_CHECK(ids != nullptr && ws != nullptr && err != nullptr, fn, ": null pointer (ids=", (const void *)ids, ", ws=", ws,
              ", err=", (const void *)err, ")");
    SXB_CHECK(M >= 1 && A >= 1 && A <= 64 && E_local >= 1 && E_local <= kMoeMaxExperts && M * A <= kMoeMaxSlots, fn,
              ": M = ", M, ", A = ", A, ", E = ", E_local, " (A 1..64, E 1..", kMoeMaxExperts, ", M*A <= ", kMoeMaxSlots, ")");
    SXB_CHECK(e_lo >= 0 && e_lo + E_local <= E_total, fn, ": experts [", e_lo, ", ", e_lo + E_local, ") outside [0, ",
              E_total, ")");
    const RouteWords L = route_words(M, A, E_local);
    SXB_CHECK(ws_bytes >= (size_t)L.total * 4, fn, ": workspace of ", ws_bytes, " bytes, needs ", L.total * 4);
    SXB_CHECK(reinterpret_cast<uintptr_t>(ws) % 4 == 0, fn, ": workspace ", ws, " must be 4-byte aligned");
    auto st = static_cast<cudaStream_t>(stream);
    auto *w = static_cast<int32_t *>(ws);
    if (L.S <= kSmallSlots) {
        launch_behind(pack_small_kernel, 1, kPackThreads, 0, st, 1, ids, L, (int)E_total, (int)e_lo, ep, w, err, let_in);
    } else {
        const unsigned ctas = (unsigned)L.nseg;
        launch_behind(pack_hist_kernel, ctas, 32 * kSegWarps, 0, st, 1, ids, L, (int)E_total, (int)e_lo, w);
        launch_behind(pack_scan_kernel, 1, kPackThreads, 0, st, 1, ids, L, ep, w, err);
        launch_behind(pack_scatter_kernel, ctas, 32 * kSegWarps, 0, st, 1, ids, L, (int)e_lo, w, let_in);
    }
    SXB_CHECK_LAUNCH(fn, " M=", M, " A=", A, " E=", E_local);
    return SXB_OK;
}

int route_small(const char *fn, const float *logits, int64_t ld, int64_t M, int64_t E_total, int64_t k, int64_t e_lo, int64_t E_local, int32_t *ids, float *coef,
                void *ws, size_t ws_bytes, uint32_t *router_err, uint32_t *expert_err, bool let_in, sxb_stream_t stream) {
    SXB_CHECK(logits != nullptr && ids != nullptr && coef != nullptr && ws != nullptr && router_err != nullptr && expert_err != nullptr,
              fn, ": null pointer");
    SXB_CHECK(E_total >= 1 && E_total <= 1024 && k >= 1 && k <= E_total && k <= 32 && ld >= E_total, fn, ": E = ", E_total, ", k = ", k,
              ", ld = ", ld, " (E 1..1024, k 1..min(E, 32), ld >= E)");
    SXB_CHECK(M >= 1 && M * k <= kSmallSlots, fn, ": M * k = ", M * k, " slots, this one-CTA form takes at most ", kSmallSlots,
              " (use moe_router + moe_group_routes)");
    SXB_CHECK(E_local >= 1 && E_local <= kMoeMaxExperts && e_lo >= 0 && e_lo + E_local <= E_total, fn, ": experts [", e_lo, ", ",
              e_lo + E_local, ") outside [0, ", E_total, ")");
    const bool ep = E_local != E_total;
    const RouteWords L = route_words(M, k, E_local);
    SXB_CHECK(ws_bytes >= (size_t)L.total * 4, fn, ": workspace of ", ws_bytes, " bytes, needs ", L.total * 4);
    auto st = static_cast<cudaStream_t>(stream);
    auto *w = static_cast<int32_t *>(ws);
    // One CTA routes 32 tokens at a time, so from there on the router has a launch of its own, with a warp a token over the
    // machine (150 tokens x 512 experts, top-10: 87 us as one launch).
    if (M > kPackThreads / 32) {
        if (int rc = sxb_moe_router(logits, ld, M, E_total, k, nullptr, 1, 0, ids, coef, SXB_ACT_F32, router_err, stream)) return rc;
        launch_behind(pack_small_kernel, 1, kPackThreads, 0, st, 1, ids, L, (int)E_total, (int)e_lo, ep, w, expert_err, let_in);
        SXB_CHECK_LAUNCH(fn, " M=", M, " E=", E_total, " k=", k);
        return SXB_OK;
    }
#define SXB_ROUTE_SMALL(NV) \
    launch_behind(route_small_kernel<NV>, 1, kPackThreads, 0, st, 1, logits, ld, (int)M, (int)E_total, (int)k, ids, coef, L, (int)e_lo, ep, w, router_err, expert_err, let_in)
    if (E_total <= 128) SXB_ROUTE_SMALL(4);
    else if (E_total <= 256) SXB_ROUTE_SMALL(8);
    else if (E_total <= 512) SXB_ROUTE_SMALL(16);
    else SXB_ROUTE_SMALL(32);
#undef SXB_ROUTE_SMALL
    SXB_CHECK_LAUNCH(fn, " M=", M, " E=", E_total, " k=", k);
    return SXB_OK;
}

}  // namespace sxb

using namespace sxb;

namespace sxb {
// {2, work item, role}: the record of a device-side wait that ran out, of the tcgen05 kernels (grouped_tc.cu) or of the exact grouped forms
// (kRoleStaged and kRoleLeft, the item being a tile of eight tokens).
int tc_status_error(const char *what, const uint32_t e[3]) {
    static const char *roles[] = {"an unknown role",
                                  "a weight producer waiting for a free operand stage",
                                  "an MMA warp waiting for free accumulators",
                                  "an MMA warp waiting for a filled operand stage",
                                  "the epilogue waiting for the accumulators",
                                  "the activation copy thread waiting for a free operand stage",
                                  "the weight-code copy thread waiting for a free ring slot",
                                  "a weight producer waiting for its packed codes",
                                  "a warp waiting for the description of its next work item",
                                  "the work-item thread waiting for room in its ring",
                                  "a warp waiting for the tile's staged activations",
                                  "a staging warp waiting for the last warp to leave its buffer"};
    static_assert(sizeof(roles) / sizeof(roles[0]) == kRoleLeft + 1, "a text for each role");
    const bool streaming = e[2] == kRoleStaged || e[2] == kRoleLeft;
    last_error() = cat(what ? what : "", streaming ? ": the streaming expert kernel gave up a wait at tile " : ": a tcgen05 kernel gave up a wait at work item ",
                       e[1], " (", roles[e[2] >= 1 && e[2] <= kRoleLeft ? e[2] : 0], "); its outputs are incomplete");
    return SXB_ERR_DATA;
}
}  // namespace sxb

extern "C" {

size_t sxb_moe_route_workspace_bytes(int64_t M, int64_t A, int64_t E) {
    if (!(M >= 1 && A >= 1 && E >= 1 && E <= kMoeMaxExperts && M * A <= kMoeMaxSlots)) {
        fail_check(SXB_FILE_, __LINE__, __func__, "M >= 1 && A >= 1 && 1 <= E <= 1023 && M * A <= 2^20",
                   cat("moe_route_workspace_bytes: M = ", M, ", A = ", A, ", E = ", E));
        return 0;
    }
    return (size_t)route_words(M, A, E).total * 4;
}

int sxb_route_layout(int64_t M, int64_t A, int64_t E, int64_t out[8]) {
    SXB_CHECK(out != nullptr && M >= 1 && A >= 1 && E >= 1 && E <= kMoeMaxExperts && M * A <= kMoeMaxSlots,
              "route_layout: M = ", M, ", A = ", A, ", E = ", E);
    const RouteWords L = route_words(M, A, E);
    out[0] = 0, out[1] = L.offsets, out[2] = L.slots, out[3] = L.t8_bucket, out[4] = L.t8_start, out[5] = L.t128_bucket,
    out[6] = L.t128_start, out[7] = L.total;
    return SXB_OK;
}

int sxb_check_grouped_status(const void *ws, const char *what) {
    SXB_CHECK(ws != nullptr, "check_grouped_status(", what, "): null workspace");
    int32_t head[8];
    SXB_CUDA(cudaMemcpy(head, ws, sizeof(head), cudaMemcpyDeviceToHost), "reading the workspace header for ", what);
    if (head[5] == 0) return SXB_OK;
    const uint32_t e[3] = {(uint32_t)head[5], (uint32_t)head[6], (uint32_t)head[7]};
    return tc_status_error(what, e);
}

int sxb_moe_group_routes(const int32_t *ids, int64_t M, int64_t A, int64_t E, void *ws, size_t ws_bytes, uint32_t *err,
                         sxb_stream_t stream) {
    return group_routes("moe_group_routes", ids, M, A, E, 0, E, false, ws, ws_bytes, err, true, stream);
}

int sxb_moe_group_routes_ep(const int32_t *ids, int64_t M, int64_t A, int64_t E_total, int64_t e_lo, int64_t E_local,
                            void *ws, size_t ws_bytes, uint32_t *err, sxb_stream_t stream) {
    return group_routes("moe_group_routes_ep", ids, M, A, E_total, e_lo, E_local, true, ws, ws_bytes, err, true, stream);
}

int sxb_moe_route_small(const float *logits, int64_t ld, int64_t M, int64_t E_total, int64_t k, int64_t e_lo, int64_t E_local,
                        int32_t *ids, float *coef, void *ws, size_t ws_bytes, uint32_t *router_err, uint32_t *expert_err,
                        sxb_stream_t stream) {
    return route_small("moe_route_small", logits, ld, M, E_total, k, e_lo, E_local, ids, coef, ws, ws_bytes, router_err, expert_err, true, stream);
}

}  // extern "C"
