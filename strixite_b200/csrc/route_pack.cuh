// Layout of the grouping workspace shared by the pack (route_pack.cu) and the expert kernels that walk it.
#pragma once

#include "common.cuh"

namespace sxb {

constexpr int64_t kMoeMaxExperts = 1023;   // E + 1 buckets fit one 1024-thread CTA (kernels/moe_grouped.hpp:43)
constexpr int64_t kMoeMaxSlots = 1 << 20;  // kernels/moe_grouped.hpp:44
constexpr int kSegSlots = 1024;            // slots one CTA places in the multi-CTA pack

// Word (int32) offsets into the workspace.
//   header [8]: n_tiles8, S, E, n_tiles128, ep_mode, 0, 0, 0
//   offsets [E + 2]: bucket b's slots are slots[offsets[b] .. offsets[b + 1]); bucket E = invalid ids (or, in
//                    expert-parallel mode, every slot that is not this rank's); offsets[E + 1] = S
//   slots [S]: slot index s = m * A + a, ascending inside a bucket
//   t8_bucket / t8_start [T8max]: tiles of up to 8 slots (the streaming kernels); t128_*: up to 128 (tcgen05)
//   segbad [nseg], scratch [nseg][E + 1]: the multi-CTA pack's per-segment first invalid slot and histograms
//   first [2][E + 2], multi-CTA pack only: every bucket's first tile in the two lists, then the list's length
struct RouteWords {
    int64_t S, E, T8max, T128max, nseg;
    int64_t offsets, slots, t8_bucket, t8_start, t128_bucket, t128_start, segbad, scratch, first, total;
};
RouteWords route_words(int64_t M, int64_t A, int64_t E);

// sxb_moe_route_small and sxb_moe_group_routes[_ep] (route_pack.cu).  let_in: whether the next launch of the stream may take its places while these few CTAs run.  In
// front of the streaming expert kernel, which takes all registers of an SM and waits there, not where a second stream has work for the SMs:
// one-token layer with the shared expert beside it, issued call by call, 64.8 us let in at once and 55.1 at the end; without a second
// stream a layer of 512 x 128, one token, 18.8 and 19.9.
int route_small(const char *fn, const float *logits, int64_t ld, int64_t M, int64_t E_total, int64_t k, int64_t e_lo, int64_t E_local, int32_t *ids, float *coef,
                void *ws, size_t ws_bytes, uint32_t *router_err, uint32_t *expert_err, bool let_in, sxb_stream_t stream);
int group_routes(const char *fn, const int32_t *ids, int64_t M, int64_t A, int64_t E_total, int64_t e_lo, int64_t E_local, bool ep, void *ws, size_t ws_bytes,
                 uint32_t *err, bool let_in, sxb_stream_t stream);

// Roles of the exact grouped forms in the status words (header words 5 .. 7), behind those of the tcgen05 kernels: a warp that waits for a tile's
// staged activations, a staging warp that waits for the last warp to leave the buffer.
constexpr int kRoleStaged = 10, kRoleLeft = 11;

// The workspace of the grouping in which slot m * E + b belongs to bucket b, for all m < per_bucket: what sxb_moe_group_routes writes for
// ids[m * E + b] = b, without the ids or the sort.  L = route_words(per_bucket * E, 1, E); by threads first, first + stride, ...
__device__ inline void write_regular_routes(const RouteWords &L, int64_t per_bucket, int32_t *ws, int64_t first, int64_t stride) {
    const int64_t E = L.E, n8 = (per_bucket + 7) / 8, n128 = (per_bucket + 127) / 128;
    for (int64_t i = first; i < L.S; i += stride) ws[L.slots + i] = (int32_t)((i % per_bucket) * E + i / per_bucket);
    for (int64_t i = first; i < E * n8; i += stride) ws[L.t8_bucket + i] = (int32_t)(i / n8), ws[L.t8_start + i] = (int32_t)(i / n8 * per_bucket + i % n8 * 8);
    for (int64_t i = first; i < E * n128; i += stride) ws[L.t128_bucket + i] = (int32_t)(i / n128), ws[L.t128_start + i] = (int32_t)(i / n128 * per_bucket + i % n128 * 128);
    for (int64_t i = first; i < E + 2; i += stride) ws[L.offsets + i] = (int32_t)(min(i, E) * per_bucket);
    for (int64_t i = first; i < 8; i += stride) ws[i] = i == 0 ? (int32_t)(E * n8) : i == 1 ? (int32_t)L.S : i == 2 ? (int32_t)E : i == 3 ? (int32_t)(E * n128) : 0;
}

}  // namespace sxb
