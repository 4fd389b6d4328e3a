// One token of the MoE router, by one warp: top-k of the token's E logits (larger first, a tie to the lower index), the
// softmax over the picks, the optional shared slot.  Shared by the router kernel (router.cu) and the one-CTA
// router + pack kernel of small batches (route_pack.cu).  Arithmetic: kernels/moe_router.hip:82-111.
#pragma once

#include "common.cuh"

#include <climits>

namespace sxb {

constexpr int kRouterLanes = 32;

// Order-preserving map float -> uint32 (finite values and infinities): a < b  <=>  key(a) < key(b).
// -0 is folded onto +0 first, so the two compare equal as they do as floats.  key_value: the way back.
__device__ inline uint32_t order_key(float v) {
    const uint32_t u = __float_as_uint(v + 0.0f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

__device__ inline float key_value(uint32_t key) { return __uint_as_float((key & 0x80000000u) ? key ^ 0x80000000u : ~key); }

// Sorts the lanes' values, largest in lane 0: a bitonic network over shuffles, fifteen steps.
template <typename V>
__device__ inline V sorted_down(V v, int lane) {
#pragma unroll
    for (int run = 2; run <= 32; run <<= 1)
#pragma unroll
        for (int j = run >> 1; j > 0; j >>= 1) {
            const V other = __shfl_xor_sync(0xffffffffu, v, j);
            const bool keep_larger = ((lane & run) == 0) == ((lane & j) == 0);
            v = (other > v) == keep_larger ? other : v;
        }
    return v;
}

// The k of the picks by sort (picked_by_sort).  Above 16 the candidates are too many to be sorted; below the other line a few rounds cost less than the
// two sorts: us of rounds and of the sort, 16384 tokens, E = 128 k = 4 8.7 and 9.2, k = 6 11.0 and 9.2; E = 256 k = 3 9.9 and 11.5, k = 4 13.1 and 11.6;
// E = 512 k = 1 15.7 and 18.0, k = 3 21.3 and 18.0; E = 1000 k = 1 37 and 40, k = 3 46 and 40.
constexpr int kPickSort = 16;
template <int NV> constexpr int kPickSortMin = NV <= 4 ? 6 : NV <= 8 ? 4 : 3;

// The top k of the warp's keys (0 = no key), pick r in lane r as {key, ~index}, k <= kPickSort.  The k-th largest of the lanes' own largest keys
// bounds the k-th pick from below: k different keys reach it.  What reaches it - a dozen of 512 for a top-10 - is gathered in shared memory (cand,
// the warp's 32 words) and sorted, a tie to the lower index.  False, with nothing picked, where that is more than 32 keys (ties).
// Against a round of two reductions and a scan of the owner's sixteen keys for each pick: a third of the chain and half the instructions.
template <int NV>
__device__ inline bool picked_by_sort(const uint32_t (&key)[NV], int lane, int k, unsigned long long *cand, unsigned long long &mine) {
    uint32_t most = 0u;
#pragma unroll
    for (int j = 0; j < NV; ++j) most = max(most, key[j]);
    const uint32_t bound = max(1u, __shfl_sync(0xffffffffu, sorted_down(most, lane), k - 1));
    int n = 0;
#pragma unroll
    for (int j = 0; j < NV; ++j) {
        const uint32_t who = __ballot_sync(0xffffffffu, key[j] >= bound);
        const int at = n + __popc(who & ((1u << lane) - 1u));
        if (key[j] >= bound && at < 32) cand[at] = (unsigned long long)key[j] << 32 | ~(uint32_t)(lane + j * kRouterLanes);
        n += __popc(who);
    }
    if (n > 32) return false;
    __syncwarp();
    mine = sorted_down(lane < n ? cand[lane] : 0ull, lane);
    __syncwarp();  // the words may be written again
    return true;
}

// row: the token's logits; cand: 32 words of shared memory of the warp's own; id_row / coef_row: its A output slots.  The whole warp calls this (lane = its lane).
template <typename T, int NV>
__device__ inline void route_token(const T *__restrict__ row, int lane, int64_t m, int E, int k, const T *__restrict__ shared,
                                   int64_t shared_ld, int32_t shared_id, int32_t *__restrict__ id_row,
                                   float *__restrict__ coef_row, int A, uint32_t *err, unsigned long long *cand) {
    constexpr int kLanes = kRouterLanes;
    uint32_t key[NV];
    int bad = INT_MAX;  // smallest index of a non-finite logit (E = the shared gate)
#pragma unroll
    for (int j = 0; j < NV; ++j) {
        const int e = lane + j * kLanes;
        const float x = e < E ? load_as_f32(row, e) : -INFINITY;
        key[j] = e < E ? order_key(x) : 0u;  // 0 sorts below every real key (key(-inf) = 0x007fffff)
        if (e < E && !isfinite(x)) bad = min(bad, e);
    }
    float sl = 0.f;
    if (shared != nullptr) {
        sl = load_as_f32(shared, m * shared_ld);
        if (!isfinite(sl)) bad = min(bad, E);
    }
    bad = __reduce_min_sync(0xffffffffu, bad);
    if (bad != INT_MAX) {
        if (lane == 0) raise_error(err, (uint32_t)m, (uint32_t)bad);
        for (int a = lane; a < A; a += kLanes) {
            id_row[a] = -1;
            coef_row[a] = qnan_f32();
        }
        return;
    }

    float my_v = 0.f, top = 0.f;
    int my_i = -1;
    unsigned long long pick;
    if (k >= kPickSortMin<NV> && k <= kPickSort && picked_by_sort<NV>(key, lane, k, cand, pick)) {
        my_v = key_value((uint32_t)(pick >> 32)), my_i = (int)~(uint32_t)pick;
        top = __shfl_sync(0xffffffffu, my_v, 0);
    } else {
        // This lane's best: ascending scan with a strict > keeps the lower index on a tie.
        uint32_t lk;
        int li, lj;
        auto lane_best = [&] {
            lk = 0u, li = INT_MAX, lj = -1;
#pragma unroll
            for (int j = 0; j < NV; ++j)
                if (key[j] > lk) lk = key[j], li = lane + j * kLanes, lj = j;
        };
        lane_best();
        for (int r = 0; r < k; ++r) {
            const uint32_t best_key = __reduce_max_sync(0xffffffffu, lk);
            const int best_i = __reduce_min_sync(0xffffffffu, lk == best_key ? li : INT_MAX);
            if (lane == best_i % kLanes) {
#pragma unroll
                for (int j = 0; j < NV; ++j)
                    if (j == lj) key[j] = 0u;  // static register indices only
                lane_best();
            }
            __syncwarp();
            const float bv = key_value(best_key);
            if (r == 0) top = bv;
            if (lane == r) my_v = bv, my_i = best_i;
        }
    }

    // Softmax over the k picks; the sum is the reference's 32-lane xor butterfly, so equal exps give equal sums.
    const float ex = lane < k ? expf(my_v - top) : 0.f;
    float sum = ex;
#pragma unroll
    for (int off = kLanes / 2; off > 0; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
    if (lane < k) {
        id_row[lane] = my_i;
        coef_row[lane] = ex / sum;
    }
    if (shared != nullptr && lane == 0) {
        id_row[k] = shared_id;
        coef_row[k] = 1.0f / (1.0f + expf(-sl));
    }
}

}  // namespace sxb
