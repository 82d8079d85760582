// One-to-one keys (one per target: distance << 32 | query, all ones where the target has no match) to
// matches ordered by target (matching._unique, app/planesite/matching.py:103-110).
#pragma once

#include <stdint.h>

namespace fsb {

// target-ordered compaction of the one-to-one keys by one block: one launch where flags, a device
// select (two kernels) and a gather take four; up to kCompactMax targets (5 us at 9000)
constexpr int kCompactMax = 32768;
constexpr int COMPACT_T = 1024;
__device__ __forceinline__ void unique_compact(const unsigned long long* __restrict__ key, int nb, int64_t* __restrict__ q,
                                               int64_t* __restrict__ t, int32_t* __restrict__ n_out) {
    // each warp owns a run of the targets and walks it 32 at a time, twice: count, then place
    __shared__ int s_cnt[COMPACT_T / 32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int per = ((nb + COMPACT_T - 1) / COMPACT_T) * 32;
    const int t0 = min(w * per, nb), t1 = min(t0 + per, nb);
    int cnt = 0;
#pragma unroll 4
    for (int i = t0; i < t1; i += 32)
        cnt += __popc(__ballot_sync(0xffffffffu, i + lane < t1 && key[i + lane] != ~0ull));
    if (lane == 0) s_cnt[w] = cnt;
    __syncthreads();
    int off = 0, total = 0;
    for (int k = 0; k < COMPACT_T / 32; ++k) {
        off += k < w ? s_cnt[k] : 0;
        total += s_cnt[k];
    }
    for (int i = t0; i < t1; i += 32) {
        const unsigned long long k = i + lane < t1 ? key[i + lane] : ~0ull;
        const unsigned m = __ballot_sync(0xffffffffu, k != ~0ull);
        if (k != ~0ull) {
            const int at = off + __popc(m & ((1u << lane) - 1u));
            q[at] = (int64_t)(k & 0xffffffffull);
            t[at] = i + lane;
        }
        off += __popc(m);
    }
    if (threadIdx.x == 0) *n_out = total;
}

}  // namespace fsb
