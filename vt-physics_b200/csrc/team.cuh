// Neighbour passes with several lanes per row, summing in list order.
//
// A row's L lanes (a team, consecutive lanes of a warp) take its list entries l, l + L, ... and
// evaluate each pair, kTeamDepth gathers in flight per lane, leaving the pair's terms in the warp's
// shared memory; then the team's lanes add the terms up entry by entry in list order, each lane
// its own accumulator.  The sums are the bits one thread walking the row gets, whatever L is; the
// gathers and the pair arithmetic - the latency and most of the instructions - run L rows' worth
// wide (the next batch's indices load while a batch is evaluated).  Used where a thread per row
// leaves most of the GPU idle and a pass takes one thread's serial walk (kTeamMaxRows, internal.h,
// says where that ends).
#pragma once

#include "common.cuh"

namespace vtp {

constexpr uint32_t kTeamRows = 32;                   // rows per block
constexpr uint32_t kTeamDepth = 4;                   // gathers in flight per lane

// Terms of a warp's rows: W words per entry (1, 4 or 8), L lanes per row (4 or 8), 4 L entries at a
// time; an odd number of entries between rows, so that rows fall in different banks.
template <int W, int L>
struct alignas(16) TeamTerms {
    static constexpr uint32_t kBatch = L * kTeamDepth, kPitch = kBatch + 1, kWarps = kTeamRows * L / 32;
    float t[kWarps][(32 / L) * kPitch * W];
};

template <int L>
__device__ __forceinline__ uint32_t team_lane() { return threadIdx.x % L; }
template <int L>
__device__ __forceinline__ uint32_t team_row() { return threadIdx.x / L; }   // row within the block

// The value lane `l` of the thread's team holds.
template <int L>
__device__ __forceinline__ float team_get(float v, uint32_t l) {
    return __shfl_sync(0xffffffffu, v, (int)l, L);
}

// Walks the `cnt` entries (0 for rows that do not exist) of every row of the warp; all lanes call
// it.  load(j) gathers neighbour j, term(j, data, out) evaluates the pair's W words, and add(entry)
// accumulates the calling lane's share of an entry's words, in list order.
template <int L, int W, class Load, class Term, class Add>
__device__ __forceinline__ void team_walk(TeamTerms<W, L> &S, const uint32_t *__restrict__ lst, uint32_t cnt, Load load,
                                          Term term, Add add) {
    static_assert(W == 1 || W == 4 || W == 8, "words per entry");
    using T = decltype(load(0u));
    constexpr uint32_t kBatch = TeamTerms<W, L>::kBatch;
    const uint32_t l = team_lane<L>();
    float *const mine = S.t[threadIdx.x >> 5] + ((threadIdx.x & 31u) / L) * (TeamTerms<W, L>::kPitch * W);
    uint32_t nxt[kTeamDepth];
#pragma unroll
    for (uint32_t u = 0; u < kTeamDepth; ++u)
        if (u * L + l < cnt) nxt[u] = __ldcs(lst + team_slot(u * L + l));
    for (uint32_t c0 = 0; __any_sync(0xffffffffu, c0 < cnt); c0 += kBatch) {
        uint32_t j[kTeamDepth];
        T d[kTeamDepth];
#pragma unroll
        for (uint32_t u = 0; u < kTeamDepth; ++u) j[u] = nxt[u];
#pragma unroll
        for (uint32_t u = 0; u < kTeamDepth; ++u)
            if (c0 + u * L + l < cnt) d[u] = load(j[u]);
        // the next batch's indices load while this batch is evaluated
#pragma unroll
        for (uint32_t u = 0; u < kTeamDepth; ++u) {
            const uint32_t t = c0 + kBatch + u * L + l;
            if (t < cnt) nxt[u] = __ldcs(lst + team_slot(t));
        }
#pragma unroll
        for (uint32_t u = 0; u < kTeamDepth; ++u) {
            const uint32_t e = u * L + l;
            if (c0 + e < cnt) {
                float o[W];
                term(j[u], d[u], o);
                float *p = mine + e * W;
                if constexpr (W == 1) {
                    *p = o[0];
                } else {
#pragma unroll
                    for (int w = 0; w < W; w += 4)
                        *reinterpret_cast<float4 *>(p + w) = make_float4(o[w], o[w + 1], o[w + 2], o[w + 3]);
                }
            }
        }
        __syncwarp();
        const uint32_t m = cnt > c0 ? min(cnt - c0, kBatch) : 0u;
#pragma unroll
        for (uint32_t e = 0; e < kBatch; ++e)
            if (e < m) add(mine + e * W);
        __syncwarp();
    }
}

}  // namespace vtp
