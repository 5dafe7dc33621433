// Pieces of the list builders that share work among a warp's lanes (ugns.cu, noalloc.cu): rows of one
// cell together (cell_rows), and several lanes per row that walk its cells (walk_rows).
#pragma once

#include "common.cuh"

namespace vtp {

// Two FP32 lanes of one 64-bit register pair (sm_100 packed arithmetic; each lane rounds as the
// scalar instruction does).
__device__ __forceinline__ uint64_t f2_pack(float a, float b) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float2 f2_unpack(uint64_t v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ uint64_t f2_add(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t f2_mul(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t f2_fma(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

// The general interleaving of a cell's fluid and boundary runs: merged by attach id.
__device__ __forceinline__ uint32_t merge_next(uint32_t &f, uint32_t f1, uint32_t &b, uint32_t b1,
                                               const uint32_t *__restrict__ orig) {
    if (b >= b1) return f++;
    if (f >= f1) return b++;
    return __ldg(orig + f) < __ldg(orig + b) ? f++ : b++;
}

constexpr int kCellWarps = 4;            // warps per block
constexpr uint32_t kCellWindow = 320;    // candidates laid out at a time (4 lanes x 80, 8 lanes x 40)
constexpr uint32_t kCellKept = 84;       // bytes of a lane's accepted candidates (80 used; 21 words apart: few conflicts)

// Rows a warp takes (SCAN): 8 up to this many, above that k_walk_lists or 32.
constexpr uint32_t kScan8Rows = 131072;
// Rows of one cell that follow one another are built together, 8 (SCAN 4: 4) at a time; the warp that
// holds the first builds the group, so a cell is spread over as many warps as it has groups.  A group
// of fewer rows than this is walked, unless its cell has kCrowded rows: a lane would walk their
// neighbourhood for each of them.  100,000 rows (B200, us) with groups of at least 3 / 4 / 5 / 6 rows: 50.6 / 53.8
// / 57.8 / 61.2 at half a cell's spacing, 90.6 / 102 / 103 / 124 at 0.35, 31.9 / 31.2 / 33.1 / 31.2
// at one; without walks 55.7, 162 and 88.4 (a warp per cell then).
constexpr uint32_t kGroupMin = 3, kGroupMin4 = 2;
constexpr uint32_t kCrowded = 64;
// With a lane per walked row (SCAN 32) the rows of a cell of more than this are walked: 400,000
// particles at 0.35 cells' spacing 499 us in groups, 358 so, at half a cell's spacing 206 us.
constexpr uint32_t kSharedRows = 16;

struct CellScratch {
    float x[3][kCellWindow];             // candidate positions of the window, in list order
    uint32_t cand[kCellWindow];          // their rows
    uint8_t kept[32][kCellKept];         // each lane's accepted candidates, as offsets into its share
};

// The fluid and boundary runs of one neighbour cell, and where its candidates start in list order.
// The t-th offset's are held by lane t < 27.
struct CellRuns {
    uint32_t f0, f1, b0, b1, excl;
};

// Places the lanes' runs one after another; returns the number of candidates.
__device__ __forceinline__ uint32_t place_runs(CellRuns &r) {
    constexpr unsigned kAll = 0xffffffffu;
    const uint32_t len = (r.f1 - r.f0) + (r.b1 - r.b0);
    uint32_t incl = len;
#pragma unroll
    for (uint32_t d = 1; d < 32u; d <<= 1) {
        const uint32_t y = __shfl_up_sync(kAll, incl, d);
        if ((threadIdx.x & 31u) >= d) incl += y;
    }
    r.excl = incl - len;
    return __shfl_sync(kAll, incl, 31);
}

// How many of the first o candidates of a cell merged by id are fluid rows: the merge path's crossing
// of diagonal o.
__device__ __forceinline__ uint32_t merge_split(const CellRuns &R, uint32_t o, const uint32_t *__restrict__ orig) {
    const uint32_t nf = R.f1 - R.f0, nb = R.b1 - R.b0;
    uint32_t lo = o > nb ? o - nb : 0u, hi = min(o, nf);
    while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        if (__ldg(orig + R.f0 + mid) < __ldg(orig + R.b0 + (o - mid - 1u))) lo = mid + 1u;
        else hi = mid;
    }
    return lo;
}

// Candidates [o, end) of a cell in list order into cand[0 .. end - o).
template <int MODE>
__device__ __forceinline__ void lay_out(uint32_t *cand, const CellRuns &R, uint32_t o, uint32_t end, uint32_t split,
                                        const uint32_t *__restrict__ orig) {
    if (MODE == 2) {
        uint32_t f = R.f0 + split, b = R.b0 + (o - split);
        for (; o < end; ++o) *cand++ = merge_next(f, R.f1, b, R.b1, orig);
    } else {
        const uint32_t a0 = MODE == 0 ? R.f0 : R.b0, na = (MODE == 0 ? R.f1 : R.b1) - a0;
        const uint32_t c0 = (MODE == 0 ? R.b0 : R.f0) - na;
        for (; o < end; ++o) *cand++ = (o < na ? a0 : c0) + o;
    }
}

// Runs longer than this are laid out by the whole warp, others by the lane that holds them (B200, us:
// 30,000 rows with 10,000 in one cell 578 -> 450, with 3,000 and 3,000 interleaved wall particles 887 ->
// 203; a fluid at rest has runs of eight, the same time).
constexpr uint32_t kLongRun = 32;

// Lays candidates [wb, wb + wl) out: rows (their ids from pos.w with IDS) and positions, infinity
// from wl up to `padded`.
template <int MODE, bool IDS>
__device__ __forceinline__ void stage_candidates(CellScratch &S, const CellRuns &R, uint32_t wb, uint32_t wl,
                                                 uint32_t padded, const float4 *__restrict__ pos,
                                                 const uint32_t *__restrict__ orig) {
    constexpr unsigned kAll = 0xffffffffu;
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t len = (R.f1 - R.f0) + (R.b1 - R.b0);
    // the part of this lane's runs that lies in the window
    const uint32_t o0 = wb > R.excl ? min(wb - R.excl, len) : 0u;
    const uint32_t o1 = wb + wl > R.excl ? min(wb + wl - R.excl, len) : 0u;
    __syncwarp();
    if (len <= kLongRun && o0 < o1)
        lay_out<MODE>(S.cand + (R.excl + o0 - wb), R, o0, o1, MODE == 2 ? merge_split(R, o0, orig) : 0u, orig);
    for (unsigned todo = __ballot_sync(kAll, len > kLongRun && o0 < o1); todo; todo &= todo - 1u) {
        const int src = __ffs((int)todo) - 1;
        CellRuns r;
        r.f0 = __shfl_sync(kAll, R.f0, src);
        r.f1 = __shfl_sync(kAll, R.f1, src);
        r.b0 = __shfl_sync(kAll, R.b0, src);
        r.b1 = __shfl_sync(kAll, R.b1, src);
        r.excl = __shfl_sync(kAll, R.excl, src);
        const uint32_t beg = __shfl_sync(kAll, o0, src), end = __shfl_sync(kAll, o1, src);
        const uint32_t each = (end - beg + 31u) / 32u, o = min(beg + lane * each, end);   // a lane's share of it
        if (o < end)
            lay_out<MODE>(S.cand + (r.excl + o - wb), r, o, min(o + each, end),
                          MODE == 2 ? merge_split(r, o, orig) : 0u, orig);
    }
    __syncwarp();
    for (uint32_t q = lane; q < padded; q += 32u) {
        const float far = __int_as_float(0x7f800000);
        float4 v = make_float4(far, far, far, 0.f);
        if (q < wl) {
            v = __ldg(pos + S.cand[q]);
            if (IDS) S.cand[q] = __float_as_uint(v.w);
        }
        S.x[0][q] = v.x;
        S.x[1][q] = v.y;
        S.x[2][q] = v.z;
    }
    __syncwarp();
}

// Appends `off` to the lane's accepted candidates at shared address `to` if 0 < d2 <= d2max
// (`0 < |x_i - x_j|` also drops the row itself): predicated, no branch.  The asm names no memory
// clobber, so that the next candidates' loads are not held up by it; kept_done() after the last of
// them tells the compiler of the stores.
__device__ __forceinline__ void keep_candidate(uint32_t &to, uint32_t off, float d2, float d2max) {
    asm(
        "{\n\t.reg .pred p;\n\t"
        "setp.gt.f32 p, %2, 0f00000000;\n\t"
        "setp.le.and.f32 p, %2, %3, p;\n\t"
        "@p st.shared.u8 [%0], %1;\n\t"
        "@p add.u32 %0, %0, 1;\n\t}"
        : "+r"(to)
        : "r"(off), "f"(d2), "f"(d2max));
}

// What keep_candidate stored may be read from here on.
__device__ __forceinline__ void kept_done() { asm volatile("" ::: "memory"); }

// Tests the 4 candidates at index `at` (offset `off` of the lane's share) against -p = (px, py, pz).
__device__ __forceinline__ void test4(const CellScratch &S, uint32_t at, uint32_t off, uint32_t &to, uint64_t px,
                                      uint64_t py, uint64_t pz, float d2max) {
    const ulonglong2 x = *reinterpret_cast<const ulonglong2 *>(&S.x[0][at]);
    const ulonglong2 y = *reinterpret_cast<const ulonglong2 *>(&S.x[1][at]);
    const ulonglong2 z = *reinterpret_cast<const ulonglong2 *>(&S.x[2][at]);
    const uint64_t ax = f2_add(px, x.x), ay = f2_add(py, y.x), az = f2_add(pz, z.x);
    const uint64_t bx = f2_add(px, x.y), by = f2_add(py, y.y), bz = f2_add(pz, z.y);
    const float2 a = f2_unpack(f2_fma(az, az, f2_fma(ay, ay, f2_mul(ax, ax))));
    const float2 b = f2_unpack(f2_fma(bz, bz, f2_fma(by, by, f2_mul(bx, bx))));
    keep_candidate(to, off, a.x, d2max);
    keep_candidate(to, off + 1u, a.y, d2max);
    keep_candidate(to, off + 2u, b.x, d2max);
    keep_candidate(to, off + 3u, b.y, d2max);
}

// Lists of up to R rows of one cell.  Lane l works for row l % R, lane h * R + k taking the h-th
// share of the candidates for row k: p is that row's position, `live` says whether it exists.
// `out` takes the entries (0-based, without the row itself).  Returns the row's number of entries,
// those past its list's end included.
template <int MODE, uint32_t R, class Out>
__device__ __forceinline__ uint32_t cell_rows(CellScratch &S, const CellRuns &runs, uint32_t total, bool live, float4 p,
                                              float d2max, const float4 *__restrict__ pos,
                                              const uint32_t *__restrict__ orig, const Out &out) {
    constexpr unsigned kAll = 0xffffffffu;
    constexpr uint32_t H = 32u / R;   // lanes per row
    const uint32_t lane = threadIdx.x & 31u, k = lane % R, h = lane / R;
    const uint64_t px = f2_pack(-p.x, -p.x), py = f2_pack(-p.y, -p.y), pz = f2_pack(-p.z, -p.z);
    const uint32_t to0 = (uint32_t)__cvta_generic_to_shared(&S.kept[lane][0]);
    uint32_t found = 0;   // entries of the row in earlier windows
    for (uint32_t wb = 0; wb < total; wb += kCellWindow) {
        const uint32_t wl = min(kCellWindow, total - wb);
        const uint32_t share = ((wl + H - 1u) / H + 7u) & ~7u;   // candidates per lane, in eights
        stage_candidates<MODE, Out::kIds>(S, runs, wb, wl, H * share, pos, orig);
        uint32_t to = to0;
        for (uint32_t off = 0; off < share; off += 8u) {
            test4(S, h * share + off, off, to, px, py, pz, d2max);
            test4(S, h * share + off + 4u, off + 4u, to, px, py, pz, d2max);
        }
        kept_done();
        const uint32_t mine = live ? to - to0 : 0u;
        uint32_t x = mine;
#pragma unroll
        for (uint32_t o = R; o < 32u; o <<= 1) {
            const uint32_t y = __shfl_up_sync(kAll, x, o);
            if (lane >= o) x += y;
        }
        __syncwarp();
        // The lists leave as they are stored: 8 entries of 4 rows, or H entries of R rows, at a
        // time.  Entry e of a row is in the share of the last lane whose entries start at or
        // before e.
        auto flush = [&](uint32_t kk, uint32_t e0, uint32_t step) {
            uint32_t lo[H];
#pragma unroll
            for (uint32_t t = 0; t < H; ++t) lo[t] = __shfl_sync(kAll, x - mine, (int)(kk + R * t));
            const uint32_t n = __shfl_sync(kAll, x, (int)(kk + 32u - R));
            const uint32_t before = __shfl_sync(kAll, found, (int)kk);
            uint32_t *dst = out.of(kk);
            for (uint32_t e = e0; e < n; e += step) {
                uint32_t at = kk * kCellKept + e, share_of = 0;
#pragma unroll
                for (uint32_t t = 1; t < H; ++t)
                    if (e >= lo[t]) at = (kk + R * t) * kCellKept + (e - lo[t]), share_of = t * share;
                out.put(dst, before + e, S.cand[share_of + (&S.kept[0][0])[at]]);
            }
        };
        if (out.eights()) {
#pragma unroll
            for (uint32_t r = 0; r < R; r += 4) flush(r + (lane >> 3), lane & 7u, 8u);
        } else {
            flush(k, h, H);
        }
        found += __shfl_sync(kAll, x, (int)(k + 32u - R));
    }
    return found;
}

// Accepted candidates a lane of walk_rows keeps.
constexpr uint32_t kWalkKeep = 3u * kCellWindow / 32u;

// The candidates of one cell in list order, positions loaded four at a time: use(j, its position).
template <int MODE, class Use>
__device__ __forceinline__ void visit_cell(const CellRuns &r, const float4 *__restrict__ pos,
                                           const uint32_t *__restrict__ orig, Use use) {
    auto run = [&](uint32_t j, uint32_t end) {
        for (; j + 4 <= end; j += 4) {
            const float4 q0 = __ldg(pos + j), q1 = __ldg(pos + j + 1), q2 = __ldg(pos + j + 2), q3 = __ldg(pos + j + 3);
            use(j, q0);
            use(j + 1, q1);
            use(j + 2, q2);
            use(j + 3, q3);
        }
        for (; j < end; ++j) use(j, __ldg(pos + j));
    };
    if (MODE == 0) {
        run(r.f0, r.f1);
        run(r.b0, r.b1);
    } else if (MODE == 1) {
        run(r.b0, r.b1);
        run(r.f0, r.f1);
    } else {
        for (uint32_t f = r.f0, b = r.b0; f < r.f1 || b < r.b1;) {
            const uint32_t j = merge_next(f, r.f1, b, r.b1, orig);
            use(j, __ldg(pos + j));
        }
    }
}

// Lists of rows whatever cells they lie in, walked side by side: the lanes of `todo` hold a row each.
// The warp's lanes are shared out among them (32 rows a lane each, 16 two, ... one all), a row's lanes
// each taking a contiguous part of its 27 cells.  A lane keeps what it accepts in a column of the
// scratch until the lanes before it are counted; one with more than fits there walks its cells again.
// open(lane) gives the row that lane holds (called by all lanes), with its position `p`, runs(t), the
// runs of its t-th offset, and `out`; close(row, found, lead) ends it (lead: one lane per row).
template <int MODE, class Open, class Close>
__device__ __forceinline__ void walk_rows(CellScratch &S, unsigned todo, float d2max, const float4 *__restrict__ pos,
                                          const uint32_t *__restrict__ orig, const Open &open, const Close &close) {
    constexpr unsigned kAll = 0xffffffffu;
    const uint32_t lane = threadIdx.x & 31u, w = (uint32_t)__popc(todo);
    if (w == 0u) return;
    __syncwarp();
    if ((todo >> lane) & 1u) S.cand[__popc(todo & ((1u << lane) - 1u))] = lane;
    __syncwarp();
    const uint32_t lg = w > 1u ? 32u - (uint32_t)__clz((int)(w - 1u)) : 0u;   // 2^lg >= w rows side by side
    const uint32_t k = lane & ((1u << lg) - 1u), h = lane >> lg, lgh = 5u - lg;
    const bool live = k < w;
    const auto row = open(S.cand[live ? k : 0u]);
    const float4 p = row.p;
    const int t0 = (int)((27u * h) >> lgh), t1 = live ? (int)((27u * (h + 1u)) >> lgh) : t0;
    uint32_t *const dst = row.out.mine();
    constexpr bool kIds = decltype(row.out)::kIds;
    auto walk = [&](auto accept) {
        for (int t = t0; t < t1; ++t)
            visit_cell<MODE>(row.runs(t), pos, orig, [&](uint32_t j, const float4 &q) {
                const float d2 = dist2(p.x - q.x, p.y - q.y, p.z - q.z);
                accept(kIds ? __float_as_uint(q.w) : j, d2 > 0.f && d2 <= d2max);
            });
    };
    uint32_t slot = 0, x = 0;
    bool kept = false;
    if (lgh > 0u) {
        uint32_t *const keep = reinterpret_cast<uint32_t *>(&S.x[0][0]) + lane;   // entry e at keep[32 e]
        uint32_t n = 0;
        walk([&](uint32_t j, bool yes) {
            if (yes && n < kWalkKeep) keep[32u * n] = j;
            n += yes ? 1u : 0u;
        });
        x = n;
        for (uint32_t o = 1u << lg; o < 32u; o <<= 1) {
            const uint32_t y = __shfl_up_sync(kAll, x, o);
            if (lane >= o) x += y;
        }
        slot = x - n;
        kept = n <= kWalkKeep;
        if (kept)
            for (uint32_t e = 0; e < n; ++e) row.out.put(dst, slot + e, keep[32u * e]);
    }
    if (!kept) {
        walk([&](uint32_t j, bool yes) {
            if (yes) row.out.put(dst, slot, j);
            slot += yes ? 1u : 0u;
        });
        if (lgh == 0u) x = slot;
    }
    close(row, __shfl_sync(kAll, x, (int)(k + 32u - (1u << lg))), live && h == 0u);
    __syncwarp();
}

}  // namespace vtp
