// Uniform-grid neighbour search for sm_100a.
//
// Replaces UniformGirdNeighborSearcher::update / cu_update
// (Simulator/Runtime/Source/Modules/NeighborSearch/UGNS/UGNSCudaImpl.cu:96-227).
// Instead of two thrust::sort_by_key calls, a 27-cell neighbour walk over
// particles in attach order and a padded N x maxNbr list, each substep does:
//   hash    : cell key per row + arrival rank inside the cell (atomicAdd)
//   scan    : exclusive scan of the per-cell counts -> cell start table
//   scatter : rows placed into their cell's segment (arrival order)
//   rank    : inside each segment, rank by attach id -> stable (cell, id)
//             order, identical to the reference's stable radix sort, and
//             move the particle state to its new row (float4 SoA)
//   lists   : neighbour list per row in the reference's order (27 offsets
//             in fixed order, ascending attach id inside a cell), stored as
//             a warp-interleaved ELL array of sorted row indices.
#include "internal.h"
#include "cells.cuh"
#include "staged.h"

#include <type_traits>


namespace vtp {

namespace {

// Up to this many rows a warp of k_build_lists takes 4, with eight lanes a row: twice the warps, each
// with half the work in sequence.
constexpr uint32_t kScan4Rows = 16384;
constexpr int kWalkBlock = 128;
constexpr int kScanThreads = 256;
constexpr int kScanItems = 8;
constexpr int kScanTile = kScanThreads * kScanItems;

__device__ __forceinline__ float4 apply_force(float4 p, float4 &v, float dt, float3 g) {
    // apply_ext_force_cuda (PBFCudaImpl.cu:146-157): v += g dt; x += v dt.
    v.x = __fmaf_rn(g.x, dt, v.x);
    v.y = __fmaf_rn(g.y, dt, v.y);
    v.z = __fmaf_rn(g.z, dt, v.z);
    p.x = __fmaf_rn(v.x, dt, p.x);
    p.y = __fmaf_rn(v.y, dt, p.y);
    p.z = __fmaf_rn(v.z, dt, p.z);
    return p;
}

// Bucket and arrival rank of one row, its bucket's counter advanced.
__device__ __forceinline__ uint32_t hash_row(const Scenes &sc, uint32_t row0, uint32_t i,
                                             const float4 *__restrict__ pos, const float4 *__restrict__ vel,
                                             float force_dt, uint32_t *__restrict__ rank,
                                             uint32_t *__restrict__ count) {
    const SceneGrid g = load_scene(sc, row0 + i);
    float4 p = pos[row0 + i];
    if (force_dt > 0.f) {
        float4 v = vel[row0 + i];
        p = apply_force(p, v, force_dt, make_float3(g.grav_x, g.grav_y, g.grav_z));
    }
    int3 c = cell_of(p.x, p.y, p.z, g, sc.cell);
    const bool outside = !cell_available(c, g);
    uint32_t k = g.key_base + (outside ? g.nkey : cell_key(c, g));
    const unsigned om = __ballot_sync(__activemask(), outside);
    if (outside) {
        // Every row outside its scene's grid counts into the scene's one outside bucket (whole
        // scenes can leave the box); one atomic per group of lanes with the same bucket keeps
        // that counter from serialising the kernel.  The order inside the outside bucket is
        // arbitrary either way: its rows have no neighbours and are nobody's neighbour.
        const unsigned grp = __match_any_sync(om, k);
        const unsigned lane = threadIdx.x & 31u;
        const int leader = __ffs(grp) - 1;
        uint32_t base = 0;
        if ((int)lane == leader) base = atomicAdd(&count[k], (uint32_t)__popc(grp));
        base = __shfl_sync(grp, base, leader);
        rank[i] = base + (uint32_t)__popc(grp & ((1u << lane) - 1u));
    } else {
        rank[i] = atomicAdd(&count[k], 1u);
    }
    return k;
}

// `sums` (or null): the scan's tile sums are counted as well.
__global__ void k_hash(Scenes sc, uint32_t row0, uint32_t cnt, const float4 *__restrict__ pos,
                       const float4 *__restrict__ vel, float force_dt, uint32_t *__restrict__ key,
                       uint32_t *__restrict__ rank, uint32_t *__restrict__ count, uint32_t *__restrict__ sums) {
    pdl_enter();
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t k = 0;
    if (i < cnt) {
        k = hash_row(sc, row0, i, pos, vel, force_dt, rank, count);
        key[i] = k;
    }
    if (!sums) return;
    // The rows are nearly sorted already: a block's rows mostly fall in its first row's tile, and
    // go in with one atomic (one per warp cost 10 us at 1,000,000 rows).
    __shared__ uint32_t first;
    const uint32_t t = k / kScanTile;
    if (threadIdx.x == 0) first = t;
    __syncthreads();
    const bool other = i < cnt && t != first;
    const int n = __syncthreads_count(i < cnt && !other);
    if (threadIdx.x == 0) atomicAdd(&sums[first], (uint32_t)n);
    if (other) atomicAdd(&sums[t], 1u);
}

// Block-wide exclusive scan of one value per thread; returns the block total.
__device__ __forceinline__ uint32_t block_excl_scan(uint32_t v, uint32_t &total) {
    __shared__ uint32_t warp_sums[32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) warp_sums[wid] = x;
    __syncthreads();
    const int nw = blockDim.x >> 5;
    if (wid == 0) {
        uint32_t s = lane < nw ? warp_sums[lane] : 0u;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            uint32_t y = __shfl_up_sync(0xffffffffu, s, o);
            if (lane >= o) s += y;
        }
        if (lane < nw) warp_sums[lane] = s;
    }
    __syncthreads();
    uint32_t warp_off = wid > 0 ? warp_sums[wid - 1] : 0u;
    total = warp_sums[nw - 1];
    __syncthreads();
    return warp_off + x - v;
}

__global__ void __launch_bounds__(kScanThreads) k_scan_tile_sums(const uint32_t *__restrict__ in, size_t n,
                                                                 uint32_t *__restrict__ sums) {
    pdl_enter();
    size_t base = (size_t)blockIdx.x * kScanTile + threadIdx.x;
    uint32_t s = 0;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        size_t idx = base + (size_t)k * kScanThreads;
        if (idx < n) s += in[idx];
    }
    uint32_t total;
    block_excl_scan(s, total);
    if (threadIdx.x == 0) sums[blockIdx.x] = total;
}

__global__ void __launch_bounds__(1024) k_scan_sums(uint32_t *sums, size_t tiles) {
    pdl_enter();
    // One block; each thread owns a contiguous run of tiles.
    const size_t per = (tiles + blockDim.x - 1) / blockDim.x;
    size_t b = threadIdx.x * per;
    uint32_t local = 0;
    for (size_t k = 0; k < per; ++k)
        if (b + k < tiles) local += sums[b + k];
    uint32_t total;
    uint32_t off = block_excl_scan(local, total);
    for (size_t k = 0; k < per; ++k) {
        if (b + k < tiles) {
            uint32_t v = sums[b + k];
            sums[b + k] = off;
            off += v;
        }
    }
}

// Exclusive scan of the counters into `out` (plus `base_add`), out[n] = grand
// total.  The counters are zeroed after they are read, so the next hash starts
// from zero without a separate clear.  PREFIX: `sums` holds the tiles' own sums
// (counted by k_hash) and each block adds up those before it; else their scan.
template <bool PREFIX>
__global__ void __launch_bounds__(kScanThreads) k_scan_tiles(uint32_t *__restrict__ in, size_t n,
                                                             const uint32_t *__restrict__ sums, uint32_t base_add,
                                                             uint32_t *__restrict__ out) {
    pdl_enter();
    uint32_t before = 0;
    if (PREFIX) {
        uint32_t v = 0;
        for (uint32_t t = threadIdx.x; t < blockIdx.x; t += kScanThreads) v += sums[t];
        block_excl_scan(v, before);
    }
    // Each thread scans kScanItems consecutive counters.
    __shared__ uint32_t tile[kScanTile];
    size_t t0 = (size_t)blockIdx.x * kScanTile;
    for (int k = 0; k < kScanItems; ++k) {
        size_t idx = t0 + (size_t)k * kScanThreads + threadIdx.x;
        tile[k * kScanThreads + threadIdx.x] = idx < n ? in[idx] : 0u;
        if (idx < n) in[idx] = 0u;
    }
    __syncthreads();
    uint32_t vals[kScanItems];
    uint32_t s = 0;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        vals[k] = tile[threadIdx.x * kScanItems + k];
        s += vals[k];
    }
    uint32_t total;
    uint32_t off = block_excl_scan(s, total) + (PREFIX ? before : sums[blockIdx.x]) + base_add;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        const size_t idx = t0 + (size_t)threadIdx.x * kScanItems + k;
        if (idx + 1 == n) out[n] = off + vals[k];
        tile[threadIdx.x * kScanItems + k] = off;
        off += vals[k];
    }
    __syncthreads();
    for (int k = 0; k < kScanItems; ++k) {
        size_t idx = t0 + (size_t)k * kScanThreads + threadIdx.x;
        if (idx < n) out[idx] = tile[k * kScanThreads + threadIdx.x];
    }
}

__global__ void k_scatter(uint32_t row0, uint32_t cnt, const uint32_t *__restrict__ key,
                          const uint32_t *__restrict__ rank, const uint32_t *__restrict__ start,
                          const uint32_t *__restrict__ orig, uint32_t *__restrict__ tmp_src,
                          uint32_t *__restrict__ tmp_orig, uint32_t *__restrict__ tmp_key, uint32_t *status,
                          uint32_t *__restrict__ sums, uint32_t tiles) {
    pdl_enter();
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (sums)   // the scan has read them: zero for the next hash
        for (uint32_t t = i; t < tiles; t += gridDim.x * blockDim.x) sums[t] = 0u;
    if (i >= cnt) return;
    uint32_t k = key[i];
    uint32_t d = start[k] - row0 + rank[i];
#ifdef VTP_CHECKED
    if (d >= cnt) {   // a cell segment slot outside the sorted range: record it and skip the write
        if (status) atomicOr(status, ST_BOUNDS);
        return;
    }
#endif
    tmp_src[d] = i;
    tmp_orig[d] = orig[row0 + i];
    tmp_key[d] = k;
}

__global__ void k_rank_reorder(Scenes sc, uint32_t row0, uint32_t cnt, const uint32_t *__restrict__ start,
                               const uint32_t *__restrict__ tmp_src, const uint32_t *__restrict__ tmp_orig,
                               const uint32_t *__restrict__ tmp_key, const float4 *__restrict__ pos_in,
                               float4 *__restrict__ pos_out, const float4 *__restrict__ vel_in,
                               float4 *__restrict__ vel_out, uint32_t *__restrict__ orig_out, Carry carry,
                               float force_dt) {
    pdl_enter();
    uint32_t d = blockIdx.x * blockDim.x + threadIdx.x;
    if (d >= cnt) return;
    // A row keeps its scene: slot d lies in the same scene range as its source row.
    const SceneGrid g = load_scene(sc, row0 + d);
    uint32_t k = tmp_key[d];
    uint32_t my = tmp_orig[d];
    uint32_t dst = d;
    if (k < g.key_base + g.nkey) {
        // Stable order inside the cell: rank by attach id.
        uint32_t s0 = start[k] - row0, s1 = start[k + 1] - row0;
        uint32_t r = 0;
        for (uint32_t x = s0; x < s1; ++x) r += (tmp_orig[x] < my) ? 1u : 0u;
        dst = s0 + r;
    }
    uint32_t s = tmp_src[d];
    float4 p = pos_in[row0 + s];
    float4 v = vel_in[row0 + s];
    if (force_dt > 0.f) p = apply_force(p, v, force_dt, make_float3(g.grav_x, g.grav_y, g.grav_z));
    pos_out[row0 + dst] = p;
    vel_out[row0 + dst] = v;
    orig_out[row0 + dst] = my;
    for (int f = 0; f < carry.nf4; ++f) carry.dst4[f][row0 + dst] = carry.src4[f][row0 + s];
    for (int f = 0; f < carry.nf1; ++f) carry.dst1[f][row0 + dst] = carry.src1[f][row0 + s];
}

// Cell culling: distances from a row's position to the six faces of its own
// cell, shrunk by a safety margin.  A neighbour cell whose nearest point lies
// farther than h (d2 > d2max) holds no particle the membership test can accept
// (UGNSCudaImpl.cu:189-199 tests every particle of all 27 cells), so skipping
// it leaves the list unchanged.  The margin (1e-3 cell plus 1e-6 of the
// coordinate's magnitude) covers the rounding of the face positions and of
// the cell assignment floor((x - lb) / cell), both a few ulps of the
// coordinate; a cell inside the margin is simply walked.
struct FaceGaps {
    float lx, hx, ly, hy, lz, hz;   // clearance below / above along each axis (>= 0)

    __device__ __forceinline__ void init(const float4 &p, int3 c, const SceneGrid &g, float cell) {
        gap(p.x, c.x, g.lbx, cell, lx, hx);
        gap(p.y, c.y, g.lby, cell, ly, hy);
        gap(p.z, c.z, g.lbz, cell, lz, hz);
    }
    __device__ __forceinline__ static void gap(float x, int c, float lb, float cell, float &lo, float &hi) {
        const float f0 = __fmaf_rn((float)c, cell, lb);           // lower face of the cell
        const float m = __fmaf_rn(1e-6f, fabsf(f0) + cell, 1e-3f * cell);
        lo = fmaxf(x - f0 - m, 0.f);
        hi = fmaxf(f0 + cell - x - m, 0.f);
    }
    // Whether the neighbour cell at offset o can hold a particle within h.
    __device__ __forceinline__ bool reachable(int3 o, float d2max) const {
        const float ex = o.x < 0 ? lx : (o.x > 0 ? hx : 0.f);
        const float ey = o.y < 0 ? ly : (o.y > 0 ? hy : 0.f);
        const float ez = o.z < 0 ? lz : (o.z > 0 ? hz : 0.f);
        return dist2(ex, ey, ez) <= d2max;
    }
};

// One candidate of the neighbour walk (UGNSCudaImpl.cu:189-199).
template <class Slots>
struct Walker {
    float px, py, pz;
    uint32_t self;
    uint32_t cnt;        // entries written incl. self
    uint32_t maxnbr;
    uint32_t *out;       // the row's first list entry
    Slots at;            // offsets of the others
    bool overflow;

    // The row itself (d2 == 0) fails `d2 > 0` like every coincident particle,
    // as the reference's `0 < |x_i - x_j|` test excludes it.
    __device__ __forceinline__ void accept(uint32_t j, const float4 &q, float d2max) {
        float d2 = dist2(px - q.x, py - q.y, pz - q.z);
        if (d2 > 0.f && d2 <= d2max) {
            if (cnt < maxnbr) {
                out[at(cnt - 1)] = j;
                ++cnt;
            } else {
                overflow = true;
            }
        }
    }

    // Same test without the capacity check, for a cell whose candidates all fit
    // in the list.
    __device__ __forceinline__ void accept_room(uint32_t j, const float4 &q, float d2max) {
        const float d2 = dist2(px - q.x, py - q.y, pz - q.z);
        const bool acc = d2 > 0.f && d2 <= d2max;
        if (acc) out[at(cnt - 1)] = j;
        cnt += acc ? 1u : 0u;
    }

    template <bool ROOM>
    __device__ __forceinline__ void test(uint32_t j, const float4 &q, float d2max) {
        if (ROOM) accept_room(j, q, d2max);
        else accept(j, q, d2max);
    }

    template <bool ROOM>
    __device__ __forceinline__ void visit(uint32_t j, const float4 *__restrict__ pos, float d2max) {
        test<ROOM>(j, __ldg(pos + j), d2max);
    }

    // Candidates [j0, j1) in order; positions loaded four at a time.
    template <bool ROOM>
    __device__ __forceinline__ void visit_run(uint32_t j0, uint32_t j1, const float4 *__restrict__ pos,
                                              float d2max) {
        uint32_t j = j0;
        for (; j + 4 <= j1; j += 4) {
            const float4 q0 = __ldg(pos + j), q1 = __ldg(pos + j + 1), q2 = __ldg(pos + j + 2),
                         q3 = __ldg(pos + j + 3);
            test<ROOM>(j, q0, d2max);
            test<ROOM>(j + 1, q1, d2max);
            test<ROOM>(j + 2, q2, d2max);
            test<ROOM>(j + 3, q3, d2max);
        }
        for (; j < j1; ++j) visit<ROOM>(j, pos, d2max);
    }

    // One cell: fluid run [f0, f1) and boundary run [b0, b1) in MODE's order.
    template <int MODE, bool ROOM>
    __device__ __forceinline__ void visit_cell(uint32_t f0, uint32_t f1, uint32_t b0, uint32_t b1,
                                               const float4 *__restrict__ pos, const uint32_t *__restrict__ orig,
                                               float d2max) {
        if (MODE == 0) {
            visit_run<ROOM>(f0, f1, pos, d2max);
            visit_run<ROOM>(b0, b1, pos, d2max);
        } else if (MODE == 1) {
            visit_run<ROOM>(b0, b1, pos, d2max);
            visit_run<ROOM>(f0, f1, pos, d2max);
        } else {
            // Merge the two id-sorted runs by attach id.
            while (f0 < f1 || b0 < b1) {
                uint32_t j;
                if (b0 >= b1) j = f0++;
                else if (f0 >= f1) j = b0++;
                else j = (__ldg(orig + f0) < __ldg(orig + b0)) ? f0++ : b0++;
                visit<ROOM>(j, pos, d2max);
            }
        }
    }
};

// One thread per row walks its 27 cells and appends to its list: the builder of more than
// kScan8Rows rows in lists of shape lg 0, where every SM has rows enough.  250,000 rows (B200, us),
// against a warp per cell and against k_build_lists with 32 rows a warp: a dam break at rest 74 (70,
// 64), after 150 substeps 101 (119, 124), clouds 0.35, 0.5, 0.7 and 1 cells apart 229 (348, 235), 98
// (117, 104), 76 (125, 111), 44 (191, 51), with 4,000 rows in one cell 390 (8,230, 740).
template <int MODE, bool CULL, class Slots>
__global__ void k_walk_lists(Scenes sc, uint32_t row0, uint32_t cnt, ListShape shape,
                              const float4 *__restrict__ pos, const uint32_t *__restrict__ orig,
                              const uint32_t *__restrict__ fstart, const uint32_t *__restrict__ bstart,
                              uint32_t *__restrict__ nbr, uint32_t *__restrict__ ncnt,
                              uint32_t *__restrict__ status, uint32_t *__restrict__ overflow_count) {
    pdl_enter();
    uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= cnt) return;
    uint32_t i = row0 + r;
    const SceneGrid g = load_scene(sc, i);
    float4 p = pos[i];
    int3 c = cell_of(p.x, p.y, p.z, g, sc.cell);
    if (!cell_available(c, g)) {  // outside the grid: no neighbours, not even self
        ncnt[r] = 0;
        return;
    }
    Walker<Slots> w;
    w.px = p.x; w.py = p.y; w.pz = p.z;
    w.self = i;
    w.cnt = 1;
    w.maxnbr = sc.maxnbr;
    if constexpr (std::is_same_v<Slots, AnySlots>) w.at = AnySlots{shape};
    w.out = nbr + ell_index(r, 0, shape);
    w.overflow = false;
    const float d2max = sc.d2max;
    FaceGaps fg;
    if (CULL) fg.init(p, c, g, sc.cell);
    for (int t = 0; t < 27; ++t) {
        int3 cc = c;
        int3 o = nbr_offset(t);
        cc.x += o.x; cc.y += o.y; cc.z += o.z;
        if (!cell_available(cc, g)) continue;
        if (CULL && !fg.reachable(o, d2max)) continue;
        uint32_t k = g.key_base + cell_key(cc, g);
        uint32_t f0 = __ldg(fstart + k), f1 = __ldg(fstart + k + 1);
        uint32_t b0 = __ldg(bstart + k), b1 = __ldg(bstart + k + 1);
        // The capacity check is needed only when the cell's candidates could
        // overflow the list.
        if (w.cnt + (f1 - f0) + (b1 - b0) <= w.maxnbr) w.visit_cell<MODE, true>(f0, f1, b0, b1, pos, orig, d2max);
        else w.visit_cell<MODE, false>(f0, f1, b0, b1, pos, orig, d2max);
    }
    ncnt[r] = w.cnt;
    if (w.overflow) {
        atomicAdd(overflow_count, 1u);
        atomicOr(status, ST_BOUNDS);
    }
}

// Where the entries of a solver's lists go.  `row`: list row of this lane's row.
struct ListOut {
    static constexpr bool kIds = false;   // entries are sorted rows
    ListShape shape;
    uint32_t *nbr;
    uint32_t row, cap;
    __device__ __forceinline__ bool eights() const { return shape.lg != 0u; }
    __device__ __forceinline__ uint32_t *mine() const { return nbr + ell_index(row, 0, shape); }
    __device__ __forceinline__ uint32_t *of(uint32_t lane) const {
        return nbr + ell_index(__shfl_sync(0xffffffffu, row, (int)lane), 0, shape);
    }
    __device__ __forceinline__ void put(uint32_t *dst, uint32_t slot, uint32_t j) const {
        if (slot < cap) dst[ell_slot(slot, shape)] = j;
    }
};

// The runs of the neighbour cell at offset t of cell c.
__device__ __forceinline__ CellRuns runs_at(int3 c, int t, const SceneGrid &g, const uint32_t *__restrict__ fstart,
                                            const uint32_t *__restrict__ bstart) {
    CellRuns r{};
    const int3 o = nbr_offset(t);
    const int3 cc = make_int3(c.x + o.x, c.y + o.y, c.z + o.z);
    if (cell_available(cc, g)) {
        const uint32_t b = g.key_base + cell_key(cc, g);
        r.f0 = __ldg(fstart + b); r.f1 = __ldg(fstart + b + 1);
        r.b0 = __ldg(bstart + b); r.b1 = __ldg(bstart + b + 1);
    }
    return r;
}

// A row for walk_rows.
struct WalkedRow {
    float4 p;
    int3 c;
    uint32_t i;
    SceneGrid g;
    const uint32_t *fstart, *bstart;
    ListOut out;
    __device__ __forceinline__ CellRuns runs(int t) const { return runs_at(c, t, g, fstart, bstart); }
};

// The list builder up to kScan8Rows rows: a warp takes SCAN consecutive sorted rows.  The rows of a
// cell share their 27 neighbour cells, so groups of rows of one cell are built together: the warp lays
// the candidates of those cells out in shared memory, in list order (27 offsets in the reference's
// order, each cell's two runs in MODE's order), the row's lanes each test a contiguous share of them,
// two to a packed FP32 instruction (the roundings of dist2), and keep the accepted ones as byte
// offsets into the share; the lanes' counts, scanned over the row, give each lane its first slot
// (cell_rows, cells.cuh).  Rows of groups too small to share that work are walked side by side
// (walk_rows).  Event-timed launches (B200, us), eight lanes per row -> a warp per cell -> this.  Dam
// breaks at rest: PBF 16,000 rows 23 -> 13 -> 15, 64,000 rows 68 -> 25 -> 23, 120,000 rows 109 -> 44 ->
// 41, DFSPH 16,000 rows 23 -> 17 -> 17, 128,000 rows 113 -> 50 -> 48.  After 100-200 substeps: 21 -> 21 ->
// 23, 50 -> 48 -> 47, 80 -> 72 -> 64, 21 -> 21 -> 23, 80 -> 76 -> 62.  Clouds of 100,000 rows 0.35, 0.7 and
// 1 cells apart: 188 -> 162 -> 91, 44 -> 58 -> 56, 27 -> 88 -> 33.  30,000 rows with 10,000 in one cell:
// 750 -> 46,900 -> 450.  Bound by latencies: at 120,000 rows 44 % of the issue slots, 64 % of the L1
// rate, and the 36 % of the warp slots that its shared memory allows.
template <int MODE, uint32_t SCAN>
__global__ void __launch_bounds__(kCellWarps * 32, 7) k_build_lists(
    Scenes sc, uint32_t row0, uint32_t cnt, ListShape shape, const float4 *__restrict__ pos,
    const uint32_t *__restrict__ orig, const uint32_t *__restrict__ start, const uint32_t *__restrict__ fstart,
    const uint32_t *__restrict__ bstart, uint32_t *__restrict__ nbr, uint32_t *__restrict__ ncnt,
    uint32_t *__restrict__ status, uint32_t *__restrict__ overflow_count) {
    pdl_enter();
    __shared__ __align__(16) CellScratch scratch[kCellWarps];
    constexpr unsigned kAll = 0xffffffffu;
    constexpr uint32_t R = SCAN == 4u ? 4u : 8u;   // rows of a group
    const uint32_t lane = threadIdx.x & 31u, k = lane % SCAN;
    const uint32_t first = (blockIdx.x * kCellWarps + (threadIdx.x >> 5)) * SCAN;
    if (first >= cnt) return;
    CellScratch &S = scratch[threadIdx.x >> 5];
    const float d2max = sc.d2max;
    const uint32_t cap = sc.maxnbr - 1u;

    // This lane's row of the warp's SCAN rows, and the group it is in.
    const uint32_t n = min(SCAN, cnt - first), i = row0 + first + min(k, n - 1u);
    const SceneGrid g = load_scene(sc, i);
    const float4 p = pos[i];
    const int3 own = cell_of(p.x, p.y, p.z, g, sc.cell);
    uint32_t rows = 0;   // of the group that starts at row i
    bool walked = false;
    if (cell_available(own, g)) {
        const uint32_t b = g.key_base + cell_key(own, g), s = __ldg(start + b), e = __ldg(start + b + 1);
        const uint32_t in_group = (i - s) % R, m = min(R, e - (i - in_group));
        const bool together = m >= (SCAN == 4u ? kGroupMin4 : kGroupMin) || e - s > kCrowded;
        if (together && in_group == 0u && lane < n) rows = m;
        walked = !together && k < n;
    } else if (lane < n) {
        ncnt[first + lane] = 0;   // outside the grid: no neighbours, not even self
    }
    for (unsigned todo = __ballot_sync(kAll, rows != 0u); todo; todo &= todo - 1u) {
        const int leader = __ffs((int)todo) - 1;
        const uint32_t m = __shfl_sync(kAll, rows, leader), beg = __shfl_sync(kAll, i, leader);
        const uint32_t kr = lane % R, row = beg + min(kr, m - 1u);
        const SceneGrid gg = load_scene(sc, beg);
        const float4 q = pos[row];
        int3 c0 = make_int3(__shfl_sync(kAll, own.x, leader), __shfl_sync(kAll, own.y, leader),
                            __shfl_sync(kAll, own.z, leader));
        // A bucket of the bricked order is one cell.  In the linear order a cell on the grid's
        // inclusive upper face shares its bucket with another cell: one round per cell then.
        for (unsigned left = (1u << m) - 1u; left;) {
            bool mine = kr < m;
            if (gg.brick) {
                left = 0;
            } else {
                const int3 c = cell_of(q.x, q.y, q.z, gg, sc.cell);
                const int f = __ffs((int)left) - 1;
                c0 = make_int3(__shfl_sync(kAll, c.x, f), __shfl_sync(kAll, c.y, f), __shfl_sync(kAll, c.z, f));
                mine = ((left >> kr) & 1u) && c.x == c0.x && c.y == c0.y && c.z == c0.z;
                left &= ~__ballot_sync(kAll, mine);
            }
            CellRuns runs{};
            if (lane < 27u) runs = runs_at(c0, (int)lane, gg, fstart, bstart);
            const uint32_t total = place_runs(runs);
            const ListOut out{shape, nbr, row - row0, cap};
            const uint32_t found = cell_rows<MODE, R>(S, runs, total, mine, q, d2max, pos, orig, out);
            if (mine && lane < R) {
                ncnt[row - row0] = min(found, cap) + 1u;
                if (found > cap) {
                    atomicAdd(overflow_count, 1u);
                    atomicOr(status, ST_BOUNDS);
                }
            }
            __syncwarp();
        }
    }
    walk_rows<MODE>(
        S, __ballot_sync(kAll, walked && lane < SCAN), d2max, pos, orig,
        [&](uint32_t l) {
            WalkedRow r;
            r.i = __shfl_sync(kAll, i, (int)l);
            r.p = make_float4(__shfl_sync(kAll, p.x, (int)l), __shfl_sync(kAll, p.y, (int)l),
                              __shfl_sync(kAll, p.z, (int)l), 0.f);
            r.c = make_int3(__shfl_sync(kAll, own.x, (int)l), __shfl_sync(kAll, own.y, (int)l),
                            __shfl_sync(kAll, own.z, (int)l));
            r.g = load_scene(sc, r.i);
            r.fstart = fstart;
            r.bstart = bstart;
            r.out = ListOut{shape, nbr, r.i - row0, cap};
            return r;
        },
        [&](const WalkedRow &r, uint32_t found, bool lead) {
            if (!lead) return;
            ncnt[r.i - row0] = min(found, cap) + 1u;
            if (found > cap) {
                atomicAdd(overflow_count, 1u);
                atomicOr(status, ST_BOUNDS);
            }
        });
}

#ifdef VTP_CHECKED
// Checked build (-DVTP_CHECKED): every list entry of rows [row0, row0 + cnt)
// after each build - count <= maxNbr, entries inside the solver's rows, no
// row listed as its own neighbour - with the first offence recorded in
// `status` (ST_BOUNDS); the passes consume only validated lists.
__global__ void k_check_lists(uint32_t row0, uint32_t cnt, uint32_t nrows, ListShape shape, uint32_t maxnbr,
                              const uint32_t *__restrict__ nbr, const uint32_t *__restrict__ ncnt,
                              uint32_t *__restrict__ status) {
    const uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= cnt) return;
    const uint32_t n = ncnt[r];
    bool bad = n > maxnbr;
    for (uint32_t t = 0; !bad && t + 1 < n; ++t) {
        const uint32_t j = nbr[ell_index(r, t, shape)];
        bad = j >= nrows || j == row0 + r;
    }
    if (bad) atomicOr(status, ST_BOUNDS);
}
#endif

// Staged list builder: one block per brick (staged.h).  The block stages
// the brick's 6 x 6 x 6-cell neighbourhood - positions, with each row's index
// in w - in shared memory once, and every row of the group walks its 27 cells
// (the reference's offset order, a cell's runs in list order, cells beyond h
// culled) over the staged copy, writing the global list entry and the slot
// list entry of each accepted candidate.  A group whose neighbourhood exceeds
// the staging capacity walks global memory with the one-thread walker and
// writes no slot list (the solve passes then gather it from global memory);
// block `ngroups` gives the rows outside the grid empty lists.
template <int MODE, bool CULL>
__global__ void __launch_bounds__(kStageBlock) k_build_lists_staged(
    Scenes sc, Staging stg, ListShape shape, const float4 *__restrict__ pos, uint32_t *__restrict__ nbr,
    uint32_t *__restrict__ ncnt, uint32_t *__restrict__ status, uint32_t *__restrict__ overflow_count) {
    pdl_enter();
    extern __shared__ float4 stage[];
    __shared__ GroupPlan P;
    const uint32_t grp = blockIdx.x;
    const SceneGrid g = sc.sg[0];
    if (grp == stg.ngroups) {   // rows outside the grid: no neighbours, not even self
        const uint32_t k = g.key_base + g.nkey;
        const uint32_t r1 = __ldg(stg.fstart + k + 1);
        for (uint32_t r = __ldg(stg.fstart + k) + threadIdx.x; r < r1; r += blockDim.x) ncnt[r] = 0;
        return;
    }
    const uint2 rows = group_rows(grp, g, stg);
    if (rows.x == rows.y) return;
    plan_group(P, grp, g, stg);
    const bool staged = P.total <= stg.scap;
    if (staged) {
        for (uint32_t s = threadIdx.x; s < P.total; s += blockDim.x) {
            bool b;
            const uint32_t j = slot_row<MODE>(P, slot_cell(P, s), s, b);
            float4 q = __ldg(pos + j);
            q.w = __uint_as_float(j);
            stage[s] = q;
        }
    }
    __syncthreads();
    const float d2max = sc.d2max;
    const uint32_t maxnbr = sc.maxnbr;
    for (uint32_t r = P.r0 + threadIdx.x; r < P.r1; r += blockDim.x) {
        const float4 p = pos[r];
        const int3 c = cell_of(p.x, p.y, p.z, g, sc.cell);
        FaceGaps fg;
        if (CULL) fg.init(p, c, g, sc.cell);
        if (!staged) {
            Walker<RowSlots> w;
            w.px = p.x; w.py = p.y; w.pz = p.z;
            w.self = r;
            w.cnt = 1;
            w.maxnbr = maxnbr;
            w.out = nbr + row_index(r, shape);
            w.overflow = false;
            for (int t = 0; t < 27; ++t) {
                const int3 o = nbr_offset(t);
                const int3 cc = make_int3(c.x + o.x, c.y + o.y, c.z + o.z);
                if (!cell_available(cc, g)) continue;
                if (CULL && !fg.reachable(o, d2max)) continue;
                const uint32_t k = g.key_base + cell_key(cc, g);
                const uint32_t f0 = __ldg(stg.fstart + k), f1 = __ldg(stg.fstart + k + 1);
                const uint32_t b0 = __ldg(stg.bstart + k), b1 = __ldg(stg.bstart + k + 1);
                if (w.cnt + (f1 - f0) + (b1 - b0) <= w.maxnbr)
                    w.visit_cell<MODE, true>(f0, f1, b0, b1, pos, nullptr, d2max);
                else
                    w.visit_cell<MODE, false>(f0, f1, b0, b1, pos, nullptr, d2max);
            }
            ncnt[r] = w.cnt;
            if (w.overflow) {
                atomicAdd(overflow_count, 1u);
                atomicOr(status, ST_BOUNDS);
            }
            continue;
        }
        uint32_t *const out = nbr + row_index(r, shape);
        uint16_t *const sout = stg.snbr + row_index(r, shape);
        uint32_t cnt = 1;
        bool over = false;
        for (int t = 0; t < 27; ++t) {
            const int3 o = nbr_offset(t);
            const int3 cc = make_int3(c.x + o.x, c.y + o.y, c.z + o.z);
            if (!cell_available(cc, g)) continue;
            if (CULL && !fg.reachable(o, d2max)) continue;
            const int lx = cc.x - P.ox, ly = cc.y - P.oy, lz = cc.z - P.oz;
            if ((unsigned)lx >= (unsigned)kStageUx || (unsigned)ly >= (unsigned)kStageUy ||
                (unsigned)lz >= (unsigned)kStageUz) {   // a row outside its group's block: never expected
                atomicOr(status, ST_BOUNDS);
                continue;
            }
            const int u = (lz * kStageUy + ly) * kStageUx + lx;
            const uint32_t s0 = P.off[u], s1 = P.off[u + 1];
            // first boundary slot (mode 0) / first fluid slot (mode 1) of the cell
            const uint32_t sb = s0 + (MODE == 0 ? P.nfl[u] : P.nbl[u]);
            const bool room = cnt + (s1 - s0) <= maxnbr;
            for (uint32_t sl = s0; sl < s1; ++sl) {
                const float4 q = stage[sl];
                const float d2 = dist2(p.x - q.x, p.y - q.y, p.z - q.z);
                if (d2 > 0.f && d2 <= d2max) {
                    if (room || cnt < maxnbr) {
                        const bool bnd = MODE == 0 ? sl >= sb : sl < sb;
                        out[(size_t)(cnt - 1) * 32u] = __float_as_uint(q.w);
                        sout[(size_t)(cnt - 1) * 32u] = (uint16_t)(sl | (bnd ? kSlotBoundary : 0u));
                        ++cnt;
                    } else {
                        over = true;
                    }
                }
            }
        }
        ncnt[r] = cnt;
        if (over) {
            atomicAdd(overflow_count, 1u);
            atomicOr(status, ST_BOUNDS);
        }
    }
}

__global__ void k_scatter_f4(uint32_t n, const float4 *__restrict__ src, const uint32_t *__restrict__ orig,
                             float *__restrict__ dst3) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float4 v = src[i];
    size_t o = (size_t)orig[i] * 3;
    dst3[o] = v.x;
    dst3[o + 1] = v.y;
    dst3[o + 2] = v.z;
}

__global__ void k_scatter_f1(uint32_t n, const float *__restrict__ src, const uint32_t *__restrict__ orig,
                             float *__restrict__ dst) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    dst[orig[i]] = src[i];
}

__global__ void k_gather_f4(uint32_t n, const float *__restrict__ src3, const uint32_t *__restrict__ orig,
                            float4 *__restrict__ dst, int keep_w) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    size_t o = (size_t)orig[i] * 3;
    float4 v = dst[i];
    v.x = src3[o];
    v.y = src3[o + 1];
    v.z = src3[o + 2];
    if (!keep_w) v.w = 0.f;
    dst[i] = v;
}

__global__ void k_gather_f1(uint32_t n, const float *__restrict__ src, const uint32_t *__restrict__ orig,
                            float *__restrict__ dst) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    dst[i] = src[orig[i]];
}

// Rows whose attach id lies in [first, first + count): scatter to / gather from a
// compact buffer indexed by id - first.
__global__ void k_scatter_f4_range(uint32_t n, const float4 *__restrict__ src, const uint32_t *__restrict__ orig,
                                   uint32_t first, uint32_t count, float *__restrict__ dst3) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint32_t id = orig[i] - first;
    if (id >= count) return;
    const float4 v = src[i];
    dst3[3 * (size_t)id] = v.x;
    dst3[3 * (size_t)id + 1] = v.y;
    dst3[3 * (size_t)id + 2] = v.z;
}

__global__ void k_gather_f4_range(uint32_t n, const float *__restrict__ src3, const uint32_t *__restrict__ orig,
                                  uint32_t first, uint32_t count, float4 *__restrict__ dst,
                                  float4 *__restrict__ dst2) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint32_t id = orig[i] - first;
    if (id >= count) return;
    float4 v = dst[i];
    v.x = src3[3 * (size_t)id];
    v.y = src3[3 * (size_t)id + 1];
    v.z = src3[3 * (size_t)id + 2];
    dst[i] = v;
    if (dst2) {
        float4 w = dst2[i];
        w.x = v.x; w.y = v.y; w.z = v.z;
        dst2[i] = w;
    }
}

// Positions and velocities of one attach-id range together (one pass each way).
__global__ void k_scatter_state_range(uint32_t n, const float4 *__restrict__ pos, const float4 *__restrict__ vel,
                                      const uint32_t *__restrict__ orig, uint32_t first, uint32_t count,
                                      float *__restrict__ p3, float *__restrict__ v3) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint32_t id = orig[i] - first;
    if (id >= count) return;
    const float4 p = pos[i], v = vel[i];
    p3[3 * (size_t)id] = p.x;
    p3[3 * (size_t)id + 1] = p.y;
    p3[3 * (size_t)id + 2] = p.z;
    v3[3 * (size_t)id] = v.x;
    v3[3 * (size_t)id + 1] = v.y;
    v3[3 * (size_t)id + 2] = v.z;
}

__global__ void k_gather_state_range(uint32_t n, const float *__restrict__ p3, const float *__restrict__ v3,
                                     const uint32_t *__restrict__ orig, uint32_t first, uint32_t count,
                                     float4 *__restrict__ pos, float4 *__restrict__ vel, float4 *__restrict__ vadv) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint32_t id = orig[i] - first;
    if (id >= count) return;
    float4 p = pos[i], v = vel[i];
    p.x = p3[3 * (size_t)id]; p.y = p3[3 * (size_t)id + 1]; p.z = p3[3 * (size_t)id + 2];
    v.x = v3[3 * (size_t)id]; v.y = v3[3 * (size_t)id + 1]; v.z = v3[3 * (size_t)id + 2];
    pos[i] = p;
    vel[i] = v;
    if (vadv) {
        float4 w = vadv[i];
        w.x = v.x; w.y = v.y; w.z = v.z;
        vadv[i] = w;
    }
}

// Slot of attach id `id` in buffers that hold several particle ranges back to back:
// tab[3k], tab[3k + 1], tab[3k + 2] = first, count, first slot of range k, the ranges
// ascending and disjoint; ~0u outside every range.
__device__ __forceinline__ uint32_t range_slot(uint32_t id, const uint32_t *__restrict__ tab, uint32_t nr) {
    uint32_t lo = 0, hi = nr;   // the first range that starts after id
    while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        if (tab[3 * mid] <= id) lo = mid + 1;
        else hi = mid;
    }
    if (lo == 0) return ~0u;
    const uint32_t k = lo - 1, d = id - tab[3 * k];
    return d < tab[3 * k + 1] ? tab[3 * k + 2] + d : ~0u;
}

__global__ void k_scatter_state_ranges(uint32_t n, const float4 *__restrict__ pos, const float4 *__restrict__ vel,
                                       const uint32_t *__restrict__ orig, const uint32_t *__restrict__ tab,
                                       uint32_t nr, float *__restrict__ p3, float *__restrict__ v3) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint32_t id = range_slot(orig[i], tab, nr);
    if (id == ~0u) return;
    const float4 p = pos[i], v = vel[i];
    p3[3 * (size_t)id] = p.x;
    p3[3 * (size_t)id + 1] = p.y;
    p3[3 * (size_t)id + 2] = p.z;
    v3[3 * (size_t)id] = v.x;
    v3[3 * (size_t)id + 1] = v.y;
    v3[3 * (size_t)id + 2] = v.z;
}

__global__ void k_gather_state_ranges(uint32_t n, const float *__restrict__ p3, const float *__restrict__ v3,
                                      const uint32_t *__restrict__ orig, const uint32_t *__restrict__ tab,
                                      uint32_t nr, float4 *__restrict__ pos, float4 *__restrict__ vel,
                                      float4 *__restrict__ vadv) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint32_t id = range_slot(orig[i], tab, nr);
    if (id == ~0u) return;
    float4 p = pos[i], v = vel[i];
    p.x = p3[3 * (size_t)id]; p.y = p3[3 * (size_t)id + 1]; p.z = p3[3 * (size_t)id + 2];
    v.x = v3[3 * (size_t)id]; v.y = v3[3 * (size_t)id + 1]; v.z = v3[3 * (size_t)id + 2];
    pos[i] = p;
    vel[i] = v;
    if (vadv) {
        float4 w = vadv[i];
        w.x = v.x; w.y = v.y; w.z = v.z;
        vadv[i] = w;
    }
}

__global__ void k_iota(uint32_t n, uint32_t *dst, uint32_t base) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) dst[i] = base + i;
}

__global__ void k_export_neighbors(uint32_t row0, uint32_t cnt, ListShape shape,
                                   const uint32_t *__restrict__ nbr, const uint32_t *__restrict__ ncnt,
                                   const uint32_t *__restrict__ orig, uint32_t maxnbr,
                                   uint32_t *__restrict__ out_cnt, uint32_t *__restrict__ out_nbr) {
    uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= cnt) return;
    uint32_t i = row0 + r;
    uint32_t o = orig[i];
    uint32_t c = ncnt[r];
    out_cnt[o] = c;
    uint32_t *dst = out_nbr + (size_t)o * maxnbr;
    for (uint32_t t = 0; t < maxnbr; ++t) dst[t] = 0xffffffffu;
    if (c == 0) return;
    dst[0] = o;
    for (uint32_t t = 1; t < c; ++t) dst[t] = orig[nbr[ell_index(r, t - 1, shape)]];
}

__global__ void k_export_sorted(Scenes sc, uint32_t n, const float4 *__restrict__ pos,
                                const uint32_t *__restrict__ orig, uint32_t *__restrict__ ids,
                                uint32_t *__restrict__ keys) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const SceneGrid g = load_scene(sc, i);
    float4 p = pos[i];
    int3 c = cell_of(p.x, p.y, p.z, g, sc.cell);
    ids[i] = orig[i];
    keys[i] = cell_available(c, g) ? ref_cell_key(c, g) : 0xffffffffu;
}

inline unsigned nblk(uint32_t n, int b) { return (unsigned)((n + b - 1) / b); }

}  // namespace

__global__ void k_cubic_sigma(float h, float *out) {
    const float PI = 3.14159265f;
    if (threadIdx.x == 0) out[0] = 8.f / PI / powf(h, 3.f);
}

// cube_rn against powf(t, 3.f) for every t = k * 2^-24, k in [0, 2^23]:
// number of differing inputs and the largest distance in ulps (both are
// positive floats, so the distance is the difference of the bit patterns).
__global__ void k_selftest_cube(uint32_t *mismatches, uint32_t *max_ulp) {
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k > (1u << 23)) return;
    const float t = (float)k * 0x1p-24f;
    const int a = (int)__float_as_uint(cube_rn(t)), b = (int)__float_as_uint(powf(t, 3.f));
    if (a != b) {
        atomicAdd(mismatches, 1u);
        atomicMax(max_ulp, (uint32_t)(a > b ? a - b : b - a));
    }
}

int selftest_cube(cudaStream_t st, uint32_t *mismatches, uint32_t *max_ulp) {
    uint32_t *d = nullptr;
    if (cudaMalloc(&d, 2 * sizeof(uint32_t)) != cudaSuccess) return 1;
    uint32_t out[2] = {0u, 0u};
    cudaError_t e = cudaMemsetAsync(d, 0, 2 * sizeof(uint32_t), st);
    if (e == cudaSuccess) {
        k_selftest_cube<<<nblk((1u << 23) + 1u, 256), 256, 0, st>>>(d, d + 1);
        e = cudaMemcpyAsync(out, d, sizeof(out), cudaMemcpyDeviceToHost, st);
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    cudaFree(d);
    *mismatches = out[0];
    *max_ulp = out[1];
    return e == cudaSuccess ? 0 : 1;
}

int cubic_sigma_device(cudaStream_t st, float h, float *out_host) {
    float *d = nullptr;
    if (cudaMalloc(&d, sizeof(float)) != cudaSuccess) return 1;
    k_cubic_sigma<<<1, 32, 0, st>>>(h, d);
    cudaError_t e = cudaMemcpyAsync(out_host, d, sizeof(float), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    cudaFree(d);
    return e == cudaSuccess ? 0 : 1;
}

// Up to this many scan tiles (2,048 cells each) the hash counts the tiles' sums as well and each
// block of the scan adds up the sums before its own (at most 4 a thread): one launch in place of
// three, which for a small grid is most of the scan's time.  B200, event-timed, about 5 us of it
// the events: 2,000 rows 12.3 -> 8.4 us, 250,000 rows 12.6 -> 8.6, 1,000,000 rows 16.7 -> 8.7; the
// hash keeps its time (14.5 -> 15.3 at 1,000,000 rows).
constexpr size_t kPrefixTiles = 1024;

static void scan_counts(cudaStream_t st, uint32_t *count, size_t n, uint32_t base_add, uint32_t *out,
                        UgnsBuffers &u) {
    size_t tiles = (n + kScanTile - 1) / kScanTile;
    if (tiles <= kPrefixTiles) {
        launch(k_scan_tiles<true>, (unsigned)tiles, kScanThreads, 0, st, count, n, u.scan_sums, base_add, out);
        return;
    }
    launch(k_scan_tile_sums, (unsigned)tiles, kScanThreads, 0, st, count, n, u.scan_sums);
    launch(k_scan_sums, 1, 1024, 0, st, u.scan_sums, tiles);
    launch(k_scan_tiles<false>, (unsigned)tiles, kScanThreads, 0, st, count, n, u.scan_sums, base_add, out);
}

uint32_t ugns_sort_launches(uint32_t nbuckets) {   // hash, scan, scatter, rank / reorder
    return ((size_t)nbuckets + kScanTile - 1) / kScanTile <= kPrefixTiles ? 4u : 6u;
}

void ugns_sort(cudaStream_t st, const Scenes &sc, uint32_t nbuckets, uint32_t row0, uint32_t cnt,
               const float4 *pos_in, float4 *pos_out, const float4 *vel_in, float4 *vel_out,
               const uint32_t *orig_in, uint32_t *orig_out, const Carry &carry, float force_dt, UgnsBuffers &u,
               uint32_t *start, Profiler *prof) {
    const size_t nb = nbuckets;  // buckets incl. every scene's outside bucket
    auto B = [&] { if (prof) prof->begin(); };
    auto E = [&](const char *nm) { if (prof) prof->end_(nm); };
    B();
    // u.count is all zero here: zeroed once at allocation and by every scan after reading it; the
    // same holds for u.scan_sums (by the scatter) where the hash counts into it.
    const size_t tiles = (nb + kScanTile - 1) / kScanTile;
    uint32_t *const sums = tiles <= kPrefixTiles ? u.scan_sums : nullptr;
    if (cnt > 0) {
        launch(k_hash, nblk(cnt, 256), 256, 0, st, sc, row0, cnt, pos_in, vel_in, force_dt, u.key, u.rank, u.count,
               sums);
    }
    E("ugns_clear_hash");
    B();
    scan_counts(st, u.count, nb, row0, start, u);
    E("ugns_cell_scan");
    if (cnt == 0) return;
    B();
    launch(k_scatter, nblk(cnt, 256), 256, 0, st, row0, cnt, u.key, u.rank, start, orig_in, u.tmp_src, u.tmp_orig,
           u.tmp_key, u.status, sums, (uint32_t)tiles);
    E("ugns_scatter");
    B();
    launch(k_rank_reorder, nblk(cnt, 256), 256, 0, st, sc, row0, cnt, start, u.tmp_src, u.tmp_orig, u.tmp_key, pos_in,
                                                   pos_out, vel_in, vel_out, orig_out, carry, force_dt);
    E("ugns_rank_reorder");
}

void ugns_build_lists(cudaStream_t st, const Scenes &sc, const Layout &L, uint32_t row0, uint32_t cnt,
                      const float4 *pos, const uint32_t *orig, const UgnsBuffers &u, uint32_t *nbr, uint32_t *ncnt,
                      uint32_t *status, uint32_t *overflow) {
    if (cnt == 0) return;
    const uint32_t *start = row0 == L.nf ? u.bstart : u.fstart;   // the table of the rows themselves
    using M0 = std::integral_constant<int, 0>;
    using M1 = std::integral_constant<int, 1>;
    using M2 = std::integral_constant<int, 2>;
    // Lists of either builder are the same; a thread per row writes shape lg 0 well (its stores of
    // one entry index share a line), so it takes the large solvers, whose lists have that shape.
    if (L.list_lanes == 1 || (L.list_lanes == 0 && cnt > kScan8Rows && L.shape.lg == 0)) {
        auto walk_as = [&](auto mode, auto cull, auto slots) {
            constexpr int M = decltype(mode)::value;
            constexpr bool C = decltype(cull)::value;
            launch(k_walk_lists<M, C, decltype(slots)>, nblk(cnt, kWalkBlock), kWalkBlock, 0, st, sc, row0, cnt,
                   L.shape, pos, orig, u.fstart, u.bstart, nbr, ncnt, status, overflow);
        };
        auto walk = [&](auto mode, auto cull) {
            if (L.shape.lg == 0) walk_as(mode, cull, RowSlots{});
            else walk_as(mode, cull, AnySlots{});
        };
        const std::true_type T;
        const std::false_type F;
        switch (L.merge_mode) {
            case 0: L.cell_cull ? walk(M0{}, T) : walk(M0{}, F); break;
            case 1: L.cell_cull ? walk(M1{}, T) : walk(M1{}, F); break;
            default: L.cell_cull ? walk(M2{}, T) : walk(M2{}, F); break;
        }
    } else {
        auto cells = [&](auto mode, auto scan) {
            constexpr uint32_t SCAN = decltype(scan)::value;
            launch(k_build_lists<decltype(mode)::value, SCAN>, nblk(cnt, kCellWarps * SCAN), kCellWarps * 32, 0, st, sc,
                   row0, cnt, L.shape, pos, orig, start, u.fstart, u.bstart, nbr, ncnt, status, overflow);
        };
        auto build = [&](auto mode) {
            if (cnt <= kScan4Rows) cells(mode, std::integral_constant<uint32_t, 4>{});
            else cells(mode, std::integral_constant<uint32_t, 8>{});
        };
        switch (L.merge_mode) {
            case 0: build(M0{}); break;
            case 1: build(M1{}); break;
            default: build(M2{}); break;
        }
    }
#ifdef VTP_CHECKED
    k_check_lists<<<nblk(cnt, 256), 256, 0, st>>>(row0, cnt, L.n, L.shape, sc.maxnbr, nbr, ncnt, status);
#endif
}

void ugns_build_lists_staged(cudaStream_t st, const Scenes &sc, const Layout &L, const Staging &stg,
                             const float4 *pos, uint32_t *nbr, uint32_t *ncnt, uint32_t *status,
                             uint32_t *overflow) {
    const size_t smem = (size_t)stg.scap * sizeof(float4);
    const unsigned grid = stg.ngroups + 1;
    // the staged rows may exceed the 48 KB of dynamic shared memory a kernel gets by default
    auto room = [&](auto kern) { cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); };
    if (stg.mode == 0 && L.cell_cull) {
        room(k_build_lists_staged<0, true>);
        launch(k_build_lists_staged<0, true>, grid, kStageBlock, smem, st, sc, stg, L.shape, pos, nbr, ncnt,
               status, overflow);
    } else if (stg.mode == 0) {
        room(k_build_lists_staged<0, false>);
        launch(k_build_lists_staged<0, false>, grid, kStageBlock, smem, st, sc, stg, L.shape, pos, nbr, ncnt,
               status, overflow);
    } else if (L.cell_cull) {
        room(k_build_lists_staged<1, true>);
        launch(k_build_lists_staged<1, true>, grid, kStageBlock, smem, st, sc, stg, L.shape, pos, nbr, ncnt,
               status, overflow);
    } else {
        room(k_build_lists_staged<1, false>);
        launch(k_build_lists_staged<1, false>, grid, kStageBlock, smem, st, sc, stg, L.shape, pos, nbr, ncnt,
               status, overflow);
    }
#ifdef VTP_CHECKED
    k_check_lists<<<nblk(L.nf, 256), 256, 0, st>>>(0, L.nf, L.n, L.shape, sc.maxnbr, nbr, ncnt, status);
#endif
}

void scatter_f4_to_orig(cudaStream_t st, uint32_t n, const float4 *src, const uint32_t *orig, float *dst3) {
    if (n) k_scatter_f4<<<nblk(n, 256), 256, 0, st>>>(n, src, orig, dst3);
}
void scatter_f1_to_orig(cudaStream_t st, uint32_t n, const float *src, const uint32_t *orig, float *dst) {
    if (n) k_scatter_f1<<<nblk(n, 256), 256, 0, st>>>(n, src, orig, dst);
}
void gather_orig_to_f4(cudaStream_t st, uint32_t n, const float *src3, const uint32_t *orig, float4 *dst,
                       int keep_w) {
    if (n) k_gather_f4<<<nblk(n, 256), 256, 0, st>>>(n, src3, orig, dst, keep_w);
}
void gather_orig_to_f1(cudaStream_t st, uint32_t n, const float *src, const uint32_t *orig, float *dst) {
    if (n) k_gather_f1<<<nblk(n, 256), 256, 0, st>>>(n, src, orig, dst);
}
void scatter_f4_range(cudaStream_t st, uint32_t n, const float4 *src, const uint32_t *orig, uint32_t first,
                      uint32_t count, float *dst3) {
    if (n) k_scatter_f4_range<<<nblk(n, 256), 256, 0, st>>>(n, src, orig, first, count, dst3);
}
void gather_f4_range(cudaStream_t st, uint32_t n, const float *src3, const uint32_t *orig, uint32_t first,
                     uint32_t count, float4 *dst, float4 *dst2) {
    if (n) k_gather_f4_range<<<nblk(n, 256), 256, 0, st>>>(n, src3, orig, first, count, dst, dst2);
}
void scatter_state_range(cudaStream_t st, uint32_t n, const float4 *pos, const float4 *vel, const uint32_t *orig,
                         uint32_t first, uint32_t count, float *p3, float *v3) {
    if (n) k_scatter_state_range<<<nblk(n, 256), 256, 0, st>>>(n, pos, vel, orig, first, count, p3, v3);
}
void gather_state_range(cudaStream_t st, uint32_t n, const float *p3, const float *v3, const uint32_t *orig,
                        uint32_t first, uint32_t count, float4 *pos, float4 *vel, float4 *vadv) {
    if (n) k_gather_state_range<<<nblk(n, 256), 256, 0, st>>>(n, p3, v3, orig, first, count, pos, vel, vadv);
}
void scatter_state_ranges(cudaStream_t st, uint32_t n, const float4 *pos, const float4 *vel, const uint32_t *orig,
                          const uint32_t *tab, uint32_t nr, float *p3, float *v3) {
    if (n) k_scatter_state_ranges<<<nblk(n, 256), 256, 0, st>>>(n, pos, vel, orig, tab, nr, p3, v3);
}
void gather_state_ranges(cudaStream_t st, uint32_t n, const float *p3, const float *v3, const uint32_t *orig,
                         const uint32_t *tab, uint32_t nr, float4 *pos, float4 *vel, float4 *vadv) {
    if (n) k_gather_state_ranges<<<nblk(n, 256), 256, 0, st>>>(n, p3, v3, orig, tab, nr, pos, vel, vadv);
}
void fill_iota(cudaStream_t st, uint32_t n, uint32_t *dst, uint32_t base) {
    if (n) k_iota<<<nblk(n, 256), 256, 0, st>>>(n, dst, base);
}
void export_neighbors(cudaStream_t st, const Layout &L, uint32_t row0, uint32_t cnt, const uint32_t *nbr,
                      const uint32_t *ncnt, const uint32_t *orig, uint32_t maxnbr, uint32_t *out_cnt,
                      uint32_t *out_nbr) {
    if (cnt)
        k_export_neighbors<<<nblk(cnt, 256), 256, 0, st>>>(row0, cnt, L.shape, nbr, ncnt, orig, maxnbr, out_cnt,
                                                           out_nbr);
}
void export_sorted(cudaStream_t st, const Scenes &sc, uint32_t n, const float4 *pos, const uint32_t *orig,
                   uint32_t *out_ids, uint32_t *out_keys) {
    if (n) k_export_sorted<<<nblk(n, 256), 256, 0, st>>>(sc, n, pos, orig, out_ids, out_keys);
}

}  // namespace vtp
