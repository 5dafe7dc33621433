// Internal host-side interfaces between the solver driver (capi.cu) and the
// kernel translation units (ugns.cu, pbf.cu, dfsph.cu, immct.cu).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "common.cuh"

#include <nvtx3/nvToolsExt.h>

namespace vtp {

// NVTX range over a host scope (solver stages: initialize, tick, the substep's
// enqueue stages, differentiation, export).  NVTX is header-only and does
// nothing unless a profiler is attached.  With graphs the enqueue stages are
// recorded once, at capture; every tick shows as one range around its graph
// launches.
struct NvtxRange {
    explicit NvtxRange(const char *name) { nvtxRangePushA(name); }
    ~NvtxRange() { nvtxRangePop(); }
    NvtxRange(const NvtxRange &) = delete;
    NvtxRange &operator=(const NvtxRange &) = delete;
};

// Solvers of up to this many fluid rows walk a row with a team of lanes (team.cuh), larger
// ones with a thread per row; the bits are the same.  Event-timed launches (B200, about 5 us of
// which is the events), thread per row -> team of four, us: DFSPH solve_a / solve_b / ratio + alpha /
// viscosity at 2,000 rows 13.3 / 11.6 / 16.4 / 13.4 -> 9.9 / 8.5 / 9.4 / 10.4, at 32,000 rows
// 14.5 / 12.6 / 18.7 / 14.8 -> 13.2 / 10.6 / 13.1 / 12.4, at 64,000 rows 16.4 / 14.4 / 18.8 / 16.6
// -> 18.3 / 15.1 / 20.8 / 19.0; PBF lambda / dx / XSPH at 2,000 rows 16.9 / 12.4 / 14.6 -> 10.5 /
// 10.3 / 10.6, at 32,000 rows 18.7 / 12.6 / 16.7 -> 14.7 / 12.6 / 12.6, at 64,000 rows 20.8 / 14.7
// / 18.8 -> 20.7 / 16.7 / 18.8.  A team executes 1.6 times the instructions of the thread, so past
// the row count that fills the GPU the thread wins (1,000,000 rows: solve_a 113 -> 168).
constexpr uint32_t kTeamMaxRows = 49152;
// Of them, up to this many rows take eight lanes, so that a row of 32 neighbours is one batch.  Four ->
// eight lanes, us: PBF lambda / dx / XSPH at 2,000 rows 10.6 / 10.3 / 8.5 -> 8.4 / 8.4 / 8.4, at
// 16,000 rows 12.3 / 10.5 / 10.6 -> 10.6 / 10.5 / 10.5, at 32,000 rows 14.6 / 12.6 / 12.6 -> 14.6 /
// 14.2 / 14.6; DFSPH solve_a / ratio + alpha at 2,000 rows 9.9 / 10.5 -> 9.4 / 8.5, at 16,000 rows
// 11.4 / 12.5 -> 11.8 / 10.6, at 32,000 rows 13.4 / 14.7 -> 15.0 / 14.6.
constexpr uint32_t kTeam8MaxRows = 16384;

constexpr int kConsPhases = 8;   // phases the conservation sums report (vtp_conservation.phase_mass)

// Particles are kept sorted: fluid rows [0, nf) re-sorted by (cell, attach id)
// every substep, boundary rows [nf, n) sorted once at initialize.
struct Layout {
    uint32_t n = 0, nf = 0, nb = 0;
    ListShape shape;           // neighbour-list storage (maxnbr - 1 entries per row)
    int merge_mode = 0;        // 0: fluid ids < boundary ids, 1: boundary ids < fluid ids, 2: general
    int list_lanes = 0;        // list builder: 0 by row count, 1 a thread per row, 8 groups of rows (same lists)
    bool cell_cull = false;    // the builders with a thread per row skip neighbour cells beyond h of the row (same lists)
};

// Neighbour-search working set (one per solver).
struct UgnsBuffers {
    uint32_t *key = nullptr;       // [nf] cell key per old slot
    uint32_t *rank = nullptr;      // [nf] arrival rank within the cell (atomic)
    uint32_t *count = nullptr;     // [nbuckets] (all scenes' buckets incl. their outside buckets)
    uint32_t *fstart = nullptr;    // [nbuckets + 1] fluid cell starts (absolute rows)
    uint32_t *bstart = nullptr;    // [nbuckets + 1] boundary cell starts (absolute rows)
    uint32_t *tmp_src = nullptr;   // [max(nf, nb)] scattered: old slot
    uint32_t *tmp_orig = nullptr;  // [max(nf, nb)] scattered: attach id
    uint32_t *tmp_key = nullptr;   // [max(nf, nb)] scattered: key
    uint32_t *scan_sums = nullptr; // [tiles] zero between sorts where the hash counts into it
    uint32_t *nbr = nullptr;       // ELL list for fluid rows
    uint32_t *ncnt = nullptr;      // [nf] neighbour count incl. self (0 = outside the grid)
    uint32_t *bnbr = nullptr;      // ELL list for boundary rows (init / diagnostics)
    uint32_t *bncnt = nullptr;     // [nb]
    uint32_t *status = nullptr;    // the solver's device status word (checked-build guards report here)
    size_t scan_tiles = 0;
};

// Fields a reorder carries from old slot to new slot (float4 / float / uint).
struct Carry {
    static constexpr int kMaxF4 = 8, kMaxF1 = 16;
    int nf4 = 0, nf1 = 0;
    const float4 *src4[kMaxF4];
    float4 *dst4[kMaxF4];
    const float *src1[kMaxF1];
    float *dst1[kMaxF1];
};

// Optional per-kernel timing: CUDA events recorded around each launch.
struct Profiler {
    static constexpr int kMax = 4096;
    cudaStream_t st = nullptr;
    int n = 0;
    const char *names[kMax];
    cudaEvent_t beg[kMax], end[kMax];
    bool ready = false;
    void begin() {
        if (!ready || n >= kMax) return;
        cudaEventRecord(beg[n], st);
    }
    void end_(const char *name) {
        if (!ready || n >= kMax) return;
        cudaEventRecord(end[n], st);
        names[n++] = name;
    }
};

// --- ugns.cu ---
// Sort rows [row0, row0 + cnt) by (scene, cell, attach id) into the output
// arrays; `start` receives the cell-start table (absolute rows) over all
// `nbuckets` buckets.  With `force_dt` > 0 the rows' positions get
// v += g dt; x += v dt applied first with their scene's gravity (PBF external
// force fused into the sort).
void ugns_sort(cudaStream_t st, const Scenes &sc, uint32_t nbuckets, uint32_t row0, uint32_t cnt,
               const float4 *pos_in, float4 *pos_out, const float4 *vel_in, float4 *vel_out,
               const uint32_t *orig_in, uint32_t *orig_out, const Carry &carry,
               float force_dt, UgnsBuffers &u, uint32_t *start, Profiler *prof = nullptr);

// Kernels a sort over `nbuckets` buckets launches.
uint32_t ugns_sort_launches(uint32_t nbuckets);

// Build the neighbour lists of rows [row0, row0 + cnt) (reference order:
// 27 offsets, then ascending attach id inside a cell).
void ugns_build_lists(cudaStream_t st, const Scenes &sc, const Layout &L, uint32_t row0, uint32_t cnt,
                      const float4 *pos, const uint32_t *orig, const UgnsBuffers &u,
                      uint32_t *nbr, uint32_t *ncnt, uint32_t *status, uint32_t *overflow);

// sigma of the cubic spline computed on the device (0 on success).
int cubic_sigma_device(cudaStream_t st, float h, float *out_host);
// cube_rn(t) vs powf(t, 3.f) over the outer-branch domain of cubic_w (0 on success).
int selftest_cube(cudaStream_t st, uint32_t *mismatches, uint32_t *max_ulp);

// Gather/scatter between attach order and sorted rows.
void scatter_f4_to_orig(cudaStream_t st, uint32_t n, const float4 *src, const uint32_t *orig, float *dst3);
void scatter_f1_to_orig(cudaStream_t st, uint32_t n, const float *src, const uint32_t *orig, float *dst);
void gather_orig_to_f4(cudaStream_t st, uint32_t n, const float *src3, const uint32_t *orig, float4 *dst,
                       int keep_w);
void gather_orig_to_f1(cudaStream_t st, uint32_t n, const float *src, const uint32_t *orig, float *dst);
void fill_iota(cudaStream_t st, uint32_t n, uint32_t *dst, uint32_t base);
// Attach-id range [first, first + count) <-> sorted rows [0, n) (float3 compact buffer).
void scatter_f4_range(cudaStream_t st, uint32_t n, const float4 *src, const uint32_t *orig, uint32_t first,
                      uint32_t count, float *dst3);
void gather_f4_range(cudaStream_t st, uint32_t n, const float *src3, const uint32_t *orig, uint32_t first,
                     uint32_t count, float4 *dst, float4 *dst2);
void scatter_state_range(cudaStream_t st, uint32_t n, const float4 *pos, const float4 *vel, const uint32_t *orig,
                         uint32_t first, uint32_t count, float *p3, float *v3);
void gather_state_range(cudaStream_t st, uint32_t n, const float *p3, const float *v3, const uint32_t *orig,
                        uint32_t first, uint32_t count, float4 *pos, float4 *vel, float4 *vadv);
// The same for several attach-id ranges held back to back in p3 / v3: tab (device) holds
// {first, count, first slot} per range, ascending and disjoint.
void scatter_state_ranges(cudaStream_t st, uint32_t n, const float4 *pos, const float4 *vel, const uint32_t *orig,
                          const uint32_t *tab, uint32_t nr, float *p3, float *v3);
void gather_state_ranges(cudaStream_t st, uint32_t n, const float *p3, const float *v3, const uint32_t *orig,
                         const uint32_t *tab, uint32_t nr, float4 *pos, float4 *vel, float4 *vadv);
void export_neighbors(cudaStream_t st, const Layout &L, uint32_t row0, uint32_t cnt, const uint32_t *nbr,
                      const uint32_t *ncnt, const uint32_t *orig, uint32_t maxnbr, uint32_t *out_cnt,
                      uint32_t *out_nbr);
void export_sorted(cudaStream_t st, const Scenes &sc, uint32_t n, const float4 *pos, const uint32_t *orig,
                   uint32_t *out_ids, uint32_t *out_keys);

}  // namespace vtp
