// Allocation-free neighbour search: the uniform-grid neighbour search of the
// library as one call that allocates nothing.
//
// Some callers cannot call cudaMalloc at the moment they need neighbour lists:
// hosts that hand the GPU to this library under a fixed memory budget with
// their own pool allocator, and real-time loops that forbid allocation after
// start-up (cudaMalloc may synchronise the device and can fail under
// fragmentation in the middle of a frame).  They pass device buffers for
// the input positions and the output lists; everything else the search needs
// lives in the fixed scratch arena below, which every GPU that loads this
// library holds until the process exits.
//
// The arena is shared by every call on a device: two calls whose work
// overlaps on the GPU (different streams, or different host threads without
// ordering) corrupt each other's scratch.  Calls are ordered on one stream.
#include <cmath>
#include <cstring>
#include <string>

#include "../../include/vtp.h"
#include "cells.cuh"
#include "common.cuh"

namespace vtp {
int fail(int code, const std::string &msg);
}

namespace {

constexpr uint32_t kMaxParticles = VTP_NOALLOC_MAX_PARTICLES;
constexpr uint32_t kMaxKeys = VTP_NOALLOC_MAX_CELLS;   // cell buckets incl. the outside bucket
constexpr int kScanThreads = 256;
constexpr int kScanItems = 8;
constexpr uint32_t kScanTile = kScanThreads * kScanItems;
constexpr uint32_t kMaxTiles = (kMaxKeys + 1 + kScanTile - 1) / kScanTile;

constexpr size_t align256(size_t b) { return (b + 255) / 256 * 256; }

// Arena layout (byte offsets).
constexpr size_t kOffKey = 0;
constexpr size_t kOffRank = kOffKey + align256(4ull * kMaxParticles);
constexpr size_t kOffTmp = kOffRank + align256(4ull * kMaxParticles);
constexpr size_t kOffPos = kOffTmp + align256(4ull * kMaxParticles);
constexpr size_t kOffCount = kOffPos + align256(16ull * kMaxParticles);
constexpr size_t kOffStart = kOffCount + align256(4ull * (kMaxKeys + 1));
constexpr size_t kOffTiles = kOffStart + align256(4ull * (kMaxKeys + 2));
constexpr size_t kArenaBytes = kOffTiles + align256(4ull * kMaxTiles);

static_assert(kArenaBytes == VTP_NOALLOC_SCRATCH_BYTES, "scratch size in vtp.h out of date");

__device__ __align__(256) unsigned char g_noalloc_scratch[kArenaBytes];

struct Arena {
    uint32_t *key, *rank, *tmp, *count, *start, *tiles;
    float4 *pos;
};

Arena arena_at(unsigned char *base) {
    Arena a;
    a.key = (uint32_t *)(base + kOffKey);
    a.rank = (uint32_t *)(base + kOffRank);
    a.tmp = (uint32_t *)(base + kOffTmp);
    a.pos = (float4 *)(base + kOffPos);
    a.count = (uint32_t *)(base + kOffCount);
    a.start = (uint32_t *)(base + kOffStart);
    a.tiles = (uint32_t *)(base + kOffTiles);
    return a;
}

// Device address of the arena on the current device.  In host code the
// symbol is a host-side stand-in, not a device address, so the address comes
// from cudaGetSymbolAddress.  It is looked up on every call rather than
// cached: after cudaDeviceReset (or in a new context on the same device) the
// module is loaded again and the array can sit at another address, and a
// cached pointer would then send the kernels into freed memory.  The lookup
// allocates nothing; only the first one in a context loads the module.
int arena_base(unsigned char **out) {
    void *p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess)
        return vtp::fail(VTP_ERR_CUDA, std::string("cudaGetSymbolAddress(scratch): ") + cudaGetErrorString(e));
    *out = (unsigned char *)p;
    return VTP_OK;
}

__global__ void k_na_hash(vtp::Grid g, uint32_t n, const float *__restrict__ pos, Arena a) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float x = pos[3 * (size_t)i], y = pos[3 * (size_t)i + 1], z = pos[3 * (size_t)i + 2];
    const int3 c = vtp::cell_of(x, y, z, g);
    const uint32_t k = vtp::cell_available(c, g) ? vtp::cell_key(c, g) : g.nkey;
    a.key[i] = k;
    a.rank[i] = atomicAdd(&a.count[k], 1u);
}

__device__ __forceinline__ uint32_t na_block_scan(uint32_t v, uint32_t &total) {
    __shared__ uint32_t ws[32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) ws[wid] = x;
    __syncthreads();
    if (wid == 0) {
        uint32_t s = lane < nw ? ws[lane] : 0u;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, s, o);
            if (lane >= o) s += y;
        }
        if (lane < nw) ws[lane] = s;
    }
    __syncthreads();
    const uint32_t off = wid > 0 ? ws[wid - 1] : 0u;
    total = ws[nw - 1];
    __syncthreads();
    return off + x - v;
}

__global__ void __launch_bounds__(kScanThreads) k_na_tile_sums(uint32_t nb, Arena a) {
    const size_t base = (size_t)blockIdx.x * kScanTile + threadIdx.x;
    uint32_t s = 0;
    for (int k = 0; k < kScanItems; ++k) {
        const size_t idx = base + (size_t)k * kScanThreads;
        if (idx < nb) s += a.count[idx];
    }
    uint32_t total;
    na_block_scan(s, total);
    if (threadIdx.x == 0) a.tiles[blockIdx.x] = total;
}

__global__ void __launch_bounds__(1024) k_na_scan_tiles(uint32_t tiles, Arena a) {
    const uint32_t per = (tiles + blockDim.x - 1) / blockDim.x;
    const uint32_t b = threadIdx.x * per;
    uint32_t local = 0;
    for (uint32_t k = 0; k < per; ++k)
        if (b + k < tiles) local += a.tiles[b + k];
    uint32_t total;
    uint32_t off = na_block_scan(local, total);
    for (uint32_t k = 0; k < per; ++k)
        if (b + k < tiles) {
            const uint32_t v = a.tiles[b + k];
            a.tiles[b + k] = off;
            off += v;
        }
}

__global__ void __launch_bounds__(kScanThreads) k_na_scan(uint32_t nb, Arena a) {
    __shared__ uint32_t tile[kScanTile];
    const size_t t0 = (size_t)blockIdx.x * kScanTile;
    for (int k = 0; k < kScanItems; ++k) {
        const size_t idx = t0 + (size_t)k * kScanThreads + threadIdx.x;
        tile[k * kScanThreads + threadIdx.x] = idx < nb ? a.count[idx] : 0u;
    }
    __syncthreads();
    uint32_t v[kScanItems], s = 0;
    for (int k = 0; k < kScanItems; ++k) {
        v[k] = tile[threadIdx.x * kScanItems + k];
        s += v[k];
    }
    uint32_t total;
    uint32_t off = na_block_scan(s, total) + a.tiles[blockIdx.x];
    for (int k = 0; k < kScanItems; ++k) {
        if (t0 + (size_t)threadIdx.x * kScanItems + k + 1 == nb) a.start[nb] = off + v[k];   // the grand total
        tile[threadIdx.x * kScanItems + k] = off;
        off += v[k];
    }
    __syncthreads();
    for (int k = 0; k < kScanItems; ++k) {
        const size_t idx = t0 + (size_t)k * kScanThreads + threadIdx.x;
        if (idx < nb) a.start[idx] = tile[k * kScanThreads + threadIdx.x];
    }
}

__global__ void k_na_scatter(uint32_t n, Arena a) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    a.tmp[a.start[a.key[i]] + a.rank[i]] = i;
}

// Stable (cell, id) order: rank inside the cell segment by particle id.
__global__ void k_na_rank(vtp::Grid g, uint32_t n, const float *__restrict__ pos, Arena a) {
    const uint32_t d = blockIdx.x * blockDim.x + threadIdx.x;
    if (d >= n) return;
    const uint32_t me = a.tmp[d];
    const uint32_t k = a.key[me];
    uint32_t dst = d;
    if (k < g.nkey) {
        const uint32_t s0 = a.start[k], s1 = a.start[k + 1];
        uint32_t r = 0;
        for (uint32_t x = s0; x < s1; ++x) r += a.tmp[x] < me ? 1u : 0u;
        dst = s0 + r;
    }
    a.pos[dst] = make_float4(pos[3 * (size_t)me], pos[3 * (size_t)me + 1], pos[3 * (size_t)me + 2],
                             __uint_as_float(me));
}

// Where the entries of a particle's list go: its row of the caller's array, after the particle itself.
struct ArrayOut {
    static constexpr bool kIds = true;   // entries are particle ids
    uint32_t *nbrs;
    uint32_t id, stride;                 // of this lane's particle; entries of a row of the array
    __device__ __forceinline__ bool eights() const { return true; }
    __device__ __forceinline__ uint32_t *mine() const { return nbrs + (size_t)id * stride + 1u; }
    __device__ __forceinline__ uint32_t *of(uint32_t lane) const {
        return nbrs + (size_t)__shfl_sync(0xffffffffu, id, (int)lane) * stride + 1u;
    }
    __device__ __forceinline__ void put(uint32_t *dst, uint32_t slot, uint32_t j) const {
        if (slot + 1u < stride) dst[slot] = j;
    }
};

// What a list has beside its entries: the particle itself, the count and the unused slots.  One lane
// per list has `lead` set, with the list's `found` and `out`.
__device__ __forceinline__ void finish_lists(uint32_t found, bool lead, const ArrayOut &out,
                                             uint32_t *__restrict__ counts) {
    constexpr unsigned kAll = 0xffffffffu;
    const uint32_t lane = threadIdx.x & 31u, n = min(found + 1u, out.stride);
    if (lead) {
        out.nbrs[(size_t)out.id * out.stride] = out.id;
        counts[out.id] = n;
    }
    unsigned todo = __ballot_sync(kAll, lead);
    while (todo) {   // eight lanes a list, four lists at a time
        uint32_t src = 32u;
#pragma unroll
        for (uint32_t q = 0; q < 4u; ++q) {
            if (todo && (lane >> 3) == q) src = (uint32_t)__ffs((int)todo) - 1u;
            todo &= todo - 1u;
        }
        const uint32_t nk = __shfl_sync(kAll, n, (int)(src & 31u)), id = __shfl_sync(kAll, out.id, (int)(src & 31u));
        if (src < 32u)
            for (uint32_t e = nk + (lane & 7u); e < out.stride; e += 8u) out.nbrs[(size_t)id * out.stride + e] = 0xffffffffu;
    }
}

// The run of the neighbour cell at offset t of cell c.
__device__ __forceinline__ vtp::CellRuns runs_at(int3 c, int t, const vtp::Grid &g, const uint32_t *start) {
    vtp::CellRuns r{};
    const int3 o = vtp::nbr_offset(t);
    const int3 cc = make_int3(c.x + o.x, c.y + o.y, c.z + o.z);
    if (vtp::cell_available(cc, g)) {
        const uint32_t b = vtp::cell_key(cc, g);
        r.f0 = start[b];
        r.f1 = start[b + 1];
    }
    return r;
}

// A particle for walk_rows.
struct WalkedParticle {
    float4 p;
    int3 c;
    const vtp::Grid *g;
    const uint32_t *start;
    ArrayOut out;
    __device__ __forceinline__ vtp::CellRuns runs(int t) const { return runs_at(c, t, *g, start); }
};

// Lists in the reference layout: self first, then the 27 cells in the reference's offset order,
// particles of a cell by ascending id.  As k_build_lists (ugns.cu): a warp takes SCAN sorted particles,
// builds the groups of one cell that start among them together, and walks the cells of the others.
// Whole call (B200, us), a thread per particle -> a warp per cell -> this: 400,000 particles half a
// cell apart 279 -> 216 -> 206, one cell apart 209 -> 326 -> 139, 0.35 cells apart 414 -> 499 -> 359;
// 20,000 half a cell apart 107 -> 64 -> 64, with 10,000 of them in one cell 2,156 -> 27,800 -> 510.
// At 400,000 particles 48 % of the issue slots and 66 % of the L1 rate at 36 % of the warp slots.
template <uint32_t SCAN>
__global__ void __launch_bounds__(vtp::kCellWarps * 32, 7) k_na_walk(vtp::Grid g, uint32_t n, Arena a,
                                                                     uint32_t *__restrict__ counts,
                                                                     uint32_t *__restrict__ nbrs) {
    __shared__ __align__(16) vtp::CellScratch scratch[vtp::kCellWarps];
    constexpr unsigned kAll = 0xffffffffu;
    constexpr uint32_t R = 8;
    const uint32_t lane = threadIdx.x & 31u, k = lane % SCAN;
    const uint32_t first = (blockIdx.x * vtp::kCellWarps + (threadIdx.x >> 5)) * SCAN;
    if (first >= n) return;
    vtp::CellScratch &S = scratch[threadIdx.x >> 5];
    const uint32_t m0 = min(SCAN, n - first), i = first + min(k, m0 - 1u);
    const float4 p = a.pos[i];
    const int3 own = vtp::cell_of(p.x, p.y, p.z, g);
    const bool inside = vtp::cell_available(own, g);
    uint32_t rows = 0;   // of the group that starts at particle i
    bool alone = false;   // its list is not built with a group
    if (inside) {
        const uint32_t b = vtp::cell_key(own, g), s = a.start[b], e = a.start[b + 1];
        const uint32_t in_group = (i - s) % R, m = min(R, e - (i - in_group));
        bool together = m >= vtp::kGroupMin || e - s > vtp::kCrowded;
        if (SCAN == 32u) together = together && e - s <= vtp::kSharedRows;
        if (together && in_group == 0u && lane < m0) rows = m;
        alone = !together;
    }
    for (unsigned todo = __ballot_sync(kAll, rows != 0u); todo; todo &= todo - 1u) {
        const int leader = __ffs((int)todo) - 1;
        const uint32_t m = __shfl_sync(kAll, rows, leader), beg = __shfl_sync(kAll, i, leader), kr = lane % R;
        const float4 q = a.pos[beg + min(kr, m - 1u)];
        const int3 c = vtp::cell_of(q.x, q.y, q.z, g);
        // A cell on the grid's inclusive upper face shares its bucket with another cell: one round
        // per cell among these particles.
        for (unsigned left = (1u << m) - 1u; left;) {
            const int f = __ffs((int)left) - 1;
            const int3 c0 = make_int3(__shfl_sync(kAll, c.x, f), __shfl_sync(kAll, c.y, f), __shfl_sync(kAll, c.z, f));
            const bool mine = ((left >> kr) & 1u) && c.x == c0.x && c.y == c0.y && c.z == c0.z;
            left &= ~__ballot_sync(kAll, mine);
            vtp::CellRuns runs{};
            if (lane < 27u) runs = runs_at(c0, (int)lane, g, a.start);
            const uint32_t total = vtp::place_runs(runs);
            const ArrayOut out{nbrs, __float_as_uint(q.w), g.maxnbr};
            const uint32_t found = vtp::cell_rows<0, R>(S, runs, total, mine, q, g.d2max, a.pos, nullptr, out);
            finish_lists(found, mine && lane < R, out, counts);
            __syncwarp();
        }
    }
    // Outside the grid: an empty list.
    for (unsigned todo = __ballot_sync(kAll, lane < m0 && !inside); todo; todo &= todo - 1u) {
        const uint32_t id = __float_as_uint(__shfl_sync(kAll, p.w, __ffs((int)todo) - 1));
        if (lane == 0) counts[id] = 0;
        for (uint32_t e = lane; e < g.maxnbr; e += 32u) nbrs[(size_t)id * g.maxnbr + e] = 0xffffffffu;
    }
    vtp::walk_rows<0>(
        S, __ballot_sync(kAll, alone && lane < m0), g.d2max, a.pos, nullptr,
        [&](uint32_t l) {
            WalkedParticle r;
            r.p = make_float4(__shfl_sync(kAll, p.x, (int)l), __shfl_sync(kAll, p.y, (int)l),
                              __shfl_sync(kAll, p.z, (int)l), __shfl_sync(kAll, p.w, (int)l));
            r.c = make_int3(__shfl_sync(kAll, own.x, (int)l), __shfl_sync(kAll, own.y, (int)l),
                            __shfl_sync(kAll, own.z, (int)l));
            r.g = &g;
            r.start = a.start;
            r.out = ArrayOut{nbrs, __float_as_uint(r.p.w), g.maxnbr};
            return r;
        },
        [&](const WalkedParticle &r, uint32_t found, bool lead) { finish_lists(found, lead, r.out, counts); });
}

inline unsigned nblk(uint32_t n, int b) { return (unsigned)((n + b - 1) / b); }

float sqrt_limit(float h) {
    float t = h * h;
    while (std::sqrt(t) > h) t = std::nextafter(t, 0.f);
    for (;;) {
        const float u = std::nextafter(t, INFINITY);
        if (std::sqrt(u) <= h) t = u;
        else break;
    }
    return t;
}

}  // namespace

extern "C" VTP_API int vtp_ugns_neighbors_noalloc(const float *d_pos, uint32_t n, const float lb[3],
                                                  const float size[3], float cell, uint32_t max_nbr,
                                                  uint32_t *d_counts, uint32_t *d_nbrs, void *stream) {
    if (!lb || !size || (n > 0 && (!d_pos || !d_counts || !d_nbrs)))
        return vtp::fail(VTP_ERR_ARG, "null argument");
    if (n > kMaxParticles)
        return vtp::fail(VTP_ERR_BOUNDS, "vtp_ugns_neighbors_noalloc: " + std::to_string(n) +
                                             " particles exceed the scratch limit of " +
                                             std::to_string(kMaxParticles));
    if (!(cell > 0.f) || !std::isfinite(cell) || max_nbr < 1 || max_nbr > 1024)
        return vtp::fail(VTP_ERR_ARG, "cell must be finite and > 0, and max_nbr in [1, 1024]");
    for (int a = 0; a < 3; ++a)
        if (!std::isfinite(lb[a]) || !std::isfinite(size[a]) || !(size[a] > 0.f))
            return vtp::fail(VTP_ERR_ARG, "vtp_ugns_neighbors_noalloc: lb must be finite and size finite and > 0");
    // Cells per axis, checked before the integer conversion (a tiny cell would
    // otherwise overflow int).
    double cells[3];
    for (int a = 0; a < 3; ++a) {
        cells[a] = std::ceil((double)(size[a] / cell));
        if (!(cells[a] >= 1.0) || cells[a] > (double)kMaxKeys)
            return vtp::fail(VTP_ERR_BOUNDS, "vtp_ugns_neighbors_noalloc: grid of " +
                                                 std::to_string(cells[a]) + " cells along one axis exceeds the "
                                                 "scratch limit of " + std::to_string(kMaxKeys) + " cell buckets");
    }
    vtp::Grid g{};
    g.lbx = lb[0]; g.lby = lb[1]; g.lbz = lb[2];
    g.cell = cell;
    g.gx = (int)cells[0];
    g.gy = (int)cells[1];
    g.gz = (int)cells[2];
    const uint64_t maxkey = (uint64_t)g.gz * g.gy * g.gx + (uint64_t)g.gy * g.gx + g.gx;
    if (maxkey + 2 > kMaxKeys)
        return vtp::fail(VTP_ERR_BOUNDS, "vtp_ugns_neighbors_noalloc: grid of " + std::to_string(maxkey + 2) +
                                             " cell buckets exceeds the scratch limit of " +
                                             std::to_string(kMaxKeys));
    g.nkey = (uint32_t)(maxkey + 1);
    g.d2max = sqrt_limit(cell);
    g.maxnbr = max_nbr;
    if (n == 0) return VTP_OK;
    unsigned char *base = nullptr;
    const int rc = arena_base(&base);
    if (rc) return rc;
    cudaError_t e;
    const Arena a = arena_at(base);
    cudaStream_t st = (cudaStream_t)stream;
    const uint32_t nb = g.nkey + 1;
    const uint32_t tiles = (nb + kScanTile - 1) / kScanTile;
    // The arena keeps the previous call's contents: the cell counters must start at zero.
    e = cudaMemsetAsync(a.count, 0, (size_t)nb * sizeof(uint32_t), st);
    if (e != cudaSuccess) return vtp::fail(VTP_ERR_CUDA, cudaGetErrorString(e));
    k_na_hash<<<nblk(n, 256), 256, 0, st>>>(g, n, d_pos, a);
    k_na_tile_sums<<<tiles, kScanThreads, 0, st>>>(nb, a);
    k_na_scan_tiles<<<1, 1024, 0, st>>>(tiles, a);
    k_na_scan<<<tiles, kScanThreads, 0, st>>>(nb, a);
    k_na_scatter<<<nblk(n, 256), 256, 0, st>>>(n, a);
    k_na_rank<<<nblk(n, 256), 256, 0, st>>>(g, n, d_pos, a);
    constexpr int kBlock = vtp::kCellWarps * 32;
    if (n <= vtp::kScan8Rows) k_na_walk<8><<<nblk(n, vtp::kCellWarps * 8), kBlock, 0, st>>>(g, n, a, d_counts, d_nbrs);
    else k_na_walk<32><<<nblk(n, kBlock), kBlock, 0, st>>>(g, n, a, d_counts, d_nbrs);
    e = cudaGetLastError();
    if (e != cudaSuccess) return vtp::fail(VTP_ERR_CUDA, cudaGetErrorString(e));
    return VTP_OK;
}
