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
#include <climits>
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
constexpr size_t kOffSorted = kOffTmp + align256(4ull * kMaxParticles);
constexpr size_t kOffPos = kOffSorted + align256(4ull * kMaxParticles);
constexpr size_t kOffCount = kOffPos + align256(16ull * kMaxParticles);
constexpr size_t kOffStart = kOffCount + align256(4ull * (kMaxKeys + 1));
constexpr size_t kOffTiles = kOffStart + align256(4ull * (kMaxKeys + 2));
constexpr size_t kArenaBytes = kOffTiles + align256(4ull * kMaxTiles);

static_assert(kArenaBytes == VTP_NOALLOC_SCRATCH_BYTES, "scratch size in vtp.h out of date");

__device__ __align__(256) unsigned char g_noalloc_scratch[kArenaBytes];

struct Arena {
    uint32_t *key, *rank, *tmp, *sorted, *count, *start, *tiles;
    float4 *pos;
};

Arena arena_at(unsigned char *base) {
    Arena a;
    a.key = (uint32_t *)(base + kOffKey);
    a.rank = (uint32_t *)(base + kOffRank);
    a.tmp = (uint32_t *)(base + kOffTmp);
    a.sorted = (uint32_t *)(base + kOffSorted);
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
    a.sorted[dst] = me;
    a.pos[dst] = make_float4(pos[3 * (size_t)me], pos[3 * (size_t)me + 1], pos[3 * (size_t)me + 2],
                             __uint_as_float(me));
}

// Lists of up to R rows of one cell (as cell_lists of ugns.cu, for one run per cell and lists that
// are rows of a plain array).  Lane l works for row l % R, lane h * R + k taking the h-th share of
// row k's candidates.
template <uint32_t R>
__device__ __forceinline__ void na_cell_lists(vtp::CellScratch &S, uint32_t f0, uint32_t len, uint32_t excl,
                                              uint32_t total, bool live, float4 p, const vtp::Grid &g, const Arena &a,
                                              uint32_t *__restrict__ counts, uint32_t *__restrict__ nbrs) {
    constexpr unsigned kAll = 0xffffffffu;
    constexpr uint32_t H = 32u / R;
    const uint32_t lane = threadIdx.x & 31u, k = lane % R, h = lane / R, cap = g.maxnbr - 1u;
    const uint64_t px = vtp::f2_pack(-p.x, -p.x), py = vtp::f2_pack(-p.y, -p.y), pz = vtp::f2_pack(-p.z, -p.z);
    const uint32_t to0 = (uint32_t)__cvta_generic_to_shared(&S.kept[lane][0]);
    uint32_t found = 0;
    for (uint32_t wb = 0; wb < total; wb += vtp::kCellWindow) {
        const uint32_t wl = min(vtp::kCellWindow, total - wb);
        const uint32_t share = ((wl + H - 1u) / H + 7u) & ~7u;
        // The window's candidates: sorted slots first, then positions and ids in their place.
        __syncwarp();
        const uint32_t o0 = wb > excl ? min(wb - excl, len) : 0u, o1 = wb + wl > excl ? min(wb + wl - excl, len) : 0u;
        for (uint32_t o = o0; o < o1; ++o) S.cand[excl + o - wb] = f0 + o;
        __syncwarp();
        for (uint32_t q = lane; q < H * share; q += 32u) {
            const float far = __int_as_float(0x7f800000);
            float4 v = make_float4(far, far, far, 0.f);
            if (q < wl) {
                v = __ldg(a.pos + S.cand[q]);
                S.cand[q] = __float_as_uint(v.w);
            }
            S.x[0][q] = v.x;
            S.x[1][q] = v.y;
            S.x[2][q] = v.z;
        }
        __syncwarp();
        uint32_t to = to0;
        for (uint32_t off = 0; off < share; off += 8u) {
            vtp::test4(S, h * share + off, off, to, px, py, pz, g.d2max);
            vtp::test4(S, h * share + off + 4u, off + 4u, to, px, py, pz, g.d2max);
        }
        const uint32_t mine = live ? to - to0 : 0u;
        uint32_t x = mine;
#pragma unroll
        for (uint32_t o = R; o < 32u; o <<= 1) {
            const uint32_t y = __shfl_up_sync(kAll, x, o);
            if (lane >= o) x += y;
        }
        __syncwarp();
#pragma unroll
        for (uint32_t r = 0; r < R; r += 4) {   // 8 consecutive entries of 4 rows at a time
            const uint32_t kk = r + (lane >> 3);
            uint32_t lo[H];
#pragma unroll
            for (uint32_t t = 0; t < H; ++t) lo[t] = __shfl_sync(kAll, x - mine, (int)(kk + R * t));
            const uint32_t n = __shfl_sync(kAll, x, (int)(kk + 32u - R));
            const uint32_t before = __shfl_sync(kAll, found, (int)kk);
            const uint32_t id = __float_as_uint(__shfl_sync(kAll, p.w, (int)kk));
            uint32_t *out = nbrs + (size_t)id * g.maxnbr + 1u;
            for (uint32_t e = lane & 7u; e < n && before + e < cap; e += 8u) {
                uint32_t at = kk * vtp::kCellKept + e, share_of = 0;
#pragma unroll
                for (uint32_t t = 1; t < H; ++t)
                    if (e >= lo[t]) at = (kk + R * t) * vtp::kCellKept + (e - lo[t]), share_of = t * share;
                out[before + e] = S.cand[share_of + (&S.kept[0][0])[at]];
            }
        }
        found += __shfl_sync(kAll, x, (int)(k + 32u - R));
    }
    // Self, the count and the unused slots.
#pragma unroll
    for (uint32_t r = 0; r < R; r += 4) {
        const uint32_t kk = r + (lane >> 3), e0 = lane & 7u;
        const uint32_t n = min(__shfl_sync(kAll, found, (int)kk), cap) + 1u;
        const uint32_t id = __float_as_uint(__shfl_sync(kAll, p.w, (int)kk));
        if (!__shfl_sync(kAll, (int)live, (int)kk)) continue;
        uint32_t *out = nbrs + (size_t)id * g.maxnbr;
        if (e0 == 0) {
            out[0] = id;
            counts[id] = n;
        }
        for (uint32_t e = n + e0; e < g.maxnbr; e += 8u) out[e] = 0xffffffffu;
    }
}

// Lists in the reference layout: self first, then the 27 cells in the reference's offset order,
// particles of a cell by ascending id.  One warp per occupied cell (its candidates are laid out and
// tested as in the solvers' builder), found among the kNaScan sorted slots each warp looks at.
// Bound by issue; a thread per particle wrote every entry to a line of its own and walked its 27
// cells alone.  404,891 particles, 60 slots: whole call 292 -> 205 us (B200).
constexpr uint32_t kNaScan = 8;
__global__ void __launch_bounds__(vtp::kCellWarps * 32, 7) k_na_walk(vtp::Grid g, uint32_t n, Arena a,
                                                                     uint32_t *__restrict__ counts,
                                                                     uint32_t *__restrict__ nbrs) {
    __shared__ __align__(16) vtp::CellScratch scratch[vtp::kCellWarps];
    constexpr unsigned kAll = 0xffffffffu;
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t first = (blockIdx.x * vtp::kCellWarps + (threadIdx.x >> 5)) * kNaScan;
    if (first >= n) return;
    vtp::CellScratch &S = scratch[threadIdx.x >> 5];
    const int3 o = vtp::nbr_offset((int)min(lane, 26u));
    uint32_t cell_end = 0;
    bool leads = false, outside = false;
    uint32_t id = 0;
    if (lane < kNaScan && first + lane < n) {
        const float4 p = a.pos[first + lane];
        id = __float_as_uint(p.w);
        const int3 c = vtp::cell_of(p.x, p.y, p.z, g);
        if (vtp::cell_available(c, g)) {
            const uint32_t k = vtp::cell_key(c, g);
            leads = a.start[k] == first + lane;
            cell_end = a.start[k + 1];
        } else {
            outside = true;
            counts[id] = 0;
        }
    }
    for (unsigned m = __ballot_sync(kAll, outside); m; m &= m - 1u) {   // outside the grid: an empty list
        uint32_t *out = nbrs + (size_t)__shfl_sync(kAll, id, __ffs((int)m) - 1) * g.maxnbr;
        for (uint32_t e = lane; e < g.maxnbr; e += 32u) out[e] = 0xffffffffu;
    }
    for (unsigned todo = __ballot_sync(kAll, leads); todo; todo &= todo - 1u) {
        const int leader = __ffs((int)todo) - 1;
        const uint32_t beg = first + (uint32_t)leader, end = __shfl_sync(kAll, cell_end, leader);
        int3 at = make_int3(INT_MIN, 0, 0);   // the cell whose run is held
        uint32_t f0 = 0, len = 0, excl = 0, total = 0;
        for (uint32_t rg = beg; rg < end; rg += 8u) {
            const uint32_t m = min(8u, end - rg);
            const float4 p = a.pos[rg + min(lane & 7u, m - 1u)];
            const int3 c = vtp::cell_of(p.x, p.y, p.z, g);
            // A cell on the grid's inclusive upper face shares its bucket with another cell: one
            // round per cell among these rows.
            for (unsigned left = (1u << m) - 1u; left;) {
                const int f = __ffs((int)left) - 1;
                const int3 c0 = make_int3(__shfl_sync(kAll, c.x, f), __shfl_sync(kAll, c.y, f), __shfl_sync(kAll, c.z, f));
                const bool mine = ((left >> (lane & 7u)) & 1u) && c.x == c0.x && c.y == c0.y && c.z == c0.z;
                left &= ~__ballot_sync(kAll, mine);
                if (c0.x != at.x || c0.y != at.y || c0.z != at.z) {
                    at = c0;
                    f0 = len = 0;
                    const int3 cc = make_int3(c0.x + o.x, c0.y + o.y, c0.z + o.z);
                    if (lane < 27u && vtp::cell_available(cc, g)) {
                        const uint32_t k = vtp::cell_key(cc, g);
                        f0 = a.start[k];
                        len = a.start[k + 1] - f0;
                    }
                    uint32_t incl = len;
#pragma unroll
                    for (int d = 1; d < 32; d <<= 1) {
                        const uint32_t y = __shfl_up_sync(kAll, incl, d);
                        if ((int)lane >= d) incl += y;
                    }
                    excl = incl - len;
                    total = __shfl_sync(kAll, incl, 31);
                }
                if (m <= 4u) {
                    const int s = (int)(lane & 3u);
                    const float4 p4 = make_float4(__shfl_sync(kAll, p.x, s), __shfl_sync(kAll, p.y, s),
                                                  __shfl_sync(kAll, p.z, s), __shfl_sync(kAll, p.w, s));
                    const bool live = __shfl_sync(kAll, (int)mine, s) != 0;
                    na_cell_lists<4>(S, f0, len, excl, total, live, p4, g, a, counts, nbrs);
                } else {
                    na_cell_lists<8>(S, f0, len, excl, total, mine, p, g, a, counts, nbrs);
                }
                __syncwarp();
            }
        }
    }
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
    k_na_walk<<<nblk(n, vtp::kCellWarps * kNaScan), vtp::kCellWarps * 32, 0, st>>>(g, n, a, d_counts, d_nbrs);
    e = cudaGetLastError();
    if (e != cudaSuccess) return vtp::fail(VTP_ERR_CUDA, cudaGetErrorString(e));
    return VTP_OK;
}
