// DFSPH solver passes for sm_100a (fluid rows only; rows are cell-sorted).
//
// Restates DFSPHSolver::tick (DFSPHSolver.cpp:339-406) with the kernels of
// DFSPHCudaImpl.cu regrouped into neighbour passes:
//   ratio_alpha : compute_compression_ratio_cuda + compute_df_beta_cuda (:85-140)
//   solve_a     : compute_delta_compression_ratio_cuda +
//                 update_delta_compression_ratio_from_vel_adv_cuda +
//                 compute_kappa_{div,incomp}_... (:142-196, :355-367) and the
//                 per-block FP64 partial sums of the residual
//   solve_b     : vf_update_vel_adv_from_kappa_{div,incomp}_cuda (:198-220, :369-391)
//   solve_end   : the residual (mean over fluid objects of the object's mean
//                 clamped compression error, as vfsph_div computes it with
//                 cal_mean, :449-503) in FP64 on the device, the stop test
//                 (residual < threshold or iteration > 100) and the loop
//                 condition of the CUDA-graph WHILE node
//   viscosity   : apply_pressure_acc (:505-521) evaluated on the fly for i
//                 and j, then clear_acc + add_acc_gravity +
//                 add_acc_explicit_lap_vis + acc_2_vel (:222-296, :523-554)
//   vis_normal / tension : the same with compute_surface_normal_cuda and
//                 add_acc_surface_tension_cuda (:298-353) when gamma != 0
//   finalize    : apply_pressure_acc + update_pos_cuda (:393-404)
#include "dfsph.h"
#include "team.cuh"

#include <algorithm>

namespace vtp {

namespace {

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}

// Deterministic block sum; result valid in thread 0.
__device__ __forceinline__ double block_sum(double v) {
    __shared__ double sm[32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    v = warp_sum(v);
    __syncthreads();
    if (lane == 0) sm[wid] = v;
    __syncthreads();
    const int nw = (blockDim.x + 31) >> 5;
    double s = 0.0;
    if (wid == 0) {
        s = lane < nw ? sm[lane] : 0.0;
        s = warp_sum(s);
    }
    return s;
}

__device__ __forceinline__ float4 pressure_applied(float4 v, float4 va, float inv_dt, float dt) {
    // add_acc_pressure_cuda + acc_2_vel: acc = (v* - v) / dt; v += acc dt.
    float4 o = v;
    o.x = __fmaf_rn((va.x - v.x) * inv_dt, dt, v.x);
    o.y = __fmaf_rn((va.y - v.y) * inv_dt, dt, v.y);
    o.z = __fmaf_rn((va.z - v.z) * inv_dt, dt, v.z);
    return o;
}

// Time step of the running substep: the fixed dt, or the adaptive one on the device
// (1/dt and 1/dt^2 formed as the host forms them for the fixed step).
struct StepDt {
    float dt, inv_dt, inv_dt2;
};
__device__ __forceinline__ StepDt step_dt(const DfsphArgs &a) {
    if (!a.dtp) return StepDt{a.dt, a.inv_dt, a.inv_dt2};
    const float dt = *a.dtp;
    const float inv = 1.f / dt;
    return StepDt{dt, inv, inv * inv};
}

__global__ void __launch_bounds__(256) k_rigid_volume(DfsphArgs a, const uint32_t *__restrict__ bncnt,
                                                      const uint32_t *__restrict__ bnbr,
                                                      float *__restrict__ rest_density_b) {
    // compute_rigid_volume_cuda (DFSPHCudaImpl.cu:63-83): V_b = 1 / sum_{boundary j} W_ij,
    // boundary rest_density = V_b * rho_b.
    uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= a.nb) return;
    uint32_t i = a.nf + r;
    float4 p = a.pos[i];
    uint32_t n = bncnt[r];
    float delta = n > 0 ? a.k.w0 : 0.f;
    const uint32_t *lst = bnbr + ell_index(r, 0, a.shape);
    for (uint32_t t = 0; t + 1 < n; ++t) {
        uint32_t j = lst[ell_slot(t, a.shape)];
        if (j < a.nf) continue;
        float4 q = a.pos[j];
        delta += cubic_w(dist2(p.x - q.x, p.y - q.y, p.z - q.z), a.k);
    }
    float vb = 1.f / delta;
    p.w = vb;
    a.pos[i] = p;
    rest_density_b[r] = vb * a.rho_b;
}

__device__ __forceinline__ void reset_solve(SolveState *s, LoopState *loop, int nscenes);

// What the ratio / alpha pass prepares beside its own results for the solver's substep: both
// solves' states (first block), and row r's {pos, v*} for the first one.
__device__ __forceinline__ void start_solves(const DfsphArgs &a) {
    if (!a.reset || blockIdx.x != 0) return;
    reset_solve(a.reset, a.reset_loop, a.nreset);
    reset_solve(a.reset + a.nreset, a.reset_loop + 1, a.nreset);
}
__device__ __forceinline__ void pack_row(const DfsphArgs &a, uint32_t r, const float4 &p, const float4 &v) {
    if (!a.pack) return;
    a.pack[2 * (size_t)r] = p;
    a.pack[2 * (size_t)r + 1] = v;
}

// DFSPH compression ratio and alpha of one row (compute_compression_ratio_cuda +
// compute_df_beta_cuda, DFSPHCudaImpl.cu:85-140), accumulated entry by entry in list
// order, every rounding explicit.
struct RatioAlpha {
    float ratio, a1x, a1y, a1z, a2;

    // self_w: the self term V_i W(0) (0 for a row outside the grid, which has no list)
    __device__ __forceinline__ void begin(float self_w) {
        ratio = self_w;
        a1x = a1y = a1z = 0.f;
        a2 = 1e-6f;
    }
    // One list entry j: d2 = |x_i - x_j|^2, (dx, dy, dz) = x_i - x_j, vj = V_j.
    __device__ __forceinline__ void add(float d2, float dx, float dy, float dz, float vj, bool fluid_j,
                                        const Cubic &k, float inv_mf) {
        float w, g;
        cubic_wg(d2, k, w, g);
        ratio = __fmaf_rn(vj, w, ratio);
        const float gx = __fmul_rn(g, dx), gy = __fmul_rn(g, dy), gz = __fmul_rn(g, dz);
        a1x = __fmaf_rn(vj, gx, a1x);
        a1y = __fmaf_rn(vj, gy, a1y);
        a1z = __fmaf_rn(vj, gz, a1z);
        if (fluid_j) a2 = __fmaf_rn(__fmul_rn(__fmul_rn(dist2(gx, gy, gz), vj), vj), inv_mf, a2);
    }
    __device__ __forceinline__ float alpha(float mass_f) const {
        const float al = __fadd_rn(__fdiv_rn(dist2(a1x, a1y, a1z), mass_f), a2);
        return al < 1e-6f ? 1e-6f : al;
    }
};

struct PV {
    float4 q, v;
};
struct PN {
    float4 q, n;
};

template <int U>
__global__ void __launch_bounds__(256) k_ratio_alpha(DfsphArgs a) {
    start_solves(a);
    uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= a.nf || halo_ghost(a, r)) return;
    const float4 p = a.pos[r];
    const uint32_t n = a.ncnt[r];
    RatioAlpha ra;
    ra.begin(n > 0 ? __fmul_rn(p.w, a.k.w0) : 0.f);   // self term V_i W(0)
    const float inv_mf = __fdiv_rn(1.f, a.mass_f);
    const uint32_t *lst = a.nbr + row_index(r, a.shape);
    nbr_loop<U>(lst, n > 0 ? n - 1 : 0, [&](uint32_t j) { return ldg4(a.pos + j); },
                [&](uint32_t j, const float4 &q) {
                    const float dx = p.x - q.x, dy = p.y - q.y, dz = p.z - q.z;
                    ra.add(dist2(dx, dy, dz), dx, dy, dz, q.w, j < a.nf, a.k, inv_mf);
                });
    if (a.pack) pack_row(a, r, p, a.vadv[r]);
    a.ratio[r] = ra.ratio;
    a.alpha[r] = ra.alpha(a.mass_f);
}

// The same with a team per row (team.cuh).
template <int L>
__global__ void __launch_bounds__(kTeamRows * L) k_team_ratio_alpha(DfsphArgs a) {
    __shared__ TeamTerms<8, L> S;   // V_j, W, gradW, |gradW|^2 V_j^2 (fluid j)
    start_solves(a);
    const uint32_t r = blockIdx.x * kTeamRows + team_row<L>(), l = team_lane<L>();
    const bool live = r < a.nf && !halo_ghost(a, r);
    float4 p = make_float4(0.f, 0.f, 0.f, 0.f);
    uint32_t n = 0;
    if (live) {
        p = a.pos[r];
        n = a.ncnt[r];
    }
    const float inv_mf = __fdiv_rn(1.f, a.mass_f);
    // lane 0: ratio, lanes 1..3: a1; every lane: a2
    float acc = l == 0 && n > 0 ? __fmul_rn(p.w, a.k.w0) : 0.f, a2 = 1e-6f;
    team_walk<L, 8>(
        S, a.nbr + ell_index(r, 0, a.shape), n > 0 ? n - 1 : 0, [&](uint32_t j) { return ldg4(a.pos + j); },
        [&](uint32_t j, const float4 &q, float *o) {
            const float dx = p.x - q.x, dy = p.y - q.y, dz = p.z - q.z;
            float w, g;
            cubic_wg(dist2(dx, dy, dz), a.k, w, g);
            const float gx = __fmul_rn(g, dx), gy = __fmul_rn(g, dy), gz = __fmul_rn(g, dz);
            o[0] = q.w;
            o[1] = w;
            o[2] = gx;
            o[3] = gy;
            o[4] = gz;
            o[5] = j < a.nf ? __fmul_rn(__fmul_rn(dist2(gx, gy, gz), q.w), q.w) : 0.f;
            o[6] = o[7] = 0.f;
        },
        [&](const float *e) {
            acc = __fmaf_rn(e[0], e[1 + (l & 3)], acc);
            a2 = __fmaf_rn(e[5], inv_mf, a2);
        });
    RatioAlpha ra;
    ra.ratio = acc;
    ra.a1x = team_get<L>(acc, 1);
    ra.a1y = team_get<L>(acc, 2);
    ra.a1z = team_get<L>(acc, 3);
    ra.a2 = a2;
    if (!live || l != 0) return;
    if (a.pack) pack_row(a, r, p, a.vadv[r]);
    a.ratio[r] = ra.ratio;
    a.alpha[r] = ra.alpha(a.mass_f);
}

// V_j gradW_ij . (v*_i - v*_j) of a pair: e = {x_j, V_j}, v*_j.
__device__ __forceinline__ float solve_a_term(const float4 &p, const float4 &vi, const F4x2 &e, const Cubic &k) {
    const float rx = p.x - e.a.x, ry = p.y - e.a.y, rz = p.z - e.a.z;
    const float g = cubic_g(dist2(rx, ry, rz), k);
    const float dot = g * (rx * (vi.x - e.b.x) + ry * (vi.y - e.b.y) + rz * (vi.z - e.b.z));
    return dot * e.a.w;
}

// Tile kernels run a persistent grid over the scene-offset tiles; a tile of a
// scene whose solve has stopped is skipped (block-uniform test).
template <bool MULTI, int U>
__global__ void __launch_bounds__(256) k_solve_a(DfsphArgs a) {
    const StepDt T = step_dt(a);
    for (uint32_t t = blockIdx.x; t < a.ntiles; t += gridDim.x) {
        const uint4 tile = a.tiles[t];
        const bool stopped = a.state[tile.z].stopped != 0;
        if (a.tile_ran && threadIdx.x == 0) a.tile_ran[t] = stopped ? 0u : 1u;
        if (stopped) continue;
        const uint32_t r = tile.x + threadIdx.x;
        double contrib = 0.0;
        int obj = 0;
        if (threadIdx.x < tile.y && !halo_ghost(a, r)) {
            const float4 p = a.pos[r];
            const float4 vi = a.vadv[r];
            const uint32_t n = a.ncnt[r];
            float d = a.ratio[r] - 1.f;
            const uint32_t *lst = a.nbr + row_index(r, a.shape);
            nbr_loop<U>(lst, n > 0 ? n - 1 : 0, [&](uint32_t j) { return ldg8(a.pva + 2 * (size_t)j); },
                        [&](uint32_t, const F4x2 &e) { d = __fmaf_rn(solve_a_term(p, vi, e, a.k), T.dt, d); });
            if (d < 0.f) d = 0.f;
            a.delta[r] = d;
            const float kap = d / a.alpha[r] * T.inv_dt2 / p.w;
            a.kappa[r] = kap;
            const float4 pkr = make_float4(p.x, p.y, p.z, kap);
            a.pk[r] = pkr;
            halo_each(a, r, [&](const PeerRows &P, uint32_t q) {
                P.kappa[q] = kap;
                P.pk[q] = pkr;
            });
            contrib = (double)d;
            if (MULTI) obj = (int)a.obj_of[a.orig[r]] - (int)a.scene_tiles[tile.z].obj0;
        }
        if (!MULTI) {
            double s = block_sum(contrib);
            if (threadIdx.x == 0) a.partials[t] = s;
        } else {
            const int no = (int)a.scene_tiles[tile.z].nobj;
            for (int o = 0; o < no; ++o) {
                double s = block_sum(obj == o ? contrib : 0.0);
                if (threadIdx.x == 0) a.partials[(size_t)t * a.nobj_max + o] = s;
            }
        }
    }
}

// solve_a with a team per row: a block takes a 32-row piece of a tile (`pieces` per tile) and
// leaves the sum of its rows' errors; k_solve_end adds a tile's pieces as the block sum above does.
template <bool MULTI, int L>
__global__ void __launch_bounds__(kTeamRows * L) k_team_solve_a(DfsphArgs a, uint32_t pieces) {
    __shared__ TeamTerms<1, L> S;
    __shared__ float err[kTeamRows];
    const StepDt T = step_dt(a);
    const uint32_t t = blockIdx.x / pieces, part = blockIdx.x - t * pieces;
    const uint4 tile = a.tiles[t];
    const bool stopped = a.state[tile.z].stopped != 0;
    if (a.tile_ran && part == 0 && threadIdx.x == 0) a.tile_ran[t] = stopped ? 0u : 1u;
    if (stopped) return;
    const uint32_t row = part * kTeamRows + team_row<L>(), r = tile.x + row;
    const bool live = row < tile.y && !halo_ghost(a, r);
    float4 p = make_float4(0.f, 0.f, 0.f, 1.f), vi = p;
    float d = 0.f, al = 1.f;
    uint32_t n = 0;
    if (live) {
        p = a.pos[r];
        vi = a.vadv[r];
        n = a.ncnt[r];
        al = a.alpha[r];
        d = a.ratio[r] - 1.f;
    }
    team_walk<L, 1>(
        S, a.nbr + ell_index(r, 0, a.shape), n > 0 ? n - 1 : 0,
        [&](uint32_t j) { return ldg8(a.pva + 2 * (size_t)j); },
        [&](uint32_t, const F4x2 &e, float *o) { o[0] = solve_a_term(p, vi, e, a.k); },
        [&](const float *e) { d = __fmaf_rn(e[0], T.dt, d); });
    if (d < 0.f) d = 0.f;
    if (live && team_lane<L>() == 0) {
        a.delta[r] = d;
        const float kap = d / al * T.inv_dt2 / p.w;
        a.kappa[r] = kap;
        const float4 pkr = make_float4(p.x, p.y, p.z, kap);
        a.pk[r] = pkr;
        halo_each(a, r, [&](const PeerRows &P, uint32_t q) {
            P.kappa[q] = kap;
            P.pk[q] = pkr;
        });
    }
    if (team_lane<L>() == 0) err[team_row<L>()] = live ? d : 0.f;
    __syncthreads();
    if (threadIdx.x >= 32) return;
    const double contrib = (double)err[threadIdx.x];
    if (!MULTI) {
        const double s = warp_sum(contrib);
        if (threadIdx.x == 0) a.partials[blockIdx.x] = s;
    } else {
        const uint32_t er = part * kTeamRows + threadIdx.x;
        const int obj = er < tile.y ? (int)a.obj_of[a.orig[tile.x + er]] - (int)a.scene_tiles[tile.z].obj0 : 0;
        const int no = (int)a.scene_tiles[tile.z].nobj;
        for (int o = 0; o < no; ++o) {
            const double s = warp_sum(obj == o ? contrib : 0.0);
            if (threadIdx.x == 0) a.partials[(size_t)blockIdx.x * a.nobj_max + o] = s;
        }
    }
}

// Staged solve_a: one block per brick (staged.h); the block copies the
// packed {x, v*} rows of the group's neighbourhood into shared memory and each
// row gathers through its slot list, in list order, so delta and kappa are
// the bits the unstaged pass computes.  A group whose neighbourhood exceeds
// the capacity, and the rows outside the grid (block ngroups), gather from
// global memory.  The FP64 residual partials are per group.
template <bool MULTI, int U>
__global__ void __launch_bounds__(kStageBlock) k_solve_a_staged(DfsphArgs a) {
    extern __shared__ float4 stage[];   // slot s = {stage[2s], stage[2s + 1]}
    __shared__ GroupPlan P;
    if (a.state[0].stopped) return;
    const StepDt T = step_dt(a);
    const uint32_t grp = blockIdx.x;
    const SceneGrid g = a.sc.sg[0];
    uint32_t r0, r1;
    bool staged = false;
    if (grp == a.stg.ngroups) {
        const uint32_t k = g.key_base + g.nkey;
        r0 = __ldg(a.stg.fstart + k);
        r1 = __ldg(a.stg.fstart + k + 1);
    } else {
        const uint2 rows = group_rows(grp, g, a.stg);
        r0 = rows.x;
        r1 = rows.y;
        if (r0 != r1) {
            plan_group(P, grp, g, a.stg);
            staged = P.total <= a.stg.scap;
        }
    }
    if (staged) {
        for (uint32_t s = threadIdx.x; s < P.total; s += blockDim.x) {
            bool b;
            const uint32_t j = a.stg.mode == 0 ? slot_row<0>(P, slot_cell(P, s), s, b)
                                               : slot_row<1>(P, slot_cell(P, s), s, b);
            const F4x2 e = ldg8(a.pva + 2 * (size_t)j);
            stage[2 * s] = e.a;
            stage[2 * s + 1] = e.b;
        }
        __syncthreads();
    }
    double contrib = 0.0;
    for (uint32_t r = r0 + threadIdx.x; r < r1; r += blockDim.x) {
        const float4 p = a.pos[r];
        const float4 vi = a.vadv[r];
        const uint32_t n = a.ncnt[r];
        float d = a.ratio[r] - 1.f;
        auto use = [&](auto, const F4x2 &e) {
            const float rx = p.x - e.a.x, ry = p.y - e.a.y, rz = p.z - e.a.z;
            const float gw = cubic_g(dist2(rx, ry, rz), a.k);
            const float dot = gw * (rx * (vi.x - e.b.x) + ry * (vi.y - e.b.y) + rz * (vi.z - e.b.z));
            d = __fmaf_rn(dot * e.a.w, T.dt, d);
        };
        const uint32_t cnt = n > 0 ? n - 1 : 0;
        if (staged) {
            slot_loop<U>(a.stg.snbr + row_index(r, a.shape), cnt,
                         [&](uint16_t s) {
                             uint32_t q = (uint32_t)(s & 0x7fffu);
#ifdef VTP_CHECKED
                             if (q >= P.total) {   // a slot outside the staged rows: record it, read slot 0
                                 atomicOr(a.status, ST_BOUNDS);
                                 q = 0;
                             }
#endif
                             q *= 2u;
                             return F4x2{stage[q], stage[q + 1]};
                         },
                         use);
        } else {
            nbr_loop<U>(a.nbr + row_index(r, a.shape), cnt,
                        [&](uint32_t j) { return ldg8(a.pva + 2 * (size_t)j); }, use);
        }
        if (d < 0.f) d = 0.f;
        a.delta[r] = d;
        const float kap = d / a.alpha[r] * T.inv_dt2 / p.w;
        a.kappa[r] = kap;
        a.pk[r] = make_float4(p.x, p.y, p.z, kap);
        contrib += (double)d;
    }
    if (!MULTI) {
        const double s = block_sum(contrib);
        if (threadIdx.x == 0) a.partials[grp] = s;
    } else {
        const int no = (int)a.scene_tiles[0].nobj;
        for (int o = 0; o < no; ++o) {
            double c = 0.0;
            for (uint32_t r = r0 + threadIdx.x; r < r1; r += blockDim.x)
                if ((int)a.obj_of[a.orig[r]] - (int)a.scene_tiles[0].obj0 == o) c += (double)a.delta[r];
            const double s = block_sum(c);
            if (threadIdx.x == 0) a.partials[(size_t)grp * a.nobj_max + o] = s;
        }
    }
}

// Staged solve_b: gathers the packed {x, kappa_j} (fluid) / {x, V_j}
// (boundary) rows from the group's staged copy; bit 15 of a slot marks a
// boundary neighbour.
template <int U>
__global__ void __launch_bounds__(kStageBlock) k_solve_b_staged(DfsphArgs a) {
    extern __shared__ float4 stage[];
    __shared__ GroupPlan P;
    if (a.state && a.state[0].stopped) return;
    const StepDt T = step_dt(a);
    const uint32_t grp = blockIdx.x;
    const SceneGrid g = a.sc.sg[0];
    uint32_t r0, r1;
    bool staged = false;
    if (grp == a.stg.ngroups) {
        const uint32_t k = g.key_base + g.nkey;
        r0 = __ldg(a.stg.fstart + k);
        r1 = __ldg(a.stg.fstart + k + 1);
    } else {
        const uint2 rows = group_rows(grp, g, a.stg);
        r0 = rows.x;
        r1 = rows.y;
        if (r0 == r1) return;
        plan_group(P, grp, g, a.stg);
        staged = P.total <= a.stg.scap;
    }
    if (staged) {
        for (uint32_t s = threadIdx.x; s < P.total; s += blockDim.x) {
            bool b;
            const uint32_t j = a.stg.mode == 0 ? slot_row<0>(P, slot_cell(P, s), s, b)
                                               : slot_row<1>(P, slot_cell(P, s), s, b);
            stage[s] = __ldg(a.pk + j);
        }
        __syncthreads();
    }
    for (uint32_t r = r0 + threadIdx.x; r < r1; r += blockDim.x) {
        const float4 p = a.pos[r];
        float4 v = a.vadv[r];
        const float ki = a.kappa[r];
        const uint32_t n = a.ncnt[r];
        const float mi = a.rest_density ? a.rest_density[r] * p.w : a.mass_f;
        const float ci = T.dt * p.w / mi;
        auto step = [&](bool fj, const float4 &e) {
            const float Vj = fj ? a.vol_f : e.w, kj = fj ? e.w : 0.f;
            const float rx = p.x - e.x, ry = p.y - e.y, rz = p.z - e.z;
            const float gw = cubic_g(dist2(rx, ry, rz), a.k);
            const float s = ci * Vj * (ki + kj) * gw;
            v.x = __fmaf_rn(-s, rx, v.x);
            v.y = __fmaf_rn(-s, ry, v.y);
            v.z = __fmaf_rn(-s, rz, v.z);
        };
        const uint32_t cnt = n > 0 ? n - 1 : 0;
        if (staged) {
            slot_loop<U>(a.stg.snbr + row_index(r, a.shape), cnt,
                         [&](uint16_t s) {
                             uint32_t q = (uint32_t)(s & 0x7fffu);
#ifdef VTP_CHECKED
                             if (q >= P.total) {   // a slot outside the staged rows: record it, read slot 0
                                 atomicOr(a.status, ST_BOUNDS);
                                 q = 0;
                             }
#endif
                             return stage[q];
                         },
                         [&](uint16_t s, const float4 &e) { step(!(s & kSlotBoundary), e); });
        } else {
            nbr_loop<U>(a.nbr + row_index(r, a.shape), cnt, [&](uint32_t j) { return ldg4(a.pk + j); },
                        [&](uint32_t j, const float4 &e) { step(j < a.nf, e); });
        }
        a.vadv[r] = v;
        a.pva[2 * (size_t)r + 1] = v;
    }
}

// dt V_i / m_i V_j (kappa_i + kappa_j) g_ij of a pair.  Boundary kappa is 0 (kappa_div zeroed;
// kappa_incomp never written for boundary); the packed row's w is kappa_j for fluid rows (volume
// vol_f) and V_j for boundary rows.
__device__ __forceinline__ float solve_b_factor(bool fj, float w, float d2, float ci, float ki, const DfsphArgs &a) {
    const float Vj = fj ? a.vol_f : w, kj = fj ? w : 0.f;
    const float g = cubic_g(d2, a.k);
    return ci * Vj * (ki + kj) * g;
}

template <int U>
__global__ void __launch_bounds__(256) k_solve_b(DfsphArgs a) {
    const StepDt T = step_dt(a);
    for (uint32_t t = blockIdx.x; t < a.ntiles; t += gridDim.x) {
        const uint4 tile = a.tiles[t];
        const bool skip = a.tile_ran ? a.tile_ran[t] == 0u : (a.state && a.state[tile.z].stopped);
        if (skip || threadIdx.x >= tile.y) continue;
        const uint32_t r = tile.x + threadIdx.x;
        if (halo_ghost(a, r)) continue;
        const float4 p = a.pos[r];
        float4 v = a.vadv[r];
        const float ki = a.kappa[r];
        const uint32_t n = a.ncnt[r];
        const float mi = a.rest_density ? a.rest_density[r] * p.w : a.mass_f;
        const float ci = T.dt * p.w / mi;   // dt V_i / m_i
        const uint32_t *lst = a.nbr + row_index(r, a.shape);
        nbr_loop<U>(lst, n > 0 ? n - 1 : 0, [&](uint32_t j) { return ldg4(a.pk + j); },
                    [&](uint32_t j, const float4 &e) {
                        const float rx = p.x - e.x, ry = p.y - e.y, rz = p.z - e.z;
                        const float s = solve_b_factor(j < a.nf, e.w, dist2(rx, ry, rz), ci, ki, a);
                        v.x = __fmaf_rn(-s, rx, v.x);
                        v.y = __fmaf_rn(-s, ry, v.y);
                        v.z = __fmaf_rn(-s, rz, v.z);
                    });
        a.vadv[r] = v;
        a.pva[2 * (size_t)r + 1] = v;
        halo_each(a, r, [&](const PeerRows &P, uint32_t q) {
            P.vadv[a.halo_vadv][q] = v;
            P.pva[2 * (size_t)q + 1] = v;
        });
    }
}

// solve_b with a team per row: lanes 0..2 carry a velocity component each.
template <int L>
__global__ void __launch_bounds__(kTeamRows * L) k_team_solve_b(DfsphArgs a, uint32_t pieces) {
    __shared__ TeamTerms<4, L> S;   // -s, x_i - x_j
    const StepDt T = step_dt(a);
    const uint32_t t = blockIdx.x / pieces, part = blockIdx.x - t * pieces, l = team_lane<L>();
    const uint4 tile = a.tiles[t];
    if (a.tile_ran ? a.tile_ran[t] == 0u : (a.state && a.state[tile.z].stopped)) return;
    const uint32_t row = part * kTeamRows + team_row<L>(), r = tile.x + row;
    const bool live = row < tile.y && !halo_ghost(a, r);
    float4 p = make_float4(0.f, 0.f, 0.f, 1.f);
    float ki = 0.f, ci = 0.f, v = 0.f;
    uint32_t n = 0;
    if (live) {
        p = a.pos[r];
        ki = a.kappa[r];
        n = a.ncnt[r];
        v = reinterpret_cast<const float *>(a.vadv + r)[l & 3];
        const float mi = a.rest_density ? a.rest_density[r] * p.w : a.mass_f;
        ci = T.dt * p.w / mi;   // dt V_i / m_i
    }
    const float w = v;   // lane 3: the fourth word, kept
    const uint32_t c = l < 3 ? 1 + l : 1;
    team_walk<L, 4>(
        S, a.nbr + ell_index(r, 0, a.shape), n > 0 ? n - 1 : 0, [&](uint32_t j) { return ldg4(a.pk + j); },
        [&](uint32_t j, const float4 &e, float *o) {
            o[1] = p.x - e.x;
            o[2] = p.y - e.y;
            o[3] = p.z - e.z;
            o[0] = -solve_b_factor(j < a.nf, e.w, dist2(o[1], o[2], o[3]), ci, ki, a);
        },
        [&](const float *e) { v = __fmaf_rn(e[0], e[c], v); });
    if (l == 3) v = w;
    if (live && l < 4) {
        reinterpret_cast<float *>(a.vadv + r)[l] = v;
        reinterpret_cast<float *>(a.pva + 2 * (size_t)r + 1)[l] = v;
    }
    if (a.halo) {
        const float4 o = make_float4(team_get<L>(v, 0), team_get<L>(v, 1), team_get<L>(v, 2), team_get<L>(v, 3));
        if (live && l == 0)
            halo_each(a, r, [&](const PeerRows &P, uint32_t q) {
                P.vadv[a.halo_vadv][q] = o;
                P.pva[2 * (size_t)q + 1] = o;
            });
    }
}

// After the divergence solve: the packed rows' second half becomes the
// velocity after apply_pressure_acc (DFSPHCudaImpl.cu:505-521) for fluid
// rows, so the viscosity pass gathers {x_j, v_j} with one 256-bit load; the
// first half still holds x_j from dfsph_solve_pack (positions do not change
// during the solve).
__global__ void k_pressure_pack(DfsphArgs a) {
    const StepDt T = step_dt(a);
    const uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= a.nf) return;
    a.pva[2 * (size_t)r + 1] = pressure_applied(a.vel[r], a.vadv[r], T.inv_dt, T.dt);
}

// Starts `nscenes` solve states and a loop state (called by one block).
__device__ __forceinline__ void reset_solve(SolveState *s, LoopState *loop, int nscenes) {
    for (int i = threadIdx.x; i < nscenes; i += blockDim.x) {
        s[i].iter = 0;
        s[i].stopped = 0;
    }
    if (threadIdx.x == 0) {
        loop->done = 0;
        loop->active = 0;
        loop->running = 1;
        loop->iters = 0;
    }
}

__global__ void k_solve_pack(DfsphArgs a, SolveState *state, LoopState *loop, int nscenes) {
    if (state && blockIdx.x == 0) reset_solve(state, loop, nscenes);
    const uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= a.nf) return;
    const float4 p = a.pos[r];
    a.pva[2 * (size_t)r] = p;
    a.pva[2 * (size_t)r + 1] = a.vadv[r];
    // With peer-store halos a ghost's {x, kappa} row is written only by its owner's solve_a
    // (which may already be storing it: no fence separates this pack from the peers' solve_a).
    if (halo_ghost(a, r)) return;
    a.pk[r] = make_float4(p.x, p.y, p.z, 0.f);
}

__global__ void k_pack_boundary(DfsphArgs a, float4 *pva2) {
    const uint32_t r = a.nf + blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= a.nf + a.nb) return;
    const float4 p = a.pos[r], v = a.vadv[r];
    a.pva[2 * (size_t)r] = pva2[2 * (size_t)r] = p;
    a.pva[2 * (size_t)r + 1] = pva2[2 * (size_t)r + 1] = v;
    a.pk[r] = p;
}

__global__ void k_solve_begin(SolveState *s, LoopState *loop, int nscenes) { reset_solve(s, loop, nscenes); }

// A tile's sum from the sums of its 32-row pieces, in the order a block sum over the tile adds its
// warps (block_sum: halving strides).
__device__ __forceinline__ double tile_sum(const double *__restrict__ part, uint32_t pieces, int stride) {
    double v[8];
#pragma unroll
    for (uint32_t q = 0; q < 8; ++q) v[q] = q < pieces ? part[(size_t)q * stride] : 0.0;
#pragma unroll
    for (uint32_t o = 4; o > 0; o >>= 1)
#pragma unroll
        for (uint32_t q = 0; q < o; ++q) v[q] += v[q + o];
    return v[0];
}

// One block per scene: FP64 residual of the scene from its tiles' partials,
// the stop test, and (last block to finish) the loop condition.
__global__ void __launch_bounds__(1024) k_solve_end(SolveCtl c, const double *__restrict__ partials,
                                                   uint32_t *status) {
    SolveState *st = c.state + blockIdx.x;
    const SceneTiles sct = c.scene_tiles[blockIdx.x];
    __shared__ uint32_t was_stopped;
    if (threadIdx.x == 0) was_stopped = st->stopped;
    __syncthreads();
    bool active = false;
    if (!was_stopped) {
        double acc = 0.0;
        for (uint32_t o = 0; o < sct.nobj; ++o) {
            // Each thread adds the tiles b = tid, tid + blockDim, ... in that order; the loads of
            // several tiles are issued together so that their latencies overlap.
            double s = 0.0;
            const uint32_t np = c.pieces;
            if (np == 1u) {
                for (uint32_t b = threadIdx.x; b < sct.ntiles; b += 8u * blockDim.x) {
                    double v[8];
#pragma unroll
                    for (uint32_t u = 0; u < 8; ++u) {
                        const uint32_t bb = b + u * blockDim.x;
                        v[u] = bb < sct.ntiles ? partials[(size_t)(sct.tile0 + bb) * c.nobj_max + o] : 0.0;
                    }
#pragma unroll
                    for (uint32_t u = 0; u < 8; ++u)
                        if (b + u * blockDim.x < sct.ntiles) s += v[u];
                }
            } else {   // the passes with a team per row leave a partial per 32 rows of a tile
                for (uint32_t b = threadIdx.x; b < sct.ntiles; b += blockDim.x)
                    s += tile_sum(partials + (size_t)(sct.tile0 + b) * np * c.nobj_max + o, np, c.nobj_max);
            }
            s = block_sum(s);
            if (threadIdx.x == 0) acc += s * c.inv_count[sct.obj0 + o];
        }
        if (threadIdx.x == 0) {
            const double residual = sct.nobj ? acc / (double)sct.nobj : 0.0;
            const uint32_t iter = st->iter + 1;
            st->iter = iter;
            st->residual = residual;
            uint32_t force = c.force_iters;
            if (c.force_seq && c.tick) {
                const uint64_t t = *c.tick;
                if (t < c.force_seq_len) force = c.force_seq[2 * t + c.which];
            }
            bool stop;
            if (force > 0) stop = iter >= force;
            else stop = (residual < (double)c.threshold) || iter > c.max_iters - 1;
            if (!(residual == residual)) {  // NaN residual: stop and flag
                stop = true;
                atomicOr(status, ST_NAN);
            }
            st->stopped = stop ? 1u : 0u;
            if (stop) {
                st->last_iters = iter;
                st->total_iters += iter;
                // vfsph_div / vfsph_incomp flag a crash whenever the loop ran past 100 iterations.
                if (force == 0 && iter > c.max_iters - 1) atomicOr(status, ST_NOT_CONVERGED);
            }
            active = !stop;
        }
    }
    if (threadIdx.x != 0) return;
    if (active) atomicAdd(&c.loop->active, 1u);
    __threadfence();
    const uint32_t prev = atomicAdd(&c.loop->done, 1u);
    if (prev + 1 == gridDim.x) {
        __threadfence();
        const uint32_t act = atomicAdd(&c.loop->active, 0u);
        c.loop->done = 0;
        c.loop->active = 0;
        c.loop->iters += 1;
        c.loop->total += 1;
        c.loop->running = act ? 1u : 0u;
        if (c.use_cond) cudaGraphSetConditional(c.cond, act ? 1u : 0u);
    }
}

// Gravity and the viscosity sum a* of row r (velocity vi after the pressure step): the new velocity,
// or (surface tension on) the acceleration and the normal n* for the tension pass.
template <bool TENSION_SPLIT>
__device__ __forceinline__ void finish_viscosity(const DfsphArgs &a, const StepDt &T, uint32_t r, const float4 &vi,
                                                 float ax, float ay, float az, float nx, float ny, float nz) {
    const SceneGrid &sg = a.sc.sg[a.sc.row_scene[r]];
    const float accx = sg.grav_x + ax, accy = sg.grav_y + ay, accz = sg.grav_z + az;
    if (TENSION_SPLIT) {
        a.acc_tmp[r] = make_float4(accx, accy, accz, 0.f);
        const float4 nrm = make_float4(nx, ny, nz, 0.f);
        a.normal[r] = nrm;
        halo_each(a, r, [&](const PeerRows &P, uint32_t q) { P.normal[q] = nrm; });
        return;
    }
    float4 o = vi;
    o.x = __fmaf_rn(accx, T.dt, vi.x);
    o.y = __fmaf_rn(accy, T.dt, vi.y);
    o.z = __fmaf_rn(accz, T.dt, vi.z);
    a.vel_alt[r] = o;
    a.vadv_alt[r] = o;
    if (a.pack) pack_row(a, r, a.pos[r], o);
    halo_each(a, r, [&](const PeerRows &P, uint32_t q) {
        P.vel[a.halo_vel ^ 1][q] = o;
        P.vadv[a.halo_vadv ^ 1][q] = o;
    });
}

// The tension acceleration of row r added to what the viscosity pass kept: the new velocity.
__device__ __forceinline__ void finish_tension(const DfsphArgs &a, const StepDt &T, uint32_t r, float tx, float ty,
                                               float tz) {
    const float4 vi = pressure_applied(a.vel[r], a.vadv[r], T.inv_dt, T.dt);
    const float4 acc = a.acc_tmp[r];
    float4 o = vi;
    o.x = __fmaf_rn(acc.x + tx, T.dt, vi.x);
    o.y = __fmaf_rn(acc.y + ty, T.dt, vi.y);
    o.z = __fmaf_rn(acc.z + tz, T.dt, vi.z);
    a.vel_alt[r] = o;
    a.vadv_alt[r] = o;
    if (a.pack) pack_row(a, r, a.pos[r], o);
    halo_each(a, r, [&](const PeerRows &P, uint32_t q) {
        P.vel[a.halo_vel ^ 1][q] = o;
        P.vadv[a.halo_vadv ^ 1][q] = o;
    });
}

// Cohesion and normal difference of a pair of fluid rows.
__device__ __forceinline__ void tension_term(const DfsphArgs &a, const float4 &p, const float4 &ni, const PN &e, float &x,
                                             float &y, float &z) {
    const float c1 = -a.gamma * a.mass_f * a.mass_f;
    const float c2 = -a.gamma * a.mass_f;
    const float rx = p.x - e.q.x, ry = p.y - e.q.y, rz = p.z - e.q.z;
    const float rl = sqrtf(dist2(rx, ry, rz));
    const float cs = c1 * tension_c(rl, a.k.h, a.csigma, a.h6_64) / rl;
    x = cs * rx + c2 * (ni.x - e.n.x);
    y = cs * ry + c2 * (ni.y - e.n.y);
    z = cs * rz + c2 * (ni.z - e.n.z);
}

template <bool TENSION_SPLIT, int U>
__global__ void __launch_bounds__(256) k_viscosity(DfsphArgs a) {
    const StepDt T = step_dt(a);
    const uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= a.nf || halo_ghost(a, r)) return;
    const float4 p = a.pos[r];
    const float4 vi = pressure_applied(a.vel[r], a.vadv[r], T.inv_dt, T.dt);
    const uint32_t n = a.ncnt[r];
    float ax = 0.f, ay = 0.f, az = 0.f;
    float nx = 0.f, ny = 0.f, nz = 0.f;
    const float ncoef = a.k.h * a.mass_f / a.rho0;   // h m_j / rho_rest_j (fluid)
    const uint32_t *lst = a.nbr + row_index(r, a.shape);
    nbr_loop<U>(lst, n > 0 ? n - 1 : 0,
                [&](uint32_t j) {
                    if (j >= a.nf) return F4x2{};   // same-material neighbours only
                    return ldg8(a.pva + 2 * (size_t)j);   // {x_j, v_j after the pressure step}
                },
                [&](uint32_t j, const F4x2 &e) {
                    const bool fj = j < a.nf;   // a boundary neighbour adds nothing (1M rows: 109 -> 107 us)
                    const float rx = p.x - e.a.x, ry = p.y - e.a.y, rz = p.z - e.a.z;
                    const float d2 = dist2(rx, ry, rz);
                    const float g = cubic_g(d2, a.k);
                    const float4 vj = e.b;
                    const float vx = vi.x - vj.x, vy = vi.y - vj.y, vz = vi.z - vj.z;
                    const float pi = a.vis_coef * (vx * rx + vy * ry + vz * rz) / (d2 + a.h2_001);
                    const float s = 10.f * pi * g;
                    ax = fj ? __fmaf_rn(s, rx, ax) : ax;
                    ay = fj ? __fmaf_rn(s, ry, ay) : ay;
                    az = fj ? __fmaf_rn(s, rz, az) : az;
                    if (TENSION_SPLIT) {
                        const float sn = ncoef * g;
                        nx = fj ? __fmaf_rn(sn, rx, nx) : nx;
                        ny = fj ? __fmaf_rn(sn, ry, ny) : ny;
                        nz = fj ? __fmaf_rn(sn, rz, nz) : nz;
                    }
                });
    finish_viscosity<TENSION_SPLIT>(a, T, r, vi, ax, ay, az, nx, ny, nz);
}

template <int U>
__global__ void __launch_bounds__(256) k_tension(DfsphArgs a) {
    const StepDt T = step_dt(a);
    const uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= a.nf || halo_ghost(a, r)) return;
    const float4 p = a.pos[r];
    const float4 ni = a.normal[r];
    const uint32_t n = a.ncnt[r];
    // Fluid rest densities are equal, so k = 2 rho_i / (rho_i + rho_j) is evaluated once.
    const float kk = 2.f * a.rho0 / (a.rho0 + a.rho0);
    float tx = 0.f, ty = 0.f, tz = 0.f;
    const uint32_t *lst = a.nbr + row_index(r, a.shape);
    nbr_loop<U>(lst, n > 0 ? n - 1 : 0,
                [&](uint32_t j) {
                    if (j >= a.nf) return PN{};
                    return PN{ldg4(a.pos + j), ldg4(a.normal + j)};
                },
                [&](uint32_t j, const PN &e) {
                    const bool fj = j < a.nf;
                    float x, y, z;
                    tension_term(a, p, ni, e, x, y, z);
                    tx = fj ? tx + kk * x : tx;
                    ty = fj ? ty + kk * y : ty;
                    tz = fj ? tz + kk * z : tz;
                });
    finish_tension(a, T, r, tx, ty, tz);
}

// The viscosity and tension passes with a team per row.
template <bool TENSION_SPLIT, int L>
__global__ void __launch_bounds__(kTeamRows * L) k_team_viscosity(DfsphArgs a) {
    constexpr int W = TENSION_SPLIT ? 8 : 4;
    __shared__ TeamTerms<W, L> S;   // viscosity factor, x_i - x_j, normal factor
    const StepDt T = step_dt(a);
    const uint32_t r = blockIdx.x * kTeamRows + team_row<L>(), l = team_lane<L>();
    const bool live = r < a.nf && !halo_ghost(a, r);
    float4 p = make_float4(0.f, 0.f, 0.f, 0.f), vi = p;
    uint32_t n = 0;
    if (live) {
        p = a.pos[r];
        vi = pressure_applied(a.vel[r], a.vadv[r], T.inv_dt, T.dt);
        n = a.ncnt[r];
    }
    const float ncoef = a.k.h * a.mass_f / a.rho0;   // h m_j / rho_rest_j (fluid)
    float acc = 0.f, nrm = 0.f;
    const uint32_t c = l < 3 ? 1 + l : 1;
    team_walk<L, W>(
        S, a.nbr + ell_index(r, 0, a.shape), n > 0 ? n - 1 : 0,
        [&](uint32_t j) {
            if (j >= a.nf) return F4x2{};   // same-material neighbours only
            return ldg8(a.pva + 2 * (size_t)j);
        },
        [&](uint32_t j, const F4x2 &e, float *o) {
            const float rx = p.x - e.a.x, ry = p.y - e.a.y, rz = p.z - e.a.z;
            const float d2 = dist2(rx, ry, rz);
            const float g = cubic_g(d2, a.k);
            const float4 vj = e.b;
            const float vx = vi.x - vj.x, vy = vi.y - vj.y, vz = vi.z - vj.z;
            const float pi = a.vis_coef * (vx * rx + vy * ry + vz * rz) / (d2 + a.h2_001);
            const bool fluid = j < a.nf;   // a boundary neighbour adds nothing
            o[0] = fluid ? 10.f * pi * g : 0.f;
            o[1] = rx;
            o[2] = ry;
            o[3] = rz;
            if constexpr (TENSION_SPLIT) {
                o[4] = fluid ? ncoef * g : 0.f;
                o[5] = o[6] = o[7] = 0.f;
            }
        },
        [&](const float *e) {
            acc = __fmaf_rn(e[0], e[c], acc);
            if constexpr (TENSION_SPLIT) nrm = __fmaf_rn(e[4], e[c], nrm);
        });
    const float ax = team_get<L>(acc, 0), ay = team_get<L>(acc, 1), az = team_get<L>(acc, 2);
    const float nx = team_get<L>(nrm, 0), ny = team_get<L>(nrm, 1), nz = team_get<L>(nrm, 2);
    if (!live || l != 0) return;
    finish_viscosity<TENSION_SPLIT>(a, T, r, vi, ax, ay, az, nx, ny, nz);
}

template <int L>
__global__ void __launch_bounds__(kTeamRows * L) k_team_tension(DfsphArgs a) {
    __shared__ TeamTerms<4, L> S;
    const StepDt T = step_dt(a);
    const uint32_t r = blockIdx.x * kTeamRows + team_row<L>(), l = team_lane<L>();
    const bool live = r < a.nf && !halo_ghost(a, r);
    float4 p = make_float4(0.f, 0.f, 0.f, 0.f), ni = p;
    uint32_t n = 0;
    if (live) {
        p = a.pos[r];
        ni = a.normal[r];
        n = a.ncnt[r];
    }
    const float kk = 2.f * a.rho0 / (a.rho0 + a.rho0);
    float acc = 0.f;
    team_walk<L, 4>(
        S, a.nbr + ell_index(r, 0, a.shape), n > 0 ? n - 1 : 0,
        [&](uint32_t j) {
            if (j >= a.nf) return PN{};
            return PN{ldg4(a.pos + j), ldg4(a.normal + j)};
        },
        [&](uint32_t j, const PN &e, float *o) {
            o[0] = o[1] = o[2] = o[3] = 0.f;
            if (j < a.nf) tension_term(a, p, ni, e, o[0], o[1], o[2]);
        },
        [&](const float *e) { acc += kk * e[l & 3]; });
    const float tx = team_get<L>(acc, 0), ty = team_get<L>(acc, 1), tz = team_get<L>(acc, 2);
    if (live && l == 0) finish_tension(a, T, r, tx, ty, tz);
}

__global__ void __launch_bounds__(256) k_finalize(DfsphArgs a) {
    const StepDt T = step_dt(a);
    const uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
    float v2 = 0.f;
    if (r < a.nf && !halo_ghost(a, r)) {
        const float4 v = pressure_applied(a.vel[r], a.vadv[r], T.inv_dt, T.dt);
        a.vel[r] = v;
        a.vadv[r] = v;
        if (r == 0 && a.tick) *a.tick += 1;
        float4 p = a.pos[r];
        p.x = __fmaf_rn(v.x, T.dt, p.x);
        p.y = __fmaf_rn(v.y, T.dt, p.y);
        p.z = __fmaf_rn(v.z, T.dt, p.z);
        a.pos[r] = p;
        v2 = dist2(v.x, v.y, v.z);
    }
    if (a.vmax_bits) {   // adaptive step: max |v|^2 of the new velocities for the next substep
        __shared__ uint32_t wmax[8];
        uint32_t b = __reduce_max_sync(0xffffffffu, __float_as_uint(v2));
        if ((threadIdx.x & 31u) == 0) wmax[threadIdx.x >> 5] = b;
        __syncthreads();
        if (threadIdx.x < 32) {
            b = threadIdx.x < (blockDim.x >> 5) ? wmax[threadIdx.x] : 0u;
            b = __reduce_max_sync(0xffffffffu, b);
            if (threadIdx.x == 0 && b) atomicMax(a.vmax_bits, b);   // one atomic per block
        }
    }
}

// Largest |v|^2 over the fluid rows, folded into *vmax_bits (non-negative floats order like
// their bit patterns, so an unsigned atomicMax is a float max).
__global__ void __launch_bounds__(256) k_cfl_max(DfsphArgs a, uint32_t *vmax_bits) {
    float m = 0.f;
    for (uint32_t r = blockIdx.x * blockDim.x + threadIdx.x; r < a.nf; r += gridDim.x * blockDim.x) {
        const float4 v = a.vel[r];
        m = fmaxf(m, dist2(v.x, v.y, v.z));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31u) == 0 && m > 0.f) atomicMax(vmax_bits, __float_as_uint(m));
}

// dt = min(dt_max, cfl * diameter / vmax); the scratch word is cleared for the next substep.
// A step below dt_max * 1e-4 (velocities that have blown up) is held at that floor.
__global__ void k_cfl_step(uint32_t *vmax_bits, float cfl, float diameter, float dt_max, float *dtp,
                           float *sim_time) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    const float vmax = sqrtf(__uint_as_float(*vmax_bits));
    *vmax_bits = 0u;
    float dt = dt_max;
    if (vmax > 0.f) dt = fmaxf(fminf(dt_max, cfl * diameter / vmax), dt_max * 1e-4f);
    *dtp = dt;
    *sim_time += dt;
}

inline unsigned nblk(uint32_t n, int b) { return (unsigned)((n + b - 1) / b); }

}  // namespace

unsigned dfsph_tile_grid(uint32_t ntiles, int block, bool persistent) {
    if (ntiles == 0) return 1u;
    if (!persistent) return ntiles;
    static int sms = 0;
    if (sms == 0) {
        int dev = 0;
        cudaGetDevice(&dev);
        if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0) sms = 148;
    }
    const uint32_t resident = (uint32_t)sms * (uint32_t)(2048 / block);
    return ntiles < resident ? ntiles : resident;
}

void dfsph_rigid_volume(cudaStream_t st, const DfsphArgs &a, const uint32_t *bncnt, const uint32_t *bnbr,
                        float *rest_density_b) {
    if (a.nb) k_rigid_volume<<<nblk(a.nb, 256), 256, 0, st>>>(a, bncnt, bnbr, rest_density_b);
}
#define VTP_TEAM_DISPATCH(L, ...)                \
    {                                            \
        if ((L) == 8) { constexpr int LL = 8; __VA_ARGS__ } \
        else { constexpr int LL = 4; __VA_ARGS__ }          \
    }
#define VTP_UNROLL_DISPATCH(U, ...)          \
    switch (U) {                                 \
        case 1: { constexpr int UU = 1; __VA_ARGS__; } break; \
        case 2: { constexpr int UU = 2; __VA_ARGS__; } break; \
        case 8: { constexpr int UU = 8; __VA_ARGS__; } break; \
        default: { constexpr int UU = 4; __VA_ARGS__; } break; \
    }

void dfsph_ratio_alpha(cudaStream_t st, const DfsphArgs &a, int block) {
    if (!a.nf) return;
    if (a.teams) VTP_TEAM_DISPATCH(a.teams, k_team_ratio_alpha<LL><<<nblk(a.nf, kTeamRows), kTeamRows * LL, 0, st>>>(a);)
    else VTP_UNROLL_DISPATCH(a.unroll, k_ratio_alpha<UU><<<nblk(a.nf, block), block, 0, st>>>(a))
}
void dfsph_solve_begin(cudaStream_t st, SolveState *s, LoopState *loop, int nscenes) {
    k_solve_begin<<<1, 256, 0, st>>>(s, loop, nscenes);
}
void dfsph_solve_pack(cudaStream_t st, const DfsphArgs &a, SolveState *state, LoopState *loop, int nscenes) {
    if (a.nf || state) k_solve_pack<<<nblk(std::max(a.nf, 1u), 256), 256, 0, st>>>(a, state, loop, nscenes);
}
void dfsph_pack_boundary(cudaStream_t st, const DfsphArgs &a, float4 *pva2) {
    if (a.nb) k_pack_boundary<<<nblk(a.nb, 256), 256, 0, st>>>(a, pva2);
}
template <class K>
static void launch_staged(K kern, cudaStream_t st, const DfsphArgs &a, size_t row_bytes) {
    const size_t smem = (size_t)a.stg.scap * row_bytes;
    // the staged rows may exceed the 48 KB of dynamic shared memory a kernel gets by default
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    kern<<<a.stg.ngroups + 1, kStageBlock, smem, st>>>(a);
}

void dfsph_solve_a(cudaStream_t st, const DfsphArgs &a, int block) {
    if (a.staged) {
        if (a.nobj_max > 1) VTP_UNROLL_DISPATCH(a.unroll, launch_staged(k_solve_a_staged<true, UU>, st, a, 32))
        else VTP_UNROLL_DISPATCH(a.unroll, launch_staged(k_solve_a_staged<false, UU>, st, a, 32))
        return;
    }
    if (a.teams) {
        const uint32_t pieces = solve_pieces(block), n = a.ntiles * pieces;
        if (!n) return;
        if (a.nobj_max > 1) VTP_TEAM_DISPATCH(a.teams, k_team_solve_a<true, LL><<<n, kTeamRows * LL, 0, st>>>(a, pieces);)
        else VTP_TEAM_DISPATCH(a.teams, k_team_solve_a<false, LL><<<n, kTeamRows * LL, 0, st>>>(a, pieces);)
        return;
    }
    const unsigned nb = dfsph_tile_grid(a.ntiles, block, a.persistent);
    if (a.nobj_max > 1) VTP_UNROLL_DISPATCH(a.unroll, k_solve_a<true, UU><<<nb, block, 0, st>>>(a))
    else VTP_UNROLL_DISPATCH(a.unroll, k_solve_a<false, UU><<<nb, block, 0, st>>>(a))
}
void dfsph_solve_b(cudaStream_t st, const DfsphArgs &a, int block) {
    if (a.staged) {
        VTP_UNROLL_DISPATCH(a.unroll, launch_staged(k_solve_b_staged<UU>, st, a, 16))
        return;
    }
    if (a.teams) {
        const uint32_t pieces = solve_pieces(block), n = a.ntiles * pieces;
        if (n) VTP_TEAM_DISPATCH(a.teams, k_team_solve_b<LL><<<n, kTeamRows * LL, 0, st>>>(a, pieces);)
        return;
    }
    const unsigned nb = dfsph_tile_grid(a.ntiles, block, a.persistent);
    VTP_UNROLL_DISPATCH(a.unroll, k_solve_b<UU><<<nb, block, 0, st>>>(a))
}
void dfsph_solve_end(cudaStream_t st, const SolveCtl &c, const double *partials, uint32_t *status) {
    k_solve_end<<<c.nscenes, 1024, 0, st>>>(c, partials, status);
}
void dfsph_cfl_step(cudaStream_t st, float cfl, float diameter, float dt_max, uint32_t *vmax_bits, float *dtp,
                    float *sim_time) {
    k_cfl_step<<<1, 32, 0, st>>>(vmax_bits, cfl, diameter, dt_max, dtp, sim_time);
}
void dfsph_cfl_refresh(cudaStream_t st, const DfsphArgs &a, uint32_t *vmax_bits) {
    cudaMemsetAsync(vmax_bits, 0, sizeof(uint32_t), st);
    if (a.nf) {
        const unsigned g = std::min<unsigned>(nblk(a.nf, 256), 148u * 8u);
        k_cfl_max<<<g, 256, 0, st>>>(a, vmax_bits);
    }
}
void dfsph_pressure_pack(cudaStream_t st, const DfsphArgs &a) {
    if (a.nf) k_pressure_pack<<<nblk(a.nf, 256), 256, 0, st>>>(a);
}
void dfsph_viscosity(cudaStream_t st, const DfsphArgs &a, int block) {
    if (!a.nf) return;
    if (a.teams) VTP_TEAM_DISPATCH(a.teams, k_team_viscosity<false, LL><<<nblk(a.nf, kTeamRows), kTeamRows * LL, 0, st>>>(a);)
    else VTP_UNROLL_DISPATCH(a.unroll, k_viscosity<false, UU><<<nblk(a.nf, block), block, 0, st>>>(a))
}
void dfsph_vis_normal(cudaStream_t st, const DfsphArgs &a, int block) {
    if (!a.nf) return;
    if (a.teams) VTP_TEAM_DISPATCH(a.teams, k_team_viscosity<true, LL><<<nblk(a.nf, kTeamRows), kTeamRows * LL, 0, st>>>(a);)
    else VTP_UNROLL_DISPATCH(a.unroll, k_viscosity<true, UU><<<nblk(a.nf, block), block, 0, st>>>(a))
}
void dfsph_tension(cudaStream_t st, const DfsphArgs &a, int block) {
    if (!a.nf) return;
    if (a.teams) VTP_TEAM_DISPATCH(a.teams, k_team_tension<LL><<<nblk(a.nf, kTeamRows), kTeamRows * LL, 0, st>>>(a);)
    else VTP_UNROLL_DISPATCH(a.unroll, k_tension<UU><<<nblk(a.nf, block), block, 0, st>>>(a))
}
void dfsph_finalize(cudaStream_t st, const DfsphArgs &a) {
    if (a.nf) k_finalize<<<nblk(a.nf, 256), 256, 0, st>>>(a);
}

}  // namespace vtp
