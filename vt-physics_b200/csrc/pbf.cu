// PBF solver passes for sm_100a (fluid rows only; rows are cell-sorted).
//
// Restates the reference's PBF substep (PBFSolver::tick, PBFSolver.cpp:326-376)
// with the kernels of PBFCudaImpl.cu:34-194 regrouped:
//   lambda pass  = compute_sph_density_and_error_cuda + update_lamb_cuda (:70-122)
//   dx pass      = compute_dx_cuda + apply_dx_cuda (:124-170), positions
//                  written to the second buffer so the pass stays Jacobi
//   xsph pass    = XSPH_cuda + apply_dx_cuda (:172-194, :267-281)
// apply_ext_force_cuda (:146-157) is fused into the neighbour-search sort.
#include "pbf.h"
#include "team.cuh"

namespace vtp {

namespace {

// Standard-PBF kernels (form 1): poly6 density, spiky gradient (gradW = g r).  The range is selected
// after the arithmetic, so that the pairs in flight overlap (250k rows, a call of four substeps:
// 1530 -> 1485 us).
__device__ __forceinline__ float poly6_w(float d2, const PbfArgs &a) {
    const float d = a.h2 - d2;
    const float w = a.c6 * d * d * d;
    return d2 > a.h2 ? 0.f : w;
}
__device__ __forceinline__ float spiky_g(float d2, const PbfArgs &a) {
    const float r = sqrtf(d2);
    const float d = a.k.h - r;
    const float g = a.cs * d * d / r;
    return !(d2 > 0.f) || r < 1e-6f * a.k.h || r > a.k.h ? 0.f : g;
}
__device__ __forceinline__ float pbf_w(float d2, const PbfArgs &a) {
    return a.form ? poly6_w(d2, a) : cubic_w(d2, a.k);
}
__device__ __forceinline__ float pbf_w0(const PbfArgs &a) { return a.form ? a.c6 * a.h2 * a.h2 * a.h2 : a.k.w0; }

__global__ void __launch_bounds__(256) k_pbf_init_boundary(PbfArgs a, const uint32_t *__restrict__ bncnt,
                                                           const uint32_t *__restrict__ bnbr,
                                                           ListShape shape) {
    // compute_rigid_particle_volume_cuda (PBFCudaImpl.cu:47-68): V_b = 1 / sum_{boundary j} W_ij
    // (self included), m_b = rho_b V_b.  Only boundary neighbours count.
    uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= a.nb) return;
    uint32_t i = a.nf + r;
    float4 p = a.pos[i];
    uint32_t n = bncnt[r];
    float delta = n > 0 ? pbf_w0(a) : 0.f;
    const uint32_t *lst = bnbr + ell_index(r, 0, shape);
    for (uint32_t t = 0; t + 1 < n; ++t) {
        uint32_t j = lst[ell_slot(t, shape)];
        if (j < a.nf) continue;
        float4 q = a.pos[j];
        delta += pbf_w(dist2(p.x - q.x, p.y - q.y, p.z - q.z), a);
    }
    float vb = 1.f / delta;
    a.vol[i] = vb;
    float mb = a.rho_b * vb;
    p.w = mb;
    a.pos[i] = p;
    a.pos_alt[i] = p;
}

struct PL {
    float4 q;
    float l;
};
struct PV2 {
    float4 q, v;
    float vol;
};

// W, g (times the mass in the standard form) and x_i - x_j of a pair of the lambda pass.
struct LambdaPair {
    float dx, dy, dz, w, g;
};
__device__ __forceinline__ LambdaPair lambda_pair(const PbfArgs &a, const float4 &p, const float4 &q) {
    LambdaPair t;
    t.dx = p.x - q.x; t.dy = p.y - q.y; t.dz = p.z - q.z;
    const float d2 = dist2(t.dx, t.dy, t.dz);
    if (a.form == 0) {
        cubic_wg(d2, a.k, t.w, t.g);
    } else {
        t.w = poly6_w(d2, a);
        t.g = spiky_g(d2, a) * q.w;   // mass-weighted constraint gradient
    }
    return t;
}
// Density, and lambda from the gradient sums, of row r.
__device__ __forceinline__ void finish_lambda(const PbfArgs &a, uint32_t r, float rho, float gx, float gy, float gz,
                                              float s2) {
    if (rho < a.rho0) rho = a.rho0;
    const float err = rho / a.rho0 - 1.f;
    gx /= a.rho0; gy /= a.rho0; gz /= a.rho0;
    s2 += gx * gx + gy * gy + gz * gz;
    a.density[r] = rho;
    const float lam = -err / (s2 + a.eps);
    a.lambda[r] = lam;
    halo_each(a, r, [&](const PeerRows &P, uint32_t q) { P.lambda[q] = lam; });
}

// (lambda_i + lambda_j) g, or (lambda_i m_j + lambda_j m_i) g in the standard form, of a pair.  Which
// of the two products is fused is fixed here: the compiler chose differently in the passes that inline it.
__device__ __forceinline__ float dx_factor(const PbfArgs &a, float d2, float mi, float mj, float li, float lj) {
    if (a.form == 0) return (li + lj) * cubic_g(d2, a.k);
    return __fmaf_rn(li, mj, __fmul_rn(lj, mi)) * spiky_g(d2, a);
}
// The correction sum applied to row r: position (second buffer) and velocity.
__device__ __forceinline__ void finish_dx(const PbfArgs &a, uint32_t r, const float4 &p, float dx, float dy, float dz) {
    dx /= a.rho0; dy /= a.rho0; dz /= a.rho0;
    float4 o = p;
    o.x += dx; o.y += dy; o.z += dz;
    a.pos_alt[r] = o;
    float4 v = a.vel[r];
    v.x += dx / a.dt; v.y += dy / a.dt; v.z += dz / a.dt;
    a.vel[r] = v;
    halo_each(a, r, [&](const PeerRows &P, uint32_t q) {
        P.pos[a.halo_pos ^ 1][q] = o;   // the peer's second buffer, current after its swap
        P.vel[a.halo_vel][q] = v;
    });
}

// The XSPH sum applied to row r: position and velocity (second buffers).
__device__ __forceinline__ void finish_xsph(const PbfArgs &a, uint32_t r, const float4 &p, const float4 &vi, float ax,
                                            float ay, float az) {
    const float dx = ax * a.dt, dy = ay * a.dt, dz = az * a.dt;
    float4 o = p;
    o.x += dx; o.y += dy; o.z += dz;
    a.pos_alt[r] = o;
    float4 v = vi;
    v.x += dx / a.dt; v.y += dy / a.dt; v.z += dz / a.dt;
    a.vel_alt[r] = v;
}

// One thread per row reads lists of shape lg 0; lanes per row ("rowLanes") read either shape.
template <int U, int L, class Load, class Use>
__device__ __forceinline__ void row_loop(const PbfArgs &a, const uint32_t *lst, uint32_t cnt, int lane, Load load,
                                         Use use) {
    if constexpr (L == 1) nbr_loop<U>(lst, cnt, load, use);
    else nbr_loop_lanes<U, L>(lst, a.shape, cnt, lane, load, use);
}

// Neighbour passes, U list entries in flight per thread and L lanes per row
// (L = 1: one thread walks the row's list in order; L > 1: the row's lanes
// take entries lane, lane + L, ... and their partial sums are added by a
// butterfly over the group, so a small scene keeps more of the GPU busy; the
// FP32 sums then group differently from the list order).
template <int U, int L>
__global__ void __launch_bounds__(256) k_pbf_lambda(PbfArgs a) {
    pdl_enter();
    const uint32_t gt = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t r = gt / L;
    const int lane = (int)(gt % L);
    if (r >= a.nf || halo_ghost(a, r)) return;   // the same for every lane of the row
    const float4 p = a.pos[r];
    const uint32_t n = a.ncnt[r];
    // Self is the first entry of every list: density gets m_i W(0), gradients 0.
    float rho = (n > 0 && lane == 0) ? p.w * pbf_w0(a) : 0.f;
    float gx = 0.f, gy = 0.f, gz = 0.f, s2 = 0.f;
    const uint32_t *lst = a.nbr + (L == 1 ? row_index(r, a.shape) : ell_index(r, 0, a.shape));
    row_loop<U, L>(a, lst, n > 0 ? n - 1 : 0, lane, [&](uint32_t j) { return ldg4(a.pos + j); },
                         [&](uint32_t, const float4 &q) {
                             const LambdaPair t = lambda_pair(a, p, q);
                             rho = __fmaf_rn(q.w, t.w, rho);
                             const float ex = t.g * t.dx, ey = t.g * t.dy, ez = t.g * t.dz;
                             gx += ex; gy += ey; gz += ez;
                             const float fx = ex * a.inv_rho0, fy = ey * a.inv_rho0, fz = ez * a.inv_rho0;
                             s2 += fx * fx + fy * fy + fz * fz;
                         });
    if constexpr (L > 1) {
        const unsigned m = lane_group_mask<L>();
        rho = lane_sum<L>(rho, m);
        gx = lane_sum<L>(gx, m);
        gy = lane_sum<L>(gy, m);
        gz = lane_sum<L>(gz, m);
        s2 = lane_sum<L>(s2, m);
        if (lane != 0) return;
    }
    finish_lambda(a, r, rho, gx, gy, gz, s2);
}

template <int U, int L>
__global__ void __launch_bounds__(256) k_pbf_dx(PbfArgs a) {
    pdl_enter();
    const uint32_t gt = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t r = gt / L;
    const int lane = (int)(gt % L);
    if (r >= a.nf || halo_ghost(a, r)) return;
    const float4 p = a.pos[r];
    const float li = a.lambda[r];
    const uint32_t n = a.ncnt[r];
    float dx = 0.f, dy = 0.f, dz = 0.f;
    const uint32_t *lst = a.nbr + (L == 1 ? row_index(r, a.shape) : ell_index(r, 0, a.shape));
    // Boundary lambda is never written by the reference; it is taken as 0.
    row_loop<U, L>(a, lst, n > 0 ? n - 1 : 0, lane,
                         [&](uint32_t j) { return PL{ldg4(a.pos + j), j < a.nf ? __ldg(a.lambda + j) : 0.f}; },
                         [&](uint32_t, const PL &e) {
                             const float rx = p.x - e.q.x, ry = p.y - e.q.y, rz = p.z - e.q.z;
                             const float s = dx_factor(a, dist2(rx, ry, rz), p.w, e.q.w, li, e.l);
                             dx = __fmaf_rn(s, rx, dx);
                             dy = __fmaf_rn(s, ry, dy);
                             dz = __fmaf_rn(s, rz, dz);
                         });
    if constexpr (L > 1) {
        const unsigned m = lane_group_mask<L>();
        dx = lane_sum<L>(dx, m);
        dy = lane_sum<L>(dy, m);
        dz = lane_sum<L>(dz, m);
        if (lane != 0) return;
    }
    finish_dx(a, r, p, dx, dy, dz);
}

template <int U, int L>
__global__ void __launch_bounds__(256) k_pbf_xsph(PbfArgs a) {
    pdl_enter();
    const uint32_t gt = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t r = gt / L;
    const int lane = (int)(gt % L);
    if (r >= a.nf || halo_ghost(a, r)) return;
    const float4 p = a.pos[r];
    const float4 vi = a.vel[r];
    const uint32_t n = a.ncnt[r];
    float ax = 0.f, ay = 0.f, az = 0.f;
    const uint32_t *lst = a.nbr + (L == 1 ? row_index(r, a.shape) : ell_index(r, 0, a.shape));
    row_loop<U, L>(a, lst, n > 0 ? n - 1 : 0, lane,
                         [&](uint32_t j) { return PV2{ldg4(a.pos + j), ldg4(a.vel + j), __ldg(a.vol + j)}; },
                         [&](uint32_t, const PV2 &e) {
                             const float w = pbf_w(dist2(p.x - e.q.x, p.y - e.q.y, p.z - e.q.z), a);
                             const float c = a.xsph_k * e.vol;
                             ax = __fmaf_rn(c * (e.v.x - vi.x), w, ax);
                             ay = __fmaf_rn(c * (e.v.y - vi.y), w, ay);
                             az = __fmaf_rn(c * (e.v.z - vi.z), w, az);
                         });
    if constexpr (L > 1) {
        const unsigned m = lane_group_mask<L>();
        ax = lane_sum<L>(ax, m);
        ay = lane_sum<L>(ay, m);
        az = lane_sum<L>(az, m);
        if (lane != 0) return;
    }
    finish_xsph(a, r, p, vi, ax, ay, az);
}

// The passes with a team per row (team.cuh).
template <int L>
__global__ void __launch_bounds__(kTeamRows * L) k_team_pbf_lambda(PbfArgs a) {
    pdl_enter();
    __shared__ TeamTerms<8, L> S;   // m_j, W, gradW, |gradW / rho0|^2
    const uint32_t r = blockIdx.x * kTeamRows + team_row<L>(), l = team_lane<L>();
    const bool live = r < a.nf && !halo_ghost(a, r);
    float4 p = make_float4(0.f, 0.f, 0.f, 0.f);
    uint32_t n = 0;
    if (live) {
        p = a.pos[r];
        n = a.ncnt[r];
    }
    // lane 0: density (self first: m_i W(0)), lanes 1..3: sum of gradients; every lane: s2
    float acc = n > 0 && l == 0 ? p.w * pbf_w0(a) : 0.f, s2 = 0.f;
    team_walk<L, 8>(
        S, a.nbr + ell_index(r, 0, a.shape), n > 0 ? n - 1 : 0, [&](uint32_t j) { return ldg4(a.pos + j); },
        [&](uint32_t, const float4 &q, float *o) {
            const LambdaPair t = lambda_pair(a, p, q);
            const float ex = t.g * t.dx, ey = t.g * t.dy, ez = t.g * t.dz;
            const float fx = ex * a.inv_rho0, fy = ey * a.inv_rho0, fz = ez * a.inv_rho0;
            o[0] = q.w;
            o[1] = t.w;
            o[2] = ex;
            o[3] = ey;
            o[4] = ez;
            o[5] = fx * fx + fy * fy + fz * fz;
            o[6] = 1.f;
            o[7] = 0.f;
        },
        [&](const float *e) {
            acc = __fmaf_rn(e[(l & 3) == 0 ? 0 : 6], e[1 + (l & 3)], acc);
            s2 = __fadd_rn(s2, e[5]);
        });
    const float gx = team_get<L>(acc, 1), gy = team_get<L>(acc, 2), gz = team_get<L>(acc, 3);
    if (live && l == 0) finish_lambda(a, r, acc, gx, gy, gz, s2);
}

template <int L>
__global__ void __launch_bounds__(kTeamRows * L) k_team_pbf_dx(PbfArgs a) {
    pdl_enter();
    __shared__ TeamTerms<4, L> S;   // factor, x_i - x_j
    const uint32_t r = blockIdx.x * kTeamRows + team_row<L>(), l = team_lane<L>();
    const bool live = r < a.nf && !halo_ghost(a, r);
    float4 p = make_float4(0.f, 0.f, 0.f, 0.f);
    float li = 0.f;
    uint32_t n = 0;
    if (live) {
        p = a.pos[r];
        li = a.lambda[r];
        n = a.ncnt[r];
    }
    float acc = 0.f;
    const uint32_t c = l < 3 ? 1 + l : 1;
    // Boundary lambda is never written by the reference; it is taken as 0.
    team_walk<L, 4>(
        S, a.nbr + ell_index(r, 0, a.shape), n > 0 ? n - 1 : 0,
        [&](uint32_t j) { return PL{ldg4(a.pos + j), j < a.nf ? __ldg(a.lambda + j) : 0.f}; },
        [&](uint32_t, const PL &e, float *o) {
            o[1] = p.x - e.q.x;
            o[2] = p.y - e.q.y;
            o[3] = p.z - e.q.z;
            o[0] = dx_factor(a, dist2(o[1], o[2], o[3]), p.w, e.q.w, li, e.l);
        },
        [&](const float *e) { acc = __fmaf_rn(e[0], e[c], acc); });
    const float dx = team_get<L>(acc, 0), dy = team_get<L>(acc, 1), dz = team_get<L>(acc, 2);
    if (live && l == 0) finish_dx(a, r, p, dx, dy, dz);
}

template <int L>
__global__ void __launch_bounds__(kTeamRows * L) k_team_pbf_xsph(PbfArgs a) {
    pdl_enter();
    __shared__ TeamTerms<4, L> S;   // W, k V_j (v_j - v_i)
    const uint32_t r = blockIdx.x * kTeamRows + team_row<L>(), l = team_lane<L>();
    const bool live = r < a.nf && !halo_ghost(a, r);
    float4 p = make_float4(0.f, 0.f, 0.f, 0.f), vi = p;
    uint32_t n = 0;
    if (live) {
        p = a.pos[r];
        vi = a.vel[r];
        n = a.ncnt[r];
    }
    float acc = 0.f;
    const uint32_t c = l < 3 ? 1 + l : 1;
    team_walk<L, 4>(
        S, a.nbr + ell_index(r, 0, a.shape), n > 0 ? n - 1 : 0,
        [&](uint32_t j) { return PV2{ldg4(a.pos + j), ldg4(a.vel + j), __ldg(a.vol + j)}; },
        [&](uint32_t, const PV2 &e, float *o) {
            const float k = a.xsph_k * e.vol;
            o[0] = pbf_w(dist2(p.x - e.q.x, p.y - e.q.y, p.z - e.q.z), a);
            o[1] = k * (e.v.x - vi.x);
            o[2] = k * (e.v.y - vi.y);
            o[3] = k * (e.v.z - vi.z);
        },
        [&](const float *e) { acc = __fmaf_rn(e[c], e[0], acc); });
    const float ax = team_get<L>(acc, 0), ay = team_get<L>(acc, 1), az = team_get<L>(acc, 2);
    if (live && l == 0) finish_xsph(a, r, p, vi, ax, ay, az);
}

inline unsigned nblk(uint32_t n, int b) { return (unsigned)((n + b - 1) / b); }

}  // namespace

void pbf_init_boundary(cudaStream_t st, const PbfArgs &a, const uint32_t *bncnt, const uint32_t *bnbr,
                       ListShape shape) {
    if (a.nb) k_pbf_init_boundary<<<nblk(a.nb, 256), 256, 0, st>>>(a, bncnt, bnbr, shape);
}
#define VTP_UNROLL_DISPATCH(U, ...)          \
    switch (U) {                                 \
        case 1: { constexpr int UU = 1; __VA_ARGS__; } break; \
        case 2: { constexpr int UU = 2; __VA_ARGS__; } break; \
        case 8: { constexpr int UU = 8; __VA_ARGS__; } break; \
        default: { constexpr int UU = 4; __VA_ARGS__; } break; \
    }
#define VTP_LANES_DISPATCH(L, ...)           \
    switch (L) {                                 \
        case 4: { constexpr int LL = 4; __VA_ARGS__; } break; \
        case 8: { constexpr int LL = 8; __VA_ARGS__; } break; \
        default: { constexpr int LL = 1; __VA_ARGS__; } break; \
    }

void pbf_lambda(cudaStream_t st, const PbfArgs &a, int block) {
    if (!a.nf) return;
    if (a.teams == 8 && a.lanes == 1)
        launch(k_team_pbf_lambda<8>, nblk(a.nf, kTeamRows), kTeamRows * 8, 0, st, a);
    else if (a.teams && a.lanes == 1)
        launch(k_team_pbf_lambda<4>, nblk(a.nf, kTeamRows), kTeamRows * 4, 0, st, a);
    else
        VTP_LANES_DISPATCH(a.lanes, VTP_UNROLL_DISPATCH(a.unroll, launch(k_pbf_lambda<UU, LL>, nblk(a.nf * LL, block), block, 0, st, a)))
}
void pbf_dx(cudaStream_t st, const PbfArgs &a, int block) {
    if (!a.nf) return;
    if (a.teams == 8 && a.lanes == 1)
        launch(k_team_pbf_dx<8>, nblk(a.nf, kTeamRows), kTeamRows * 8, 0, st, a);
    else if (a.teams && a.lanes == 1)
        launch(k_team_pbf_dx<4>, nblk(a.nf, kTeamRows), kTeamRows * 4, 0, st, a);
    else
        VTP_LANES_DISPATCH(a.lanes, VTP_UNROLL_DISPATCH(a.unroll, launch(k_pbf_dx<UU, LL>, nblk(a.nf * LL, block), block, 0, st, a)))
}
void pbf_xsph(cudaStream_t st, const PbfArgs &a, int block) {
    if (!a.nf) return;
    if (a.teams == 8 && a.lanes == 1)
        launch(k_team_pbf_xsph<8>, nblk(a.nf, kTeamRows), kTeamRows * 8, 0, st, a);
    else if (a.teams && a.lanes == 1)
        launch(k_team_pbf_xsph<4>, nblk(a.nf, kTeamRows), kTeamRows * 4, 0, st, a);
    else
        VTP_LANES_DISPATCH(a.lanes, VTP_UNROLL_DISPATCH(a.unroll, launch(k_pbf_xsph<UU, LL>, nblk(a.nf * LL, block), block, 0, st, a)))
}

}  // namespace vtp
