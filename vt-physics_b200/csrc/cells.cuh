// Pieces of the list builders that work a cell at a time (ugns.cu, noalloc.cu): the candidates of
// a cell's 27 neighbour cells laid out in shared memory, and their test against a row in packed
// FP32 arithmetic.
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

struct CellScratch {
    float x[3][kCellWindow];             // candidate positions of the window, in list order
    uint32_t cand[kCellWindow];          // their rows
    uint8_t kept[32][kCellKept];         // each lane's accepted candidates, as offsets into its share
};

// Appends `off` to the lane's accepted candidates at shared address `to` if 0 < d2 <= d2max
// (`0 < |x_i - x_j|` also drops the row itself): predicated, no branch.  The asm names no memory
// clobber, so that the next candidates' loads are not held up by it: what it stores is read only
// after a warp barrier.
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

}  // namespace vtp
