// Device routines shared by the particle, injection and mixed-precision
// kernels: the facet walk, barycentric coordinates and the fixed-point
// deposit.  Every FP64 product and sum is an explicit round-to-nearest
// intrinsic and every FP32 one an explicit fmaf or __f*_rn, so the results do
// not depend on the translation unit's --fmad setting.
#pragma once

#include "pg_device.cuh"

namespace pg {

__device__ __forceinline__ void raise_device_error(DevState *st, int code, int64_t idx) {
    if (atomicCAS(&st->err_code, 0, code) == 0) st->err_index = idx;
}

// c0 + c1 x + c2 y + c3 z summed left to right with each step rounded, as
// relocate_fast evaluates it (punc/include/punc/population.h:549-552).
__device__ __forceinline__ double plane64(double c0, double c1, double c2, double c3, double x, double y, double z) {
    double d = __dadd_rn(c0, __dmul_rn(c1, x));
    d = __dadd_rn(d, __dmul_rn(c2, y));
    return __dadd_rn(d, __dmul_rn(c3, z));
}

// relocate_fast (punc/include/punc/population.h:539-569) as a bounded loop
// (walk_fp64, walk_mixed below): the first facet i (0..3) with a positive
// plane value moves the walk to neighbour i or ends it with -tag; no positive
// facet ends it in the cell.
// Relative bound on |FP32 affine value - exact value| in units of the sum of
// the terms' magnitudes: one rounding per coefficient, coordinate and fmaf
// (at most five), and slack.  The absolute part of the bound is the mesh's
// (DevMesh::lam_abs, the rounding of the FP64 tables).
constexpr float kPlaneEps = 8.0f * 5.9604645e-08f;   // 8 * 2^-24

// Cell record of c: barycentric rows 0-2 in FP32 and the neighbours (int bits).
struct CellRec {
    float4 r0, r1, r2, nb;
};
__device__ __forceinline__ CellRec load_rec(const DevMesh &m, int c) {
    const float4 *R = m.cell_f + 4 * (size_t)c;
    return CellRec{__ldg(R), __ldg(R + 1), __ldg(R + 2), __ldg(R + 3)};
}

// Barycentric coordinates of the FP32 point from a cell record's rows 0-2
// (the fourth is 1 - l0 - l1 - l2) and bounds on their distance from the
// FP64 planes' values over the heights, at the FP32 point and at any FP64
// point that rounds to it.
__device__ __forceinline__ void lambdas_f32(const DevMesh &m, const CellRec &R, float x, float y, float z, float l[4],
                                            float e[4]) {
    const float4 r[3] = {R.r0, R.r1, R.r2};
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        l[k] = fmaf(r[k].w, z, fmaf(r[k].z, y, fmaf(r[k].y, x, r[k].x)));
        e[k] = fmaf(kPlaneEps, fabsf(r[k].x) + fabsf(r[k].y * x) + fabsf(r[k].z * y) + fabsf(r[k].w * z), m.lam_abs);
    }
    l[3] = __fsub_rn(__fsub_rn(__fsub_rn(1.0f, l[0]), l[1]), l[2]);
    e[3] = e[0] + e[1] + e[2] + kPlaneEps * (1.0f + fabsf(l[0]) + fabsf(l[1]) + fabsf(l[2]));
}

// Is the point outside facet f (opposite local vertex f, where lambda_f = 0)?
// Decided from the sign of lambda_f when it exceeds its error bound (lambda_f
// < 0 exactly when the facet's plane value is positive); otherwise re-tested
// in FP64 with the FP64 plane, the exact FP64 predicate at this point.
template <class T>
__device__ __forceinline__ bool facet_positive(const DevMesh &m, int c, int f, float l, float e, T x, T y, T z,
                                               int &retests) {
    if (l < -e) return true;
    if (l > e) return false;
    ++retests;
    const double2 *P = reinterpret_cast<const double2 *>(m.planes) + 8 * (size_t)c + 2 * f;
    const double2 a = __ldg(P), b = __ldg(P + 1);
    return plane64(a.x, a.y, b.x, b.y, (double)x, (double)y, (double)z) > 0;
}

// A cell near the point: the last cell of the point's location bin.
__device__ __forceinline__ int near_cell(const DevMesh &m, float x, float y, float z) {
    const float u[3] = {x, y, z};
    int b[3];
#pragma unroll
    for (int j = 0; j < 3; ++j) {
        const int k = (int)((u[j] - m.lo_f[j]) * m.bin_inv_f[j]);
        b[j] = k < 0 ? 0 : (k >= m.nbin[j] ? m.nbin[j] - 1 : k);
    }
    const int64_t bin = ((int64_t)b[0] * m.nbin[1] + b[1]) * m.nbin[2] + b[2];
    return __ldg(m.bin_cells + __ldg(m.bin_ptr + bin + 1) - 1);
}

// The point lies this many facet heights or more beyond some facet of the
// first cell: a walk of about as many cells.  Periodic moves wrap a particle
// to the other side of the box, which is a walk through every cell between,
// and its warp waits for it (24^3 cells, 663k thermal electrons, CG1 field: the
// FP64 pass 2.44 ms with long walks on FP64 planes, 0.19 ms with the restart,
// the FP32 tests and the warp kept together).
constexpr float kFarLambda = -6.0f;
constexpr int kNearSteps = 256;

// The walk of relocate_fast (walk_fp64) with each facet decided in FP32 where
// its error bound allows, every decision equal to the FP64 predicate at the
// point (T: double or float).  One 64-byte record per cell visited instead of
// 144 bytes, and no FP64 operation outside the bound (a plane test is six, at
// 1/64 of the FP32 rate; the FP64 pass over 1.5M particles at 53^3 cells 525
// us with them, 224 without, then 153 with the warp kept together).  R, have_rec:
// the first cell's record when the caller has it; R and l are the last cell's on
// return.
//
// NEAR: in a box without an inner wall (m.box; set only with a step limit that
// no walk through such a mesh reaches) a walk that starts far from its point
// starts again at a cell near it.  The result counts only if the point lies
// inside its cell by more than the error bounds: that cell is then the only one
// whose four plane values are not positive, the one where the long walk ends
// too.  Otherwise the long walk runs.
template <bool NEAR, class T>
__device__ __forceinline__ int walk_loop(const DevMesh &m, T x, T y, T z, int c, int max_steps, int &retests,
                                         CellRec &R, bool have_rec, float l[4]) {
    float xf = (float)x;
    const float yf = (float)y, zf = (float)z;
    // beyond the range of m.lam_abs (no cell holds such a point) every facet is
    // tested in FP64: the tables' errors grow with the point's distance, and the
    // relative bound does not cover them (a coefficient that should be zero is
    // 1e-17 in one FP64 table and zero in the other: at 1e12 boxes the term is
    // larger than the rounding of those that count)
    if (!(m.lam_inv_range * fmaxf(fabsf(xf), fmaxf(fabsf(yf), fabsf(zf))) <= 1.0f)) xf = nanf("");
    int cc = c;
    bool near_walk = false, may_restart = NEAR;
    for (int it = 0; it < max_steps; ++it) {
        float e[4];
        if (!have_rec) R = load_rec(m, cc);
        have_rec = false;
        lambdas_f32(m, R, xf, yf, zf, l, e);
        if (NEAR && may_restart && fminf(fminf(l[0], l[1]), fminf(l[2], l[3])) < kFarLambda) {
            cc = near_cell(m, xf, yf, zf);
            near_walk = true;
            may_restart = false;
            continue;
        }
        may_restart = false;
        int next;
        bool stay = false;
        if (facet_positive(m, cc, 0, l[0], e[0], x, y, z, retests)) next = __float_as_int(R.nb.x);
        else if (facet_positive(m, cc, 1, l[1], e[1], x, y, z, retests)) next = __float_as_int(R.nb.y);
        else if (facet_positive(m, cc, 2, l[2], e[2], x, y, z, retests)) next = __float_as_int(R.nb.z);
        else if (facet_positive(m, cc, 3, l[3], e[3], x, y, z, retests)) next = __float_as_int(R.nb.w);
        else { next = cc; stay = true; }
        if (NEAR && near_walk) {
            const bool sure = stay && l[0] > e[0] && l[1] > e[1] && l[2] > e[2] && l[3] > e[3];
            if (sure) return cc;
            if (stay || next < 0 || it >= kNearSteps) {
                near_walk = false;
                cc = c;
                it = -1;
                continue;
            }
        } else {
            if (stay) return cc;
            if (next < 0) return next;
        }
        cc = next;
    }
    return kWalkFail;
}

// A mesh without a restart takes the loop without its tests: in one loop they
// made the walk of Population::update in such meshes 10% slower (4M particles at
// 48^3 cells, mixed form, 125 -> 138 us).
template <bool NEAR, class T>
__device__ __forceinline__ int walk_screened(const DevMesh &m, T x, T y, T z, int c, int max_steps, int &retests,
                                             CellRec &R, bool have_rec, float l[4]) {
    return NEAR && m.box ? walk_loop<true>(m, x, y, z, c, max_steps, retests, R, have_rec, l)
                         : walk_loop<false>(m, x, y, z, c, max_steps, retests, R, have_rec, l);
}

__device__ __forceinline__ int walk_mixed(const DevMesh &m, float x, float y, float z, int c, int max_steps,
                                          int &retests) {
    CellRec R;
    float l[4];
    return walk_screened<false>(m, x, y, z, c, max_steps, retests, R, false, l);
}

template <bool NEAR>
__device__ __forceinline__ int walk_fp64(const DevMesh &m, double x, double y, double z, int c, int max_steps) {
    CellRec R;
    float l[4];
    int retests = 0;
    return walk_screened<NEAR>(m, x, y, z, c, max_steps, retests, R, false, l);
}

// x - L floor(x / L), one coordinate of move_periodic
// (punc/include/punc/pusher.h:666-681), without the division where the
// quotient's floor is known to be 0, 1 or -1: for 0 < x < L, L <= x < 2 L and
// -L <= x <= -1e-200 the rounded quotient stays on its side of the integers
// (it has a neighbour of the integer between), so the results are the same
// bits.  The first test, the common one, is an integer comparison (positive
// doubles order as their bits).  For L outside (0, 1e100] (negative, zero, not
// finite) the formula stands as it is; L is the same for all particles, so its
// test costs an integer comparison.
__device__ __forceinline__ double wrap_periodic(double x, double L) {
    const unsigned long long bx = (unsigned long long)__double_as_longlong(x);
    const unsigned long long bl = (unsigned long long)__double_as_longlong(L);
    if (bl - 1 < (unsigned long long)__double_as_longlong(1e100)) {
        if (bx - 1 < bl - 1) return x;
        if (x >= L && x < 2.0 * L) return __dadd_rn(x, -L);
        if (x <= -1e-200 && x >= -L) return __dadd_rn(x, L);
    }
    return __dadd_rn(x, -__dmul_rn(L, floor(__ddiv_rn(x, L))));
}

// __float2ll_rn(v) for finite |v| < 2^62 on the 32-bit conversion path:
// below 2^23 in magnitude v rounds to nearest (even) in 32 bits; larger FP32
// values are integers, rebuilt from the significand and the exponent.
__device__ __forceinline__ long long float_to_ll_rn(float v) {
    if (fabsf(v) < 8388608.0f) return (long long)__float2int_rn(v);
    const unsigned u = __float_as_uint(v);
    const int sh = (int)((u >> 23) & 0xffu) - 150;
    const long long mag = (long long)((u & 0x7fffffu) | 0x800000u) << sh;
    return (u >> 31) ? -mag : mag;
}

// Cell<3>::barycentric (punc/include/punc/population.h:885-893), FP64.
__device__ __forceinline__ void barycentric_fp64(const DevMesh &m, int c, double x, double y, double z,
                                                 double &l0, double &l1, double &l2, double &l3) {
    const double2 *A = reinterpret_cast<const double2 *>(m.bary) + 6 * (size_t)c;
    const double2 a0 = __ldg(A + 0), a1 = __ldg(A + 1), a2 = __ldg(A + 2);
    const double2 a3 = __ldg(A + 3), a4 = __ldg(A + 4), a5 = __ldg(A + 5);
    l0 = plane64(a0.x, a0.y, a1.x, a1.y, x, y, z);
    l1 = plane64(a2.x, a2.y, a3.x, a3.y, x, y, z);
    l2 = plane64(a4.x, a4.y, a5.x, a5.y, x, y, z);
    l3 = __dadd_rn(__dadd_rn(__dadd_rn(1.0, -l0), -l1), -l2);
}

// Fixed-point CG1 deposit of the mixed form: q*lambda_i in units of
// 2^-kFixedBits q_max (q_scaled = q * 2^kFixedBits / q_max in FP32), added with int64
// atomics, so the sum is the same in any order.
__device__ __forceinline__ void deposit_fixed(const DevMesh &m, int c, float x, float y, float z, float q_scaled,
                                              unsigned long long *rho_fixed) {
    const float4 *A = m.cell_f + 4 * (size_t)c;
    const float4 a0 = __ldg(A), a1 = __ldg(A + 1), a2 = __ldg(A + 2);
    const float l0 = fmaf(a0.w, z, fmaf(a0.z, y, fmaf(a0.y, x, a0.x)));
    const float l1 = fmaf(a1.w, z, fmaf(a1.z, y, fmaf(a1.y, x, a1.x)));
    const float l2 = fmaf(a2.w, z, fmaf(a2.z, y, fmaf(a2.y, x, a2.x)));
    const float l3 = __fsub_rn(__fsub_rn(__fsub_rn(1.0f, l0), l1), l2);
    const int4 d = __ldg(m.dofs + c);
    atomicAdd(rho_fixed + d.x, (unsigned long long)float_to_ll_rn(__fmul_rn(l0, q_scaled)));
    atomicAdd(rho_fixed + d.y, (unsigned long long)float_to_ll_rn(__fmul_rn(l1, q_scaled)));
    atomicAdd(rho_fixed + d.z, (unsigned long long)float_to_ll_rn(__fmul_rn(l2, q_scaled)));
    atomicAdd(rho_fixed + d.w, (unsigned long long)float_to_ll_rn(__fmul_rn(l3, q_scaled)));
}

}  // namespace pg
