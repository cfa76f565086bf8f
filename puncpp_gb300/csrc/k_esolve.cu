// CG1 electric field: ESolver (punc/src/efield.cpp:41-75, punc/ufl/EField3D.ufl)
// solves the L2 projection of -grad(phi) onto continuous piecewise-linear
// vector fields,  M E_c = b_c  for the three components, with M the consistent
// P1 mass matrix and b_c,d = integral of (-d phi/dx_c) lambda_d = sum over the
// cells T of dof d of (vol_T / 4) (-grad phi_T)_c.
//
// The rhs is gathered per dof over its cells in ascending cell order
// (deterministic).  D^-1 M has its spectrum in [1/2, 5/2] on any P1 tetrahedral
// mesh (the element mass matrices (vol/20)(I + 1 1^T) scaled by their
// diagonal), so the three systems are solved by Chebyshev iteration on that
// interval (Golub and Varga 1961): as many products as conjugate gradients
// need here (30 for 1e-12, 15 for 1e-6 from a cold start), but no inner product
// in the loop, so one grid barrier per iteration and no reduction, where CG
// took two barriers and two nine-fold FP64 block and grid sums.  The number
// of iterations comes from the first residual and the tolerance; the residual
// is measured then, and again after a few more where it is not met.
// One pass over a row of M (SELL-32, one thread per row) serves the three
// components, which are stored together ([n][4]), so an entry costs one gather.
// One cooperative launch forms the rhs, solves and packs the field.
// Arithmetic in T (double for the FP64 form, float for the mixed form); the
// residual's norm in FP64.
//
// What bounds it: the gathers and the barrier of each iteration; in FP64 also
// the 58 FP64 operations of a row at 1/64 of the FP32 rate; in the form for
// larger systems (k_mass_cheb3), which reads the matrix each time, the chain of
// loads of a row.  Measured (GB300, solve with rhs and packing), CG -> that form ->
// rows in registers (k_mass_cheb3_reg): FP64 9,260 dofs 563 -> 266 -> 101 us, FP32
// 39,298 dofs 372 -> 117 -> 75 us.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include "pg_device.cuh"

namespace cg = cooperative_groups;

namespace pg {

namespace {

constexpr int kThreads = 256;

// [n][4] vectors: three components and a pad.
template <typename T>
struct V3 {
    T x, y, z;
};
__device__ __forceinline__ V3<float> load3(const float *p, int i) {
    const float4 v = reinterpret_cast<const float4 *>(p)[i];
    return {v.x, v.y, v.z};
}
__device__ __forceinline__ V3<double> load3(const double *p, int i) {
    const double2 *q = reinterpret_cast<const double2 *>(p) + 2 * (size_t)i;
    const double2 a = q[0];
    return {a.x, a.y, q[1].x};
}
__device__ __forceinline__ void store3(float *p, int i, const V3<float> &v) {
    reinterpret_cast<float4 *>(p)[i] = make_float4(v.x, v.y, v.z, 0.0f);
}
__device__ __forceinline__ void store3(double *p, int i, const V3<double> &v) {
    double2 *q = reinterpret_cast<double2 *>(p) + 2 * (size_t)i;
    q[0] = make_double2(v.x, v.y);
    q[1] = make_double2(v.z, 0.0);
}

// Sums of N per-thread values over the block; valid in thread 0 (sh: 16 N
// doubles; blocks of at most 16 warps).
template <int N>
__device__ __forceinline__ void block_sum_n(const double (&v)[N], double *sh, double (&out)[N]) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
    for (int k = 0; k < N; ++k) {
        double a = v[k];
        for (int o = 16; o > 0; o >>= 1) a += __shfl_down_sync(0xffffffffu, a, o);
        if (lane == 0) sh[k * 16 + w] = a;
    }
    __syncthreads();
    if (threadIdx.x == 0)
        for (int k = 0; k < N; ++k) {
            double a = 0.0;
            for (int q = 0; q < nw; ++q) a += sh[k * 16 + q];
            out[k] = a;
        }
}

// Sums over the blocks of part[k * nb + b], k < N, by warp 0; valid in its lane 0.
template <int N>
__device__ __forceinline__ void grid_sum_n(const double *part, int nb, double (&out)[N]) {
    if (threadIdx.x >= 32) return;
#pragma unroll
    for (int k = 0; k < N; ++k) {
        double a = 0.0;
        for (int b = threadIdx.x; b < nb; b += 32) a += __ldcg(part + k * nb + b);
        for (int o = 16; o > 0; o >>= 1) a += __shfl_down_sync(0xffffffffu, a, o);
        out[k] = a;
    }
}

// Chebyshev iteration on [1/2, 5/2]: centre, half-width, and -log of its
// asymptotic rate (acosh(centre / half-width)).  The coefficients converge by a
// factor of seven per iteration.
constexpr double kTheta = 1.5, kDelta = 1.0;
constexpr float kRate = 0.9624237f;
constexpr int kCheb = 24;

template <typename T>
struct Cheb3Args {
    int32_t n;
    const int64_t *adj_ptr;       // dof -> cells
    const int32_t *adj_cell;
    const double *vol, *E_cell;
    const int64_t *sptr;          // M in SELL-32
    const int32_t *swidth, *scol;
    const T *sval, *dinv;
    T *x, *r, *d0, *d1;           // [n][4]; x: start on entry, solution on return
    double *partials;             // [12][grid]
    double rtol, atol;
    int32_t max_iter;
    int32_t *out_iter, *out_status;
    double *out_rr, *out_bb;      // [3] each
    double e0[3];
    double *ev;                   // [n][4] or null
    float *evf;                   // [n][4] or null
    T c1[kCheb], c2[kCheb];       // d' = c1 d + c2 D^-1 r of the iterations (the last for all later ones)
};

// Row i of M times the three components of v.
template <typename T>
__device__ __forceinline__ V3<T> mass_row(const Cheb3Args<T> &a, const T *v, int i) {
    constexpr int C = 4;
    const int64_t base = __ldg(a.sptr + (i >> 5)) + (i & 31);
    const int w = __ldg(a.swidth + (i >> 5));
    V3<T> s{0, 0, 0};
    for (int k = 0; k < w; k += C) {
        int c[C];
        T m[C];
        V3<T> g[C];
#pragma unroll
        for (int q = 0; q < C; ++q) {
            const bool ok = k + q < w;
            c[q] = ok ? __ldg(a.scol + base + 32 * (k + q)) : i;
            m[q] = ok ? __ldg(a.sval + base + 32 * (k + q)) : (T)0;
        }
#pragma unroll
        for (int q = 0; q < C; ++q) g[q] = load3(v, c[q]);
#pragma unroll
        for (int q = 0; q < C; ++q) {
            s.x = fma(m[q], g[q].x, s.x);
            s.y = fma(m[q], g[q].y, s.y);
            s.z = fma(m[q], g[q].z, s.z);
        }
    }
    return s;
}

// Iterations until ||r||^2 = rr meets tol2 at the asymptotic rate, 1 to 64.
__device__ __forceinline__ int iterations_left(double rr, double tol2, float slack) {
    const float ratio2 = (float)(rr / tol2);
    return max(1, min(64, (int)ceilf((slack + 0.5f * logf(ratio2)) / kRate)));
}

// What the blocks decide together, each for itself from the same sums.
// bad: a residual or right-hand side that is not finite (or whose square is
// not), which ends the solve as not converged.
struct Checks {
    double tol2[3], rr[3], bb[3];
    int next_check, done, bad, cold[3];
};
__device__ __forceinline__ bool finite_sum(double v) { return v < (double)INFINITY; }   // v >= 0 or NaN

// The first residual and right-hand side (loc: this thread's squares, three
// components each) against the tolerance: the iterations needed, and the
// components whose start is worse than zero, or not finite, and is dropped.
// Every comparison is written so that a NaN does not meet it.  One grid barrier.
template <typename T>
__device__ void first_check(const Cheb3Args<T> &a, const double (&loc)[6], int nb, double *sh, Checks &S) {
    double out[6];
    block_sum_n<6>(loc, sh, out);
    if (threadIdx.x == 0)
        for (int k = 0; k < 6; ++k) a.partials[k * nb + blockIdx.x] = out[k];
    cg::this_grid().sync();
    grid_sum_n<6>(a.partials, nb, out);
    if (threadIdx.x < 32) {
        // one lane per component
        const int c = threadIdx.x;
        int need = 0, bad = 0;
        double v = 0.0, u = 0.0;
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            const double r0 = __shfl_sync(0xffffffffu, out[q], 0), b0 = __shfl_sync(0xffffffffu, out[3 + q], 0);
            if (c == q) { v = r0; u = b0; }
        }
        if (c < 3) {
            const double tol = fmax(a.rtol * sqrt(u), a.atol);
            S.cold[c] = !(v <= u);
            if (!(v <= u)) v = u;
            bad = !finite_sum(u);
            S.rr[c] = v;
            S.bb[c] = u;
            S.tol2[c] = tol * tol;
            // 1 / T_k(theta / delta) = 2 exp(-rate k) <= tol / ||r||, and three
            // iterations more: the error of the slowest modes, which CG
            // damps below its residual, is then below CG's too (16^3 to
            // 31^3, CG1 runs: phi within 2e-11 of a 64-bit run, CG 1.1e-10)
            if (!(v <= tol * tol)) need = iterations_left(v, tol * tol, 3.5f);
        }
        need = max(need, __shfl_down_sync(0xffffffffu, need, 2));
        need = max(need, __shfl_down_sync(0xffffffffu, need, 1));
        bad = __any_sync(0xffffffffu, bad);
        if (c == 0) {
            S.next_check = min(need, a.max_iter);
            S.done = need == 0 && !bad;
            S.bad = bad;
        }
    }
    __syncthreads();
}

// A later residual (part: the blocks' sums, complete): met, or more iterations.
template <typename T>
__device__ void later_check(const Cheb3Args<T> &a, const double *part, int nb, int it, Checks &S) {
    double out[3];
    grid_sum_n<3>(part, nb, out);
    if (threadIdx.x == 0) {
        int need = 0;
        for (int c = 0; c < 3; ++c) {
            S.rr[c] = out[c];
            if (!finite_sum(out[c])) S.bad = 1;
            if (!(out[c] <= S.tol2[c])) need = max(need, iterations_left(out[c], S.tol2[c], 0.0f));
        }
        S.done = need == 0;
        S.next_check = min(it + need, a.max_iter);
    }
    __syncthreads();
}

template <typename T>
__global__ void __launch_bounds__(512, 2) k_mass_cheb3(const __grid_constant__ Cheb3Args<T> a) {
    cg::grid_group grid = cg::this_grid();
    __shared__ double sh[16 * 6];
    __shared__ Checks S;
    const int nb = gridDim.x, n = a.n;
    const int gtid = blockIdx.x * blockDim.x + threadIdx.x, gs = nb * blockDim.x;
    T *d = a.d0, *dn = a.d1;
    // b (into dn), r = b - M x, d = D^-1 r / theta
    {
        double loc[6] = {0, 0, 0, 0, 0, 0};
        for (int i = gtid; i < n; i += gs) {
            double bx = 0.0, by = 0.0, bz = 0.0;
            const int64_t k1 = a.adj_ptr[i + 1];
#pragma unroll 4
            for (int64_t k = a.adj_ptr[i]; k < k1; ++k) {
                const int c = __ldg(a.adj_cell + k);
                const double w = 0.25 * __ldg(a.vol + c);
                const double2 e01 = __ldg(reinterpret_cast<const double2 *>(a.E_cell) + 2 * (size_t)c);
                const double e2 = __ldg(a.E_cell + 4 * (size_t)c + 2);
                bx = bx + w * e01.x;
                by = by + w * e01.y;
                bz = bz + w * e2;
            }
            const V3<T> b{(T)bx, (T)by, (T)bz}, s = mass_row(a, a.x, i);
            const V3<T> r{b.x - s.x, b.y - s.y, b.z - s.z};
            const T f = a.dinv[i] * (T)(1.0 / kTheta);
            store3(a.r, i, r);
            store3(dn, i, b);
            store3(d, i, V3<T>{f * r.x, f * r.y, f * r.z});
            loc[0] += (double)r.x * (double)r.x;
            loc[1] += (double)r.y * (double)r.y;
            loc[2] += (double)r.z * (double)r.z;
            loc[3] += (double)b.x * (double)b.x;
            loc[4] += (double)b.y * (double)b.y;
            loc[5] += (double)b.z * (double)b.z;
        }
        first_check(a, loc, nb, sh, S);
        if (S.cold[0] || S.cold[1] || S.cold[2]) {
            for (int i = gtid; i < n; i += gs) {
                const V3<T> b = load3(dn, i);
                V3<T> x = load3(a.x, i), r = load3(a.r, i), di = load3(d, i);
                const T f = a.dinv[i] * (T)(1.0 / kTheta);
                if (S.cold[0]) { x.x = 0; r.x = b.x; di.x = f * b.x; }
                if (S.cold[1]) { x.y = 0; r.y = b.y; di.y = f * b.y; }
                if (S.cold[2]) { x.z = 0; r.z = b.z; di.z = f * b.z; }
                store3(a.x, i, x);
                store3(a.r, i, r);
                store3(d, i, di);
            }
            grid.sync();
        }
    }
    int it = 0;
    while (!S.done && !S.bad && it < a.max_iter) {
        ++it;
        const bool check = it == S.next_check;
        const T c1 = a.c1[min(it, kCheb) - 1], c2 = a.c2[min(it, kCheb) - 1];
        double *part = a.partials + (size_t)(6 + 3 * (it & 1)) * nb;   // read by all before it is written again
        double loc[3] = {0, 0, 0};
        for (int i = gtid; i < n; i += gs) {
            // x += d, r -= M d, d' = c1 d + c2 D^-1 r
            const V3<T> di = load3(d, i), ri = load3(a.r, i), xi = load3(a.x, i);
            const T f = c2 * a.dinv[i];
            const V3<T> s = mass_row(a, d, i);
            const V3<T> r{ri.x - s.x, ri.y - s.y, ri.z - s.z};
            store3(a.x, i, V3<T>{xi.x + di.x, xi.y + di.y, xi.z + di.z});
            store3(a.r, i, r);
            store3(dn, i, V3<T>{c1 * di.x + f * r.x, c1 * di.y + f * r.y, c1 * di.z + f * r.z});
            if (check) {
                loc[0] += (double)r.x * (double)r.x;
                loc[1] += (double)r.y * (double)r.y;
                loc[2] += (double)r.z * (double)r.z;
            }
        }
        T *t = d;
        d = dn;
        dn = t;
        if (check) {
            double out[3];
            block_sum_n<3>(loc, sh, out);
            if (threadIdx.x == 0)
                for (int k = 0; k < 3; ++k) part[k * nb + blockIdx.x] = out[k];
        }
        grid.sync();
        if (check) later_check(a, part, nb, it, S);
    }
    // not finite: a field that shows it, and zero as the next start
    for (int i = gtid; i < n; i += gs) {
        const V3<T> x = load3(a.x, i);
        double ex = (double)x.x + a.e0[0], ey = (double)x.y + a.e0[1], ez = (double)x.z + a.e0[2];
        if (S.bad) {
            store3(a.x, i, V3<T>{0, 0, 0});
            ex = ey = ez = nan("");
        }
        if (a.ev) {
            reinterpret_cast<double2 *>(a.ev)[2 * (size_t)i] = make_double2(ex, ey);
            reinterpret_cast<double2 *>(a.ev)[2 * (size_t)i + 1] = make_double2(ez, 0.0);
        }
        if (a.evf) reinterpret_cast<float4 *>(a.evf)[i] = make_float4((float)ex, (float)ey, (float)ez, 0.0f);
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        *a.out_iter = it;
        *a.out_status = S.done ? 0 : 1;
        for (int c = 0; c < 3; ++c) { a.out_rr[c] = S.rr[c]; a.out_bb[c] = S.bb[c]; }
    }
}

// The same solve with everything of a row that does not change in its
// thread's registers: the row's first kHeld entries, D^-1, x, r and d, so
// that an iteration is one round of gathers of d and the barrier; entries beyond
// kHeld are read each time.  One warp holds a slice of 32 rows, for all three
// components (NC 3, the FP32 form: a 16-byte gather per entry from [n][4]) or
// for one of them (NC 1, FP64, from [3][n]: 15 entries of three components
// keep a warp's FP64 unit busy for 3 us, of one for 1, and there are enough
// SMs for three times the warps).
constexpr int kHeld = 16, kRegThreads = 512;

template <typename T, int NC>
__device__ __forceinline__ void load_nc(const T *v, int n, int comp, int i, T (&g)[NC]) {
    if constexpr (NC == 3) {
        const V3<T> q = load3(v, i);
        g[0] = q.x; g[1] = q.y; g[2] = q.z;
    } else {
        g[0] = v[(size_t)comp * n + i];
    }
}
template <typename T, int NC>
__device__ __forceinline__ void store_nc(T *v, int n, int comp, int i, const T (&g)[NC]) {
    if constexpr (NC == 3) store3(v, i, V3<T>{g[0], g[1], g[2]});
    else v[(size_t)comp * n + i] = g[0];
}

template <typename T, int NC>
__global__ void __launch_bounds__(kRegThreads, 1) k_mass_cheb3_reg(const __grid_constant__ Cheb3Args<T> a) {
    cg::grid_group grid = cg::this_grid();
    __shared__ double sh[16 * 6];
    __shared__ Checks S;
    const int nb = gridDim.x, n = a.n, lane = threadIdx.x & 31;
    const int slices = (n + 31) >> 5, unit = (int)(threadIdx.x >> 5) * nb + blockIdx.x;
    const bool mine = unit < slices * (3 / NC);
    const int comp = NC == 3 || !mine ? 0 : unit / slices, slice = mine ? unit - comp * slices : 0;
    const int i = 32 * slice + lane;
    const bool live = mine && i < n;
    const int w = mine ? __ldg(a.swidth + slice) : 0;
    const int64_t base = mine ? __ldg(a.sptr + slice) + lane : 0;
    int c[kHeld];
    T m[kHeld];
#pragma unroll
    for (int k = 0; k < kHeld; ++k) {
        c[k] = k < w ? __ldg(a.scol + base + 32 * k) : 0;
        m[k] = k < w ? __ldg(a.sval + base + 32 * k) : (T)0;
    }
    const T dinv = live ? __ldg(a.dinv + i) : (T)0;
    // this row of M times v (start: the [n][4] start vector, in either form)
    auto product = [&](const T *v, bool start, T (&s)[NC]) {
        T g[kHeld][NC];
#pragma unroll
        for (int k = 0; k < kHeld; ++k) {
#pragma unroll
            for (int q = 0; q < NC; ++q) g[k][q] = (T)0;
            if (k < w) {
                if (NC == 1 && start) g[k][0] = v[4 * (size_t)c[k] + comp];
                else load_nc<T, NC>(v, n, comp, c[k], g[k]);
            }
        }
#pragma unroll
        for (int q = 0; q < NC; ++q) s[q] = (T)0;
#pragma unroll
        for (int k = 0; k < kHeld; ++k)
#pragma unroll
            for (int q = 0; q < NC; ++q) s[q] = fma(m[k], g[k][q], s[q]);
        for (int k = kHeld; k < w; ++k) {
            const int ck = __ldg(a.scol + base + 32 * k);
            const T mk = __ldg(a.sval + base + 32 * k);
            T h[NC];
            if (NC == 1 && start) h[0] = v[4 * (size_t)ck + comp];
            else load_nc<T, NC>(v, n, comp, ck, h);
#pragma unroll
            for (int q = 0; q < NC; ++q) s[q] = fma(mk, h[q], s[q]);
        }
    };
    T *d = a.d0, *dn = a.d1;
    T x[NC], r[NC], di[NC], b[NC];
    double loc[6] = {0, 0, 0, 0, 0, 0};
#pragma unroll
    for (int q = 0; q < NC; ++q) x[q] = r[q] = di[q] = b[q] = (T)0;
    {
        double bs[NC];
#pragma unroll
        for (int q = 0; q < NC; ++q) bs[q] = 0.0;
        const int64_t k1 = live ? a.adj_ptr[i + 1] : 0;
#pragma unroll 4
        for (int64_t k = live ? a.adj_ptr[i] : 0; k < k1; ++k) {
            const int cell = __ldg(a.adj_cell + k);
            const double wt = 0.25 * __ldg(a.vol + cell);
            const double *E = a.E_cell + 4 * (size_t)cell;
#pragma unroll
            for (int q = 0; q < NC; ++q) bs[q] = bs[q] + wt * __ldg(E + (NC == 1 ? comp : q));
        }
        T s[NC];
        product(a.x, true, s);
        if (live) {
#pragma unroll
            for (int q = 0; q < NC; ++q) {
                x[q] = a.x[4 * (size_t)i + (NC == 1 ? comp : q)];
                b[q] = (T)bs[q];
                r[q] = b[q] - s[q];
                di[q] = dinv * (T)(1.0 / kTheta) * r[q];
            }
            store_nc<T, NC>(d, n, comp, i, di);
        }
    }
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        const bool own = NC == 3 || comp == q;
        const T rq = NC == 3 ? r[NC == 3 ? q : 0] : r[0], bq = NC == 3 ? b[NC == 3 ? q : 0] : b[0];
        loc[q] = own ? (double)rq * (double)rq : 0.0;
        loc[3 + q] = own ? (double)bq * (double)bq : 0.0;
    }
    first_check(a, loc, nb, sh, S);
    if (S.cold[0] || S.cold[1] || S.cold[2]) {
#pragma unroll
        for (int q = 0; q < NC; ++q)
            if (S.cold[NC == 1 ? comp : q]) {
                x[q] = (T)0;
                r[q] = b[q];
                di[q] = dinv * (T)(1.0 / kTheta) * b[q];
            }
        if (live) store_nc<T, NC>(d, n, comp, i, di);
        grid.sync();
    }
    int it = 0;
    while (!S.done && !S.bad && it < a.max_iter) {
        ++it;
        const bool check = it == S.next_check;
        const T c1 = a.c1[min(it, kCheb) - 1], f = a.c2[min(it, kCheb) - 1] * dinv;
        T s[NC];
        product(d, false, s);
#pragma unroll
        for (int q = 0; q < NC; ++q) {
            x[q] += di[q];
            r[q] -= s[q];
            di[q] = fma(f, r[q], c1 * di[q]);
        }
        if (live) store_nc<T, NC>(dn, n, comp, i, di);
        T *t = d;
        d = dn;
        dn = t;
        double *part = a.partials + (size_t)(6 + 3 * (it & 1)) * nb;   // read by all before it is written again
        if (check) {
            double lr[3], out[3];
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                const T rq = NC == 3 ? r[NC == 3 ? q : 0] : r[0];
                lr[q] = NC == 3 || comp == q ? (double)rq * (double)rq : 0.0;
            }
            block_sum_n<3>(lr, sh, out);
            if (threadIdx.x == 0)
                for (int k = 0; k < 3; ++k) part[k * nb + blockIdx.x] = out[k];
        }
        grid.sync();
        if (check) later_check(a, part, nb, it, S);
    }
    if (live) {
#pragma unroll
        for (int q = 0; q < NC; ++q) {
            const int cq = NC == 1 ? comp : q;
            const size_t o = 4 * (size_t)i + cq;
            const double v = S.bad ? nan("") : (double)x[q] + a.e0[cq];
            a.x[o] = S.bad ? (T)0 : x[q];
            if (a.ev) a.ev[o] = v;
            if (a.evf) a.evf[o] = (float)v;
            if (cq == 2) {
                if (a.ev) a.ev[o + 1] = 0.0;
                if (a.evf) a.evf[o + 1] = 0.0f;
            }
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        *a.out_iter = it;
        *a.out_status = S.done ? 0 : 1;
        for (int c2 = 0; c2 < 3; ++c2) { a.out_rr[c2] = S.rr[c2]; a.out_bb[c2] = S.bb[c2]; }
    }
}

// Planar [3][n] field to the packed vertex field (a field given by the caller).
template <typename T>
__global__ void k_pack_ev(int32_t n, const T *__restrict__ x, double e0x, double e0y, double e0z,
                          double *__restrict__ ev, float *__restrict__ evf) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double ex = (double)x[i] + e0x, ey = (double)x[n + i] + e0y, ez = (double)x[2 * n + i] + e0z;
    if (ev) {
        reinterpret_cast<double2 *>(ev)[2 * (size_t)i] = make_double2(ex, ey);
        reinterpret_cast<double2 *>(ev)[2 * (size_t)i + 1] = make_double2(ez, 0.0);
    }
    if (evf) reinterpret_cast<float4 *>(evf)[i] = make_float4((float)ex, (float)ey, (float)ez, 0.0f);
}

// Blocks of 512 threads, two per SM, or for fewer rows than that blocks of 128,
// so that the rows spread over the SMs (their FP64 pipes and L1s).
template <typename T>
void launch_shape(int n, int &blocks, int &threads) {
    static int per_sm[2] = {0, 0};
    const int size[2] = {128, 512};
    for (int k = 0; k < 2; ++k)
        if (per_sm[k] == 0) {
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm[k], k_mass_cheb3<T>, size[k], 0);
            per_sm[k] = per_sm[k] < 1 ? 1 : (per_sm[k] > 2 ? 2 : per_sm[k]);
        }
    const int k = (n + size[0] - 1) / size[0] <= per_sm[0] * sm_count() ? 0 : 1;
    threads = size[k];
    const int need = (n + threads - 1) / threads, cap = per_sm[k] * sm_count();
    blocks = need < cap ? need : cap;
}

template <typename T>
int solve(const EsolveArgs &e, T *buf, const T *sval, const T *dinv, cudaStream_t st) {
    const size_t n4 = 4 * (size_t)e.n;
    Cheb3Args<T> a{e.n, e.adj_ptr, e.adj_cell, e.vol, e.E_cell, e.sptr, e.swidth, e.scol, sval, dinv, buf, buf + n4,
                   buf + 2 * n4, buf + 3 * n4, e.partials, e.rtol, e.atol, e.max_iter, e.out_iter, e.out_status,
                   e.out_rr, e.out_bb, {e.E0[0], e.E0[1], e.E0[2]}, e.ev, e.evf, {}, {}};
    double rho = kDelta / kTheta;
    for (int k = 0; k < kCheb; ++k) {
        const double next = 1.0 / (2.0 * kTheta / kDelta - rho);
        a.c1[k] = (T)(next * rho);
        a.c2[k] = (T)(2.0 / kDelta * next);
        rho = next;
    }
    void *params[] = {&a};
    // rows in registers where one warp per unit fits the grid (up to 25,900
    // dofs in FP64, 77,800 in FP32), spread over all SMs; else two blocks per SM
    // striding over the rows
    constexpr int NC = sizeof(T) == 8 ? 1 : 3;
    const int units = (e.n + 31) / 32 * (3 / NC), sms = sm_count();
    if (units <= kRegThreads / 32 * sms) {
        const int nb = units < sms ? units : sms, warps = (units + nb - 1) / nb;
        return (int)cudaLaunchCooperativeKernel((const void *)k_mass_cheb3_reg<T, NC>, dim3(nb), dim3(32 * warps),
                                                params, 0, st);
    }
    int blocks = 0, threads = 0;
    launch_shape<T>(e.n, blocks, threads);
    return (int)cudaLaunchCooperativeKernel((const void *)k_mass_cheb3<T>, dim3(blocks), dim3(threads), params, 0, st);
}

}  // namespace

int esolve_grid_blocks() { return 2 * sm_count(); }

int launch_esolve(const EsolveArgs &e, cudaStream_t st) {
    if (e.n <= 0) return 0;
    count_launches(1);
    return e.fp32 ? solve<float>(e, e.buf32, e.sval32, e.dinv32, st) : solve<double>(e, e.buf, e.sval, e.dinv, st);
}

void launch_pack_ev64(int32_t n, const double *x3, const double E0[3], double *ev, float *evf, cudaStream_t st) {
    if (n <= 0) return;
    count_launches(1);
    k_pack_ev<double><<<(n + kThreads - 1) / kThreads, kThreads, 0, st>>>(n, x3, E0[0], E0[1], E0[2], ev, evf);
}

}  // namespace pg
