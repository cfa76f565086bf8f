// PCG preconditioned by one smoothed-aggregation AMG V-cycle per iteration,
// all in one launch (a cooperative grid, or one thread-block cluster).
//
// Krylov recurrence in FP32 with the solution, the inner products, the step
// lengths and the true-residual replacements in FP64 (p.Ap and the
// recurrence's ||r||^2 from one FP32 sum per thread, r.z from FP64 products);
// the stopping test is on the FP64 true residual ||b - A x|| <= max(rtol ||b||,
// atol).  A replacement before the end of a solve (hierarchies of three or more
// levels) takes the true residual inside the iteration's own V-cycle; the one
// at the end is a new pass that restarts the cycle from the true residual.
//
// The V-cycle (one weighted-Jacobi sweep from zero before the coarse
// correction and one after, Galerkin coarse operators, dense coarsest
// inverse) is applied in the algebraically identical form
//     B_l b = W_l b + S_l B_{l+1} S_l^T b,   W = w D^-1 (2 I - A w D^-1),
//     S = (I - w D^-1 A) P,
// with the last restriction and the coarse solve in one product
// (G = C^-1 S^T) and the up-sweep of levels >= 1 collapsed into one product
// (U1 = [S_1 | S_1 S_2 | ...]).  For L >= 2 levels above the coarsest an
// iteration is L + 4 grid phases:
//   A p = A z + beta A p_old and the sum that gives alpha;
//   x, r, s = w D^-1 r of the step, and ||r||^2;
//   b_1 = S_0^T r;
//   per level 1 .. L-1: the restriction (at L-1: G) and the smoothing W_l b_l
//     on disjoint blocks;
//   y_1 = t_1 + U1 [t_2 .. t_{L-1}, y_L];
//   z = W_0 r + S_0 y_1, both products of a row together, and r.z.
// Every product gathers one plain vector: a vector's scaling by w D^-1 is
// stored with it (s, AmgLevelDev::sb).
//
// What bounds it: the chain of dependent loads of each phase (entries, then
// gathers) and the barriers; at 80^3 also the L2, at 4 to 4.5 TB/s in the two
// phases that stream the level-0 operators.  Solves (GB300): 80^3 probe (531k
// rows) 1.18 ms, 56^3 (185k) 0.75, 40^3 (68,908) 0.43, 16^3 periodic (4,096)
// 0.29.  With double-float sums, FP32 step lengths and b_1 updated from step to
// step (b_1 -= alpha S_0^T A p, a phase less) it was 1.20, 0.74, 0.37 and 0.28 ms,
// but with 48 bits where the sums have 53 and a b_1 that drifts from r.  The
// figures at Span and the launch, unless dated, compare two forms with those sums.
#include <cooperative_groups.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <type_traits>

#include "pg_device.cuh"
#include "pg_reduce.cuh"

namespace cg = cooperative_groups;

namespace pg {

namespace {

// Vectors written inside the kernel are read with plain (L1-cached) loads
// only after a grid barrier, whose acquire makes the other blocks' writes
// visible; never through the read-only path (__ldg).
//
// Code size is a resource here: every phase runs its code once or twice per
// warp between two barriers, so instructions that are not in the SM's caches
// are fetched again each time.  So each product stands at one place and a
// storage form's loop is short (an earlier form with a gather function per
// site compiled to 1.3 MB; loads of 16 bytes added to it made an iteration 40%
// slower at 185k rows).  Arrays of a conditional load are zeroed: left
// undefined, the compiler carried them around the whole loop and spilled.

constexpr int kWarps = kPcgThreads / 32;

// The barrier between phases: of a cooperative grid, or of one thread-block
// cluster (the hardware's; all threads of a warp arrive together).
struct GridSync {
    static constexpr bool kCluster = false;
    __device__ __forceinline__ static void sync() { cg::this_grid().sync(); }
};
struct ClusterSync {
    static constexpr bool kCluster = true;
    __device__ __forceinline__ static void sync() {
        __syncwarp();
        asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    }
};
constexpr int kClusterMax = 16;   // blocks of a cluster

// Store v at this shared-memory address of block `rank` of the cluster.
__device__ __forceinline__ void store_remote(double *p, double v, int rank) {
    const uint32_t a = (uint32_t)__cvta_generic_to_shared(p);
    asm volatile("{\n\t.reg .b32 q;\n\tmapa.shared::cluster.u32 q, %0, %1;\n\tst.shared::cluster.f64 [q], %2;\n\t}"
                 ::"r"(a), "r"(rank), "d"(v)
                 : "memory");
}

// Inner products are summed in FP64.  A warp-wide FP64 add takes a
// sub-partition of an SM 64 cycles, so the sums go through shared memory in
// steps that keep each addition on one warp of every sub-partition: the 512
// threads' values in four by warps 0-3, the 128 sums in four by warp 0, and its
// five rounds of shuffles (1,340 cycles with its barriers; 2,240 with every
// warp's own five rounds first, 1,980 with the rounds in four warps).
template <int N = 32>   // the sum of each N lanes
__device__ __forceinline__ double warp_sum(double v) {
    for (int o = N / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ double sum4(const double *p, int step) {
    return (p[0] + p[step]) + (p[2 * step] + p[3 * step]);
}

// The block's sum of v, for the total after the caller's barrier: stored to
// part[blockIdx.x] in global memory, or in a cluster in every block's shared
// memory (read there without a trip to the L2).  sh: 1.25 kPcgThreads values.
template <class Sync, class T>
__device__ __forceinline__ void block_part(T v, double *sh, double *part, int nb) {
    const int t = threadIdx.x, q = kPcgThreads / 4;
    T *f = reinterpret_cast<T *>(sh);
    double *s = sh + kPcgThreads;
    f[t] = v;
    __syncthreads();
    if (t < q) s[t] = ((double)f[t] + (double)f[t + q]) + ((double)f[t + 2 * q] + (double)f[t + 3 * q]);
    __syncthreads();
    if (t < 32) {
        const double a = warp_sum(sum4(s + t, 32));
        if (Sync::kCluster) {
            if (t < nb) store_remote(part + blockIdx.x, a, t);
        } else if (t == 0) {
            part[blockIdx.x] = a;
        }
    }
}

// Total of the blocks' sums (the same order in every block: the same total),
// by one warp.  Its lanes meet first and all of them load, some in vain: in a
// warp that counts as diverged (after a barrier that one lane spins in, after
// loads by a part of the lanes) a shuffle takes 250 cycles and not 25.
template <class Sync>
__device__ __forceinline__ double warp_total(const double *part, int nb) {
    const int lane = threadIdx.x & 31;
    __syncwarp();
    if (Sync::kCluster) {
        const int b = lane & (kClusterMax - 1);
        const double v = part[b];
        return warp_sum<kClusterMax>(b < nb ? v : 0.0);
    }
    double a = 0.0;
    for (int k = 0; k < nb; k += 5 * 32) {
        double v[5];
#pragma unroll
        for (int u = 0; u < 5; ++u) {
            const int i = k + 32 * u + lane;
            const double p = __ldcg(part + (i < nb ? i : 0));
            v[u] = i < nb ? p : 0.0;
        }
        a += ((v[0] + v[1]) + (v[2] + v[3])) + v[4];
    }
    return warp_sum(a);
}
// The same in warp 0, by warps 0-3 of a grid's block; every thread of the block
// calls it.
template <class Sync>
__device__ __forceinline__ double block_total(const double *part, int nb, double *sh) {
    if (Sync::kCluster) return threadIdx.x < 32 ? warp_total<Sync>(part, nb) : 0.0;
    const int t = threadIdx.x, q = kPcgThreads / 4;
    if (t < q) {
        double a = 0.0;
        for (int k = t; k < nb; k += 3 * q) {
            const double v0 = __ldcg(part + k), v1 = k + q < nb ? __ldcg(part + k + q) : 0.0;
            const double v2 = k + 2 * q < nb ? __ldcg(part + k + 2 * q) : 0.0;
            a += (v0 + v1) + v2;
        }
        sh[t] = a;
    }
    __syncthreads();
    return t < 32 ? warp_sum(sum4(sh + t, 32)) : 0.0;
}

// ---- the work of a block ------------------------------------------------------
// The threads of nb blocks, b this block's number among them.  Row r (or, with
// g lanes a row, lane r g + k) of a product goes to the r-th of them, in one of
// two orders: block by block, or (spread) the first warp of every block, then
// the second ones.  Spread where the level-0 rows are at most one per thread: its
// coarse products then have fewer rows than threads, and block by block
// the first blocks worked and the others waited (39k rows: a product over
// 4,136 rows in 16 of 77 blocks).  Block by block above, where a block's rows
// should be neighbours that share gathered lines.  Solve, block by block ->
// spread: 4,096 rows 0.30 -> 0.26 ms, 21,952 0.61 -> 0.56, 39,298 0.54 -> 0.51,
// 68,908 0.59 -> 0.57; 13,824 (16 blocks) 0.475 -> 0.50.
// (Equal contiguous ranges per block, which leave no block a round of rows more
// than another, measured 1 to 5% slower than either at all sizes.)
struct Span {
    int b, nb;
    bool spread;
    __device__ __forceinline__ int first() const {
        const int w = threadIdx.x >> 5;
        return 32 * (spread ? w * nb + b : b * kWarps + w) + (int)(threadIdx.x & 31);
    }
    __device__ __forceinline__ int stride() const { return kPcgThreads * nb; }
};

// ---- products ---------------------------------------------------------------
// Read-only loads of operator entries that ask the L2 for the 256-byte
// segment around the address, so a row's next chunks arrive with this one.
__device__ __forceinline__ uint4 ld_nc_128(const void *p) {
    uint4 v;
    asm("ld.global.nc.L2::256B.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}
__device__ __forceinline__ uint2 ld_nc_64(const void *p) {
    uint2 v;
    asm("ld.global.nc.L2::256B.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
    return v;
}
__device__ __forceinline__ uint32_t ld_nc_32(const void *p) {
    uint32_t v;
    asm("ld.global.nc.L2::256B.u32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ float half_bits(uint32_t h) { return __half2float(__ushort_as_half((unsigned short)h)); }

// A chunk of four entries in each storage form: loaded whole, decoded by entry.
struct FmtH16 {   // binary16 values and 16-bit columns in one 16-byte load
    static constexpr bool kHalf = true;
    uint4 e = {0, 0, 0, 0};
    __device__ __forceinline__ void load(const SpOp &S, int k) { e = ld_nc_128((const uint4 *)S.val + k); }
    __device__ __forceinline__ uint32_t at(int j) const { return j == 0 ? e.x : j == 1 ? e.y : j == 2 ? e.z : e.w; }
    __device__ __forceinline__ int col(int j, int b) const { return b + (int)(at(j) & 0xffffu); }
    __device__ __forceinline__ float val(int j) const { return half_bits(at(j) >> 16); }
};
struct FmtF32 {   // FP32 values, 32-bit columns
    static constexpr bool kHalf = false;
    uint4 v = {0, 0, 0, 0}, c = {0, 0, 0, 0};
    __device__ __forceinline__ void load(const SpOp &S, int k) {
        v = ld_nc_128((const uint4 *)S.val + k);
        c = ld_nc_128((const uint4 *)S.col + k);
    }
    __device__ __forceinline__ int col(int j, int) const { return (int)(j == 0 ? c.x : j == 1 ? c.y : j == 2 ? c.z : c.w); }
    __device__ __forceinline__ float val(int j) const {
        return __uint_as_float(j == 0 ? v.x : j == 1 ? v.y : j == 2 ? v.z : v.w);
    }
};
struct FmtH32 {   // binary16 values, 32-bit columns
    static constexpr bool kHalf = true;
    uint2 v = {0, 0};
    uint4 c = {0, 0, 0, 0};
    __device__ __forceinline__ void load(const SpOp &S, int k) {
        v = ld_nc_64((const uint2 *)S.val + k);
        c = ld_nc_128((const uint4 *)S.col + k);
    }
    __device__ __forceinline__ int col(int j, int) const { return (int)(j == 0 ? c.x : j == 1 ? c.y : j == 2 ? c.z : c.w); }
    __device__ __forceinline__ float val(int j) const {
        const uint32_t w = j < 2 ? v.x : v.y;
        return half_bits(j & 1 ? w >> 16 : w & 0xffffu);
    }
};

// The sum over the stored entries of a SELL row: w chunks from off, C of them
// and their gathers in flight together, the first C loaded by the caller.
template <class F, int C>
__device__ __forceinline__ void sell_load(const SpOp &S, int off, int w, F (&f)[C]) {
#pragma unroll
    for (int c = 0; c < C; ++c) {
        f[c] = F{};
        if (c < w) f[c].load(S, off + 32 * c);
    }
}
template <class F, int C>
__device__ __forceinline__ float sell_sum(const SpOp &S, const float *x, int off, int w, int cb, F (&f)[C]) {
    float sum = 0.0f;
    for (int k = 0; k < w; k += C) {
        float g[C][4];
        if (k > 0) sell_load(S, off + 32 * k, w - k, f);
#pragma unroll
        for (int c = 0; c < C; ++c)
#pragma unroll
            for (int j = 0; j < 4; ++j) g[c][j] = k + c < w ? x[f[c].col(j, cb)] : 0.0f;
#pragma unroll
        for (int c = 0; c < C; ++c)
#pragma unroll
            for (int j = 0; j < 4; ++j) sum = fmaf(f[c].val(j), g[c][j], sum);
    }
    return F::kHalf ? sum * S.vscale : sum;
}

// The off-diagonal entries of a row of A_0, stored as pairs (w of them): the
// P1 rows of these meshes hold six, and a chunk of four would pad them to
// eight in the operator that is read twice per iteration.
struct A0Pairs {
    static constexpr int C = 3;
    uint2 v[C], c[C];   // values and columns
    __device__ __forceinline__ void load(const SpOp &A, int off, int w, int cb) {
#pragma unroll
        for (int q = 0; q < C; ++q) {
            v[q] = make_uint2(0, 0);
            c[q] = make_uint2(0, 0);
            if (q < w) {
                const int o = off + 32 * q;
                v[q] = ld_nc_64((const uint2 *)A.val + o);
                if (A.c16) {
                    const uint32_t u = ld_nc_32((const uint32_t *)A.col + o);
                    c[q] = make_uint2(cb + (u & 0xffffu), cb + (u >> 16));
                } else {
                    c[q] = ld_nc_64((const uint2 *)A.col + o);
                }
            }
        }
    }
};
__device__ __forceinline__ float a0_sum(const SpOp &A, const float *x, int off, int w, int cb, A0Pairs &e) {
    constexpr int C = A0Pairs::C;
    float sum = 0.0f;
    for (int k = 0; k < w; k += C) {
        float g[C][2];
        if (k > 0) e.load(A, off + 32 * k, w - k, cb);
#pragma unroll
        for (int q = 0; q < C; ++q) {
            g[q][0] = k + q < w ? x[e.c[q].x] : 0.0f;
            g[q][1] = k + q < w ? x[e.c[q].y] : 0.0f;
        }
#pragma unroll
        for (int q = 0; q < C; ++q) {
            sum = fmaf(__uint_as_float(e.v[q].x), g[q][0], sum);
            sum = fmaf(__uint_as_float(e.v[q].y), g[q][1], sum);
        }
    }
    return sum;
}

// The heads of row r's slice of a SELL operator, loaded a row ahead.
struct SellHead {
    int2 h = {0, 0};
    int end = 0;
    __device__ __forceinline__ void load(const SpOp &S, int r, int r1) {
        if (r < r1) {
            h = __ldg(S.head + (r >> 5));
            end = __ldg(&S.head[(r >> 5) + 1].x);
        }
    }
    __device__ __forceinline__ int off(int r) const { return h.x + (r & 31); }
    __device__ __forceinline__ int width() const { return (end - h.x) >> 5; }
};

// e.row(i, (S x)_i, e.pre(i)) for every row i, over the blocks of sp.  pre
// loads the row's other operands before its gathers start.  A phase is a chain
// of dependent trips per thread (head -> entries -> gathers) over 32 warps of an
// SM; what an earlier form kept in flight per thread beyond a row (two and
// four rows together, 128 registers) cost more in code and warps than it hid
// (100^3 solve 4.12 ms against 3.38).
// CSR: g <= 32 lanes a row, two chunks per lane and step, reduced by shuffles
// (all lanes run the same rounds); g = 64..512: the warps of one block a row,
// reduced through shared memory.
template <class F, class E>
__device__ __forceinline__ void product_f(const SpOp &S, const float *x, E &e, Span sp) {
    const int g = S.g;
    if (g == 1) {
        int i = sp.first();
        const int i1 = S.n, st = sp.stride();
        SellHead h;
        h.load(S, i, i1);
        for (; i < i1; i += st) {
            const int off = h.off(i), w = h.width(), cb = h.h.y;
            h.load(S, i + st, i1);
            const typename E::Pre pv = e.pre(i);
            F f[3];
            sell_load(S, off, w, f);
            e.row(i, sell_sum(S, x, off, w, cb, f), pv);
        }
        return;
    }
    const bool wide = g > 32;
    __shared__ float red[kWarps];
    const int sh = 31 - __clz(g), lane = threadIdx.x & (g - 1);
    const int pb = kPcgThreads >> sh;              // rows per block and round
    const int i1 = S.n, step = pb * sp.nb;
    int i = wide ? sp.b * pb + (int)(threadIdx.x >> sh) : sp.first() >> sh;
    const int rounds = (S.n + step - 1) / step;
    int2 h = make_int2(0, 0);
    int end = 0;
    if (i < i1) { h = __ldg(S.head + i); end = __ldg(&S.head[i + 1].x); }
    for (int t = 0; t < rounds; ++t, i += step) {
        const int in = i + step;
        const int off = h.x, cb = h.y, len = i < i1 ? end - h.x : 0;
        if (in < i1) { h = __ldg(S.head + in); end = __ldg(&S.head[in + 1].x); }
        typename E::Pre pv{};
        if (i < i1 && lane == 0) pv = e.pre(i);
        float sum = 0.0f;
        for (int k = lane; k < len; k += 2 * g) {
            F f[2];
            float v[2][4];
            const bool two = k + g < len;
            f[0].load(S, off + k);
            if (two) f[1].load(S, off + k + g);
#pragma unroll
            for (int j = 0; j < 4; ++j) v[0][j] = x[f[0].col(j, cb)];
#pragma unroll
            for (int j = 0; j < 4; ++j) v[1][j] = two ? x[f[1].col(j, cb)] : 0.0f;
#pragma unroll
            for (int j = 0; j < 4; ++j) sum = fmaf(f[0].val(j), v[0][j], sum);
#pragma unroll
            for (int j = 0; j < 4; ++j) sum = fmaf(f[1].val(j), v[1][j], sum);
        }
        for (int o = wide ? 16 : g >> 1; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        if (wide) {
            if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = sum;
            __syncthreads();
            if (lane == 0) {
                sum = 0.0f;
                for (int w = 0; w < g / 32; ++w) sum += red[(threadIdx.x >> 5) + w];
            }
            __syncthreads();
        }
        if (lane == 0 && i < i1) e.row(i, F::kHalf ? sum * S.vscale : sum, pv);
    }
}

// The storage form by a uniform branch.  V16 operators (the preconditioner's
// transfer and coarse operators) hold binary16 values and 16-bit columns
// unless a slice or row spans more; the others (G, the coarsest inverse) FP32
// and 32-bit columns.
template <bool V16, class E>
__device__ __forceinline__ void product(const SpOp &S, const float *x, E &e, Span sp) {
    if (V16 && S.c16) product_f<FmtH16>(S, x, e, sp);
    else if (V16) product_f<FmtH32>(S, x, e, sp);
    else product_f<FmtF32>(S, x, e, sp);
}

// ---- what a product's rows become -------------------------------------------
// b = S^T x and sb = omega D^-1 b for the level's smoother (sb null: none).
struct RestrictRow {
    using Pre = float;
    float *b, *sb;
    const float *dinv;
    float om;
    __device__ __forceinline__ Pre pre(int i) const { return sb ? __ldg(dinv + i) : 0.0f; }
    __device__ __forceinline__ void row(int i, float s, Pre d) const {
        b[i] = s;
        if (sb) sb[i] = om * d * s;
    }
};
// t = W x = omega D^-1 (2 x - A omega D^-1 x) from sx = omega D^-1 x.
struct SmoothRow {
    struct Pre { float sx, d; };
    float *t;
    const float *sx, *dinv;
    float om;
    __device__ __forceinline__ Pre pre(int i) const { return Pre{sx[i], __ldg(dinv + i)}; }
    __device__ __forceinline__ void row(int i, float s, const Pre &p) const { t[i] = fmaf(-om * p.d, s, 2.0f * p.sx); }
};
struct AddRow {
    using Pre = float;
    float *y;
    const float *t;
    __device__ __forceinline__ Pre pre(int i) const { return t[i]; }
    __device__ __forceinline__ void row(int i, float s, Pre ti) const { y[i] = ti + s; }
};
// z = s and this thread's share of r.z (the coarsest level alone)
struct DirectRow {
    using Pre = float;
    float *z;
    const float *r;
    double rz;
    __device__ __forceinline__ Pre pre(int i) const { return r[i]; }
    __device__ __forceinline__ void row(int i, float s, Pre ri) {
        z[i] = s;
        rz = fma((double)s, (double)ri, rz);
    }
};

// z = W_0 r + S_0 y with W_0 r = omega D^-1 (2 r - A_0 s), s = omega D^-1 r, and
// this thread's share of r.z: both products of a row in one pass (no vector
// t_0 = W_0 r to write and read).  omega D^-1 a_ii s_i = omega s_i, so A_0's
// diagonal is not read.
// kAhead: the operands of a thread's first row that no other thread changes (the
// operators' heads and entries, s and r of its own) are loaded by first() before
// the barrier, which ends with the L1 empty: two of the phase's three trips to
// the L2 then pass while the block waits.  That needs 128 registers, so it is
// the form of one block per SM (39,298 rows, 10 CG1 steps 5.41 -> 5.12 ms; 68,908
// rows, solve 0.60 -> 0.56 ms); in 64 registers it spills, and in a cluster, whose
// barrier is short, it gained nothing (4,096 rows 1% slower).
template <class F, bool kAhead>
struct Prolong {
    SellHead ha, hs;
    A0Pairs ea;
    F es[3];
    float si = 0.0f, ri = 0.0f, di = 0.0f;
    __device__ __forceinline__ void load(const SpOp &A, const float *s, const float *r, const float *dinv, int i) {
        si = s[i]; ri = r[i]; di = __ldg(dinv + i);
        ea.load(A, ha.off(i), ha.width(), ha.h.y);
    }
    __device__ __forceinline__ void first(const SpOp &A, const SpOp &S, const float *s, const float *r,
                                          const float *dinv, int i0, int i1) {
        if (!kAhead) return;
        ha.load(A, i0, i1);
        hs.load(S, i0, i1);
        if (i0 < i1) {
            load(A, s, r, dinv, i0);
            sell_load(S, hs.off(i0), hs.width(), es);
        }
    }
    __device__ __forceinline__ double rows(const SpOp &A, const SpOp &S, const float *s, const float *y, const float *r,
                                           const float *dinv, float om, float *z, int i0, int i1, int st) {
        double rz = 0.0;
        if (!kAhead) {
            ha.load(A, i0, i1);
            hs.load(S, i0, i1);
        }
        for (int i = i0; i < i1; i += st) {
            const bool have = kAhead && i == i0;
            if (!have) load(A, s, r, dinv, i);
            const int oa = ha.off(i), wa = ha.width(), ca = ha.h.y, os = hs.off(i), ws = hs.width(), cs = hs.h.y;
            ha.load(A, i + st, i1);
            hs.load(S, i + st, i1);
            const float q = a0_sum(A, s, oa, wa, ca, ea);
            if (!have) sell_load(S, os, ws, es);
            const float u = sell_sum(S, y, os, ws, cs, es);
            const float v = fmaf(-om * di, q, (2.0f - om) * si) + u;
            z[i] = v;
            rz = fma((double)v, (double)ri, rz);
        }
        return rz;
    }
};

// p = z + beta p, Ap = A z + beta Ap (none: the first step, no reads of p and
// Ap), and this thread's share of p.Ap in FP32.
template <bool kAhead>
struct Direction {
    SellHead h;
    A0Pairs e;
    float di = 0.0f;
    __device__ __forceinline__ void load(const SpOp &A, const float *diag, int i) {
        e.load(A, h.off(i), h.width(), h.h.y);
        di = __ldg(diag + i);
    }
    __device__ __forceinline__ void first(const SpOp &A, const float *diag, int i0, int i1) {
        if (!kAhead) return;
        h.load(A, i0, i1);
        if (i0 < i1) load(A, diag, i0);
    }
    __device__ __forceinline__ float rows(const SpOp &A, const float *diag, const float *z, float *p, float *Ap,
                                          float beta, bool none, int i0, int i1, int st) {
        float pap = 0.0f;
        if (!kAhead) h.load(A, i0, i1);
        for (int i = i0; i < i1; i += st) {
            if (!kAhead || i != i0) load(A, diag, i);
            const int off = h.off(i), w = h.width(), cb = h.h.y;
            h.load(A, i + st, i1);
            const float zi = z[i];
            const float p0 = none ? 0.0f : p[i], q0 = none ? 0.0f : Ap[i];
            const float s = fmaf(di, zi, a0_sum(A, z, off, w, cb, e));
            const float pi = fmaf(beta, p0, zi), api = fmaf(beta, q0, s);
            p[i] = pi;
            Ap[i] = api;
            pap = fmaf(pi, api, pap);
        }
        return pap;
    }
};

// Blocks [0, cut) take the first and [cut, nb) the second of two independent
// products of one phase, in proportion to their stored chunks, so that their
// latency chains run side by side instead of one after another.
__device__ __forceinline__ int split_point(const SpOp &A, const SpOp &B, int nb) {
    const float a = (float)A.chunks, b = (float)B.chunks;
    const int cut = (int)((float)nb * (a / (a + b)) + 0.5f);
    return cut < 1 ? 1 : (cut > nb - 1 ? nb - 1 : cut);
}

// The FP64 true residual b - A x of this thread's rows (A the solver's FP64
// SELL matrix; x read through L2, it is written inside the kernel) into r in
// FP32 and, with s, omega D^-1 r into s; returns this thread's share of
// ||b - A x||^2 and, with want_bb, adds its share of ||b||^2 to bb.
__device__ __forceinline__ double true_residual(const PcgArgs &a, float *r, float *s, float om, bool want_bb,
                                                double &bb, int i0, int i1, int gst) {
    double rr = 0.0;
    for (int i = i0; i < i1; i += gst) {
        double q = 0.0;
        const int64_t base = a.slice_ptr[i >> 5] + (i & 31);
        const int w = a.slice_width[i >> 5];
#pragma unroll 4
        for (int k = 0; k < w; ++k) q = fma(__ldg(a.val + base + 32 * k), __ldcg(a.x + __ldg(a.col + base + 32 * k)), q);
        const double bi = a.b[i];
        const double ri = bi - q;
        const float r32 = (float)ri;
        r[i] = r32;
        if (s) s[i] = om * __ldg(a.dinv32 + i) * r32;
        rr = fma(ri, ri, rr);
        if (want_bb) bb = fma(bi, bi, bb);
    }
    return rr;
}

// x += alpha p, r -= alpha Ap, s = omega D^-1 r of this thread's rows, and its
// share of the new ||r||^2 in FP32.  The operands of its first rows (p and Ap written by the same thread) are loaded
// before the barrier and the sums that give alpha.
struct CgUpdate {
    static constexpr int R = 4;
    double x[R];
    float p[R], q[R], r[R], d[R];
    __device__ __forceinline__ void load(const PcgArgs &a, int i, int i1, int gst) {
#pragma unroll
        for (int k = 0; k < R; ++k) {
            const int j = i + k * gst;
            const bool ok = j < i1;
            x[k] = ok ? a.x[j] : 0.0;
            p[k] = ok ? a.p32[j] : 0.0f;
            q[k] = ok ? a.Ap32[j] : 0.0f;
            r[k] = ok ? a.r32[j] : 0.0f;
            d[k] = ok ? __ldg(a.dinv32 + j) : 0.0f;
        }
    }
    __device__ __forceinline__ float apply(const PcgArgs &a, float *s, float om, double alpha, int i, int i1, int gst,
                                           float rr) const {
        const float alpha32 = (float)alpha;
#pragma unroll
        for (int k = 0; k < R; ++k) {
            const int j = i + k * gst;
            if (j < i1) {
                const float n = fmaf(-alpha32, q[k], r[k]);
                a.x[j] = fma(alpha, (double)p[k], x[k]);
                a.r32[j] = n;
                s[j] = om * d[k] * n;
                rr = fmaf(n, n, rr);
            }
        }
        return rr;
    }
};

// Partial sums: p.Ap in A, r.z in C, ||r||^2 of the recurrence in E (a cluster
// keeps these in shared memory); the FP64 true residual's and the right-hand
// side's squares in B and D.  A buffer is written again only after at least one
// barrier has passed since every block read it.
template <class Sync, int kBlocks>
__global__ void __launch_bounds__(kPcgThreads, kBlocks) k_pcg_amg(const __grid_constant__ PcgArgs a,
                                                            const __grid_constant__ AmgDev M) {
    constexpr bool kAhead = kBlocks == 1 && !Sync::kCluster;
    __shared__ double sh[2 * kPcgThreads + 16];
    const int nb = gridDim.x, n = a.n, L = M.nlev - 1;
    const Span all{(int)blockIdx.x, nb, n <= nb * kPcgThreads};
    const int i0 = all.first(), i1 = n, gst = all.stride();
    __shared__ double part_cluster[Sync::kCluster ? 3 * kClusterMax : 1];
    const int pst = Sync::kCluster ? kClusterMax : nb;
    double *partA = Sync::kCluster ? part_cluster : a.partials;
    double *partC = partA + pst, *partE = partA + 2 * pst;
    double *partB = a.partials + 3 * nb, *partD = a.partials + 4 * nb;
    const float om0 = M.lev[0].omega;
    float *r = a.r32, *z = a.z32, *s0 = M.s0;
    double ra, rb;
    // solver scalars, kept by warp 0 (no registers held across the loop)
    __shared__ double t_rz, t_tol2, t_rr, t_bb, t_alpha, t_mean;
    __shared__ float t_beta;
    __shared__ int t_status, t_updates, t_pass, t_go;
    // what the recurrence's ||r||^2 asks for: go on, replace the residual
    // inside this cycle, start a new pass (the last warp's)
    enum { kGoOn, kKeep, kNewPass };
    __shared__ int t_next;

    if (a.remove_mean) {
        double s = 0.0;
        for (int i = i0; i < i1; i += gst) s += a.b[i];
        block_sum2(s, 0.0, sh, ra, rb);
        if (threadIdx.x == 0) partD[blockIdx.x] = ra;
        Sync::sync();
        grid_sum2(partD, nullptr, nb, sh, ra, rb);
        if (threadIdx.x == 0) t_mean = ra / (double)n;
        __syncthreads();
        const double mean = t_mean;
        for (int i = i0; i < i1; i += gst) a.b[i] = a.b[i] - mean;
        Sync::sync();
    }
    if (threadIdx.x == 0) {
        t_tol2 = t_rr = t_bb = t_rz = 0.0;
        t_status = 1; t_updates = 0; t_pass = 0;
    }
    int it = 0;                                   // CG steps taken
    // the recurrence's ||r||^2 (complete in E) in the last warp, beside the
    // restriction, of which it has the fewest rows: waited for by all threads it
    // is 0.8 us of an iteration.  (The warp's number by a shuffle, and t_next
    // from all its lanes: the warp then counts as converged.)
    auto look = [&] {
        if (__shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0) != kWarps - 1) return;
        const double rec = warp_total<Sync>(partE, nb);
        const bool last = rec <= t_tol2 || it >= a.max_iter, fell = rec <= 1e-6 * t_rr;
        t_next = last || (fell && L < 2) ? kNewPass : fell ? kKeep : kGoOn;
    };
    // fresh: start a pass, from the FP64 true residual; else a CG step
    bool fresh = true;
    Direction<kAhead> dir;
    for (;;) {
        int next = kGoOn;
        if (fresh) {
            double bb = 0.0;
            const double rr = true_residual(a, r, s0, om0, it == 0, bb, i0, i1, gst);
            block_sum2(rr, bb, sh, ra, rb);
            if (threadIdx.x == 0) { partB[blockIdx.x] = ra; partD[blockIdx.x] = rb; }
            Sync::sync();
            grid_sum2(partB, partD, nb, sh, ra, rb);
            if (threadIdx.x == 0) {
                // between replacements the FP32 recurrence's ||r||^2 falls by 1e6;
                // a true residual that fell by less than 100 (10 in norm) means
                // the recurrence has left the true residual at its attainable
                // accuracy above the requested tolerance: stop (status 3)
                // instead of iterating on
                const bool stalled = t_pass > 0 && ra > 1e-2 * t_rr;
                t_rr = ra;
                if (t_pass == 0) {
                    t_bb = rb;
                    const double tol = fmax(a.rtol * sqrt(t_bb), a.atol);
                    t_tol2 = tol * tol;
                } else {
                    ++t_updates;
                }
                ++t_pass;
                t_go = 0;
                if (t_rr <= t_tol2) t_status = 0;
                else if (it >= a.max_iter) t_status = 1;
                else if (stalled) t_status = 3;
                else t_go = 1;
            }
            __syncthreads();
            if (!t_go) break;
        } else {
            // p = z + beta p, Ap = A z + beta Ap, p.Ap
            const float pap32 = dir.rows(M.lev[0].A, M.diag0, z, a.p32, a.Ap32, t_beta, it == 0, i0, i1, gst);
            CgUpdate up;
            up.load(a, i0, i1, gst);
            block_part<Sync>(pap32, sh, partA, nb);
            Sync::sync();
            const double pap = block_total<Sync>(partA, nb, sh);
            if (threadIdx.x == 0) {
                t_go = pap > 0.0;
                t_alpha = t_rz / pap;
                if (!(pap > 0.0)) t_status = 2;
            }
            __syncthreads();
            ++it;
            if (!t_go) break;
            const double alpha = t_alpha;
            float rr32 = up.apply(a, s0, om0, alpha, i0, i1, gst, 0.0f);
            for (int i = i0 + CgUpdate::R * gst; i < i1; i += CgUpdate::R * gst) {
                up.load(a, i, i1, gst);
                rr32 = up.apply(a, s0, om0, alpha, i, i1, gst, rr32);
            }
            block_part<Sync>(rr32, sh, partE, nb);
            Sync::sync();
            look();
        }
        // z = B r
        if (L >= 2) {
            // b_1 = S_0^T r: a phase of its own after the update, which gathers one
            // vector; within the update's phase it would gather r and A p (80^3:
            // 15 us an iteration more)
            const AmgLevelDev &V = M.lev[1];
            RestrictRow e{V.b, V.sb, V.dinv, V.omega};
            product<true>(M.lev[0].ST, r, e, all);
        }
        if (!fresh) {
            __syncthreads();
            next = t_next;
        }
        if (L >= 2 || next == kNewPass) Sync::sync();
        if (next == kNewPass) {
            fresh = true;
            continue;
        }
        const float *yup = M.yL;
        if (L == 1) {
            RestrictRow e{M.yL, nullptr, nullptr, 0.0f};
            product<false>(M.G, r, e, all);
            Sync::sync();
        }
        for (int l = 1; l < L; ++l) {
            // the restriction to the next level (or G) and the smoothing W_l
            const bool coarse = l == L - 1;
            const AmgLevelDev &V = M.lev[l];
            int my = -1;
            Span sp = all;
            if (nb > 1) {
                const int cut = coarse ? split_point(M.G, V.A, nb) : split_point(V.ST, V.A, nb);
                my = (int)blockIdx.x < cut ? 0 : 1;
                sp = my ? Span{(int)blockIdx.x - cut, nb - cut, all.spread} : Span{(int)blockIdx.x, cut, all.spread};
            }
            if (my != 1) {
                const AmgLevelDev &N = M.lev[coarse ? l : l + 1];
                RestrictRow e{coarse ? M.yL : N.b, coarse ? nullptr : N.sb, N.dinv, N.omega};
                if (coarse) product<false>(M.G, V.b, e, sp);
                else product<true>(V.ST, V.b, e, sp);
            }
            if (my != 0) {
                SmoothRow w{V.t, V.sb, V.dinv, V.omega};
                product<true>(V.A, V.sb, w, sp);
            }
            if (next == kKeep && coarse) {
                // replacement inside the cycle: the FP64 true residual of x
                // (complete here) into r; z = B r of the recurrence's r stands
                // for B of the true one (they differ by the recurrence's drift)
                double unused = 0.0;
                const double rr = true_residual(a, r, nullptr, 0.0f, false, unused, i0, i1, gst);
                block_sum2(rr, 0.0, sh, ra, rb);
                if (threadIdx.x == 0) partD[blockIdx.x] = ra;
            }
            Sync::sync();
        }
        double rz;
        if (L >= 1) {
            const SpOp &A0 = M.lev[0].A;
            if (L >= 2) {
                AddRow e{M.y1, M.lev[1].t};
                product<true>(M.U1, M.stack, e, all);
                yup = M.y1;
            }
            auto up = [&](auto pro) {
                pro.first(A0, M.S0, s0, r, a.dinv32, i0, i1);
                if (L >= 2) Sync::sync();
                rz = pro.rows(A0, M.S0, s0, yup, r, a.dinv32, om0, z, i0, i1, gst);
            };
            if (M.S0.c16) up(Prolong<FmtH16, kAhead>{});
            else up(Prolong<FmtH32, kAhead>{});
        } else {
            DirectRow e{z, r, 0.0};
            product<false>(M.cinv, r, e, all);
            rz = e.rz;
        }
        dir.first(M.lev[0].A, M.diag0, i0, i1);
        block_part<Sync>(rz, sh, partC, nb);
        Sync::sync();
        rz = block_total<Sync>(partC, nb, sh);
        if (threadIdx.x == 0) {
            // the direction continues across replacements
            t_beta = it == 0 ? 0.0f : (float)(rz / t_rz);
            t_rz = rz;
        }
        if (next == kKeep) {
            // the true residual replaces the recurrence's (as at a pass start,
            // with the same stall test)
            grid_sum2(partD, nullptr, nb, sh, ra, rb);
            if (threadIdx.x == 0) {
                const bool stalled = ra > 1e-2 * t_rr;
                t_rr = ra;
                ++t_updates;
                t_go = 0;
                if (t_rr <= t_tol2) t_status = 0;
                else if (stalled) t_status = 3;
                else t_go = 1;
            }
            __syncthreads();
            if (!t_go) break;
        }
        __syncthreads();
        fresh = false;
    }
    if (a.remove_mean) {
        Sync::sync();
        double s = 0.0;
        for (int i = i0; i < i1; i += gst) s += a.x[i];
        block_sum2(s, 0.0, sh, ra, rb);
        if (threadIdx.x == 0) partB[blockIdx.x] = ra;
        Sync::sync();
        grid_sum2(partB, nullptr, nb, sh, ra, rb);
        if (threadIdx.x == 0) t_mean = ra / (double)n;
        __syncthreads();
        const double mean = t_mean;
        for (int i = i0; i < i1; i += gst) a.x[i] = a.x[i] - mean;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        *a.out_iter = it;
        *a.out_status = t_status;
        *a.out_rr = t_rr;
        *a.out_bb = t_bb;
        if (a.out_updates) *a.out_updates = t_updates;
    }
}

}  // namespace

// Systems of at most kClusterRows rows run on one cluster, as many blocks (a
// power of two, at most 16) as leave kClusterRowsPerBlock rows to each: its
// barrier is the hardware's (0.6 us after stores of all threads, 0.37 of it
// their release, against 1.2 us of a cooperative grid, 1.4 with two blocks per
// SM; six times an iteration) and its sums stay in shared memory, while its 16
// SMs are enough for so few rows.  Measured, solve on the grid -> on the cluster: 2,744
// rows 0.84 -> 0.45 ms, 9,260 0.49 -> 0.385, 13,824 0.467 -> 0.474 and, periodic, 0.64
// -> 0.66, 39,298 0.61 -> 0.93, so the line lies between the second and the
// third.  (With FP64 sums and the restriction in a phase of its own: 9,248 rows
// 0.437 -> 0.354, 15,606 0.466 -> 0.426, 24,362 0.462 -> 0.515; the line could lie at
// 17,000 rows now.)  Rows per block: 1,000 rows 0.50 / 0.38 / 0.33 / 0.29 ms with
// 512 / 256 / 128 / 64.
constexpr int kClusterRows = 12288, kClusterRowsPerBlock = 64;

int pcg_amg_grid_blocks() {
    static int g = 0;
    if (g == 0) {
        int per_sm = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_pcg_amg<GridSync, 2>, kPcgThreads, 0);
        if (per_sm < 1) per_sm = 1;
        if (per_sm > 2) per_sm = 2;
        g = per_sm * sm_count();
    }
    return g;
}

// Largest cluster (a power of two) of the kernel on the current device.
static int query_cluster_blocks() {
    const void *fn = (const void *)k_pcg_amg<ClusterSync, 1>;
    const bool large = cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess;
    if (!large) cudaGetLastError();
    for (int k = large ? kClusterMax : 8; k > 1; k /= 2) {
        cudaLaunchConfig_t cfg{};
        cudaLaunchAttribute at{};
        at.id = cudaLaunchAttributeClusterDimension;
        at.val.clusterDim.x = k;
        at.val.clusterDim.y = at.val.clusterDim.z = 1;
        cfg.gridDim = dim3(k);
        cfg.blockDim = dim3(kPcgThreads);
        cfg.attrs = &at;
        cfg.numAttrs = 1;
        int n = 0;
        if (cudaOccupancyMaxActiveClusters(&n, fn, &cfg) == cudaSuccess && n > 0) return k;
        cudaGetLastError();
    }
    return 1;
}

// Found once per device: a kernel's attributes are the device's, so the size
// that one device takes says nothing about another in the same process.
static int cluster_blocks() {
    constexpr int kDevices = 64;
    static std::atomic<int> known[kDevices];   // 0: not yet
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kDevices) return query_cluster_blocks();
    int g = known[dev].load(std::memory_order_relaxed);
    if (g == 0) known[dev].store(g = query_cluster_blocks(), std::memory_order_relaxed);
    return g;
}

int launch_pcg_amg(const PcgArgs &a, const AmgDev &amg, cudaStream_t st) {
    PcgArgs arg = a;
    AmgDev m = amg;
    void *params[] = {&arg, &m};
    count_launches(1);
    if (a.n <= kClusterRows) {
        int nb = cluster_blocks();
        while (nb > 1 && a.n <= nb / 2 * kClusterRowsPerBlock) nb /= 2;
        cudaLaunchConfig_t cfg{};
        cudaLaunchAttribute at{};
        at.id = cudaLaunchAttributeClusterDimension;
        at.val.clusterDim.x = nb;
        at.val.clusterDim.y = at.val.clusterDim.z = 1;
        cfg.gridDim = dim3(nb);
        cfg.blockDim = dim3(kPcgThreads);
        cfg.stream = st;
        cfg.attrs = &at;
        cfg.numAttrs = 1;
        return (int)cudaLaunchKernelExC(&cfg, (const void *)k_pcg_amg<ClusterSync, 1>, params);
    }
    int nb = pcg_amg_grid_blocks();
    // one row per thread where the blocks suffice; below one block per SM twice
    // as many, so that the coarse products have the idle SMs (39,298 rows: 0.51 ms
    // with 77 blocks, 0.48 with 152; four times as many lose to the barrier: 21,952
    // rows 0.56 ms with 43, 0.55 with 86, 0.60 with 152)
    const int need = (a.n + kPcgThreads - 1) / kPcgThreads, sms = sm_count();
    if (need < nb) nb = need > sms ? need : std::max(need, std::min(sms, 2 * need));
    const void *fn = nb <= sms ? (const void *)k_pcg_amg<GridSync, 1> : (const void *)k_pcg_amg<GridSync, 2>;
    return (int)cudaLaunchCooperativeKernel(fn, dim3(nb), dim3(kPcgThreads), params, 0, st);
}

}  // namespace pg
