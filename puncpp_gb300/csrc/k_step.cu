// Per-step bookkeeping on the device, so that a whole time step runs without
// host round trips and can be captured as a CUDA graph:
//   object currents and charges from the absorbed counts (Population::update's
//   current bookkeeping, punc/include/punc/population.h:686-698),
//   CircuitCM pre_solve / post_solve (punc/src/object_CM.cpp:53-60, 275-357)
//   in the engine's host loop order (FP64, no contraction: the same bits as the
//   host path),
//   the superposition phi = phi0 + sum V_k L_k with device potentials,
//   particle and RNG counters, and one row of step results.
#include <cuda_runtime.h>

#include "pg_device.cuh"

namespace pg {

namespace {

// CircuitCM::pre_solve (object_CM.cpp:53-60): current sources move charge;
// potentials to zero.  isrc: [n][3] (node_a, node_b, value).
__global__ void k_circuit_pre(const double *isrc, int n_isrc, double circ_dt, int n_obj, double *obj,
                              double *obj_pot) {
    for (int k = 0; k < n_isrc; ++k) {
        const int a = (int)isrc[3 * k], b = (int)isrc[3 * k + 1];
        const double dQ = isrc[3 * k + 2] * circ_dt;
        if (a != -1) obj[4 * a + 0] -= dQ;
        if (b != -1) obj[4 * b + 0] += dQ;
    }
    for (int i = 0; i < n_obj; ++i) { obj[4 * i + 2] = 0.0; obj_pot[i] = 0.0; }
}

// CircuitCM::post_solve (object_CM.cpp:275-357) with the image charges img:
// circuit vector from the charge-sharing groups and the fixed-voltage sets,
// then potentials and charges from the inverse circuit matrix.  A group, a
// fixed-voltage member and a row of the matrix each have their own thread and
// the host loop's order of additions (the same bits); sets that share an object
// (c.distinct 0) are gone through by one thread, the last one counting.  A
// chain of 2n dependent FP64 operations bounds it: 24 objects 255 us on one
// thread, 8 us with a thread per row.
__global__ void k_circuit_post(const CircuitDev c, const double *img, double *obj, double *obj_pot) {
    const int n = c.n, t = threadIdx.x;
    double *cv = c.cv;
    const int first = c.distinct ? t : (t == 0 ? 0 : 0x7fffffff), step = c.distinct ? (int)blockDim.x : 1;
    for (int g = first; g < c.n_groups; g += step) {
        double col = 0.0;
        for (int k = c.g_ptr[g]; k < c.g_ptr[g + 1]; ++k) col += obj[4 * c.g_mem[k] + 0];
        cv[n + c.g_mem[c.g_ptr[g]]] = col;
    }
    for (int g = first; g < c.n_groups; g += step) {
        const int g0 = c.g_mem[c.g_ptr[g]];
        double col = 0.0;
        for (int k = c.g_ptr[g]; k < c.g_ptr[g + 1]; ++k) col += c.inv_cap[g0 * n + c.g_mem[k]] * img[c.g_mem[k]];
        cv[g0] = col;
        for (int j = c.g_ptr[g] + 1; j < c.g_ptr[g + 1]; ++j) {
            const int gj = c.g_mem[j];
            col = 0.0;
            for (int k = c.g_ptr[g]; k < c.g_ptr[g + 1]; ++k) col += c.inv_cap[gj * n + c.g_mem[k]] * img[c.g_mem[k]];
            cv[n + gj] = col;
        }
    }
    for (int f = first; f < c.n_fv; f += step)
        for (int j = c.f_ptr[f]; j < c.f_ptr[f + 1]; ++j) {
            const int fj = c.f_mem[j];
            double col = 0.0;
            for (int k = c.f_ptr[f]; k < c.f_ptr[f + 1]; ++k) col += c.inv_cap[fj * n + c.f_mem[k]] * img[c.f_mem[k]];
            cv[n + fj] = col;
        }
    __syncthreads();
    for (int i = t; i < 2 * n; i += blockDim.x) {
        double v = 0.0;
        for (int j = 0; j < 2 * n; ++j) v += c.inv_circ[(size_t)i * 2 * n + j] * cv[j];
        if (i < n) {
            obj[4 * i + 2] = v;
            obj_pot[i] = v;
        } else {
            obj[4 * (i - n) + 0] = v;
        }
    }
}

__global__ void k_superpose_dev(const double *__restrict__ phi0, const double *__restrict__ lap,
                                const double *__restrict__ pot, const int32_t *__restrict__ rng, int n_obj, int32_t n,
                                double *__restrict__ out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double v = phi0[i];
    for (int k = 0; k < n_obj; ++k)
        if (!rng || (i >= rng[2 * k] && i < rng[2 * k + 1])) v = v + pot[k] * lap[(size_t)k * n + i];
    out[i] = v;
}

// The end of a step.  counts: [0] slots in use, [1] next particle id, [2] RNG
// step, [3] result row.  Object bookkeeping of Population::update
// (population.h:686-698), a thread per object: current = sum of the absorbed
// charge over the species; charge += current; current /= dt.  The counters
// take the injected slots, and one result row is written: KE, live particles,
// absorbed, injected (kept), PCG iterations, ||r||, then per object current,
// charge, potential.
static_assert(kMaxTags <= 256, "one thread per tag and object");
__global__ void __launch_bounds__(256) k_step_finish(double *rows, int row_len, int64_t *counts, const double *ke,
                                                     const DevState *st, const double *q, int n_species, int injected,
                                                     const int32_t *pcg_i, const double *pcg_d, const int64_t *tags,
                                                     double *obj, int n_obj, double dt) {
    __shared__ long long part[8];
    const int t = threadIdx.x;
    double *r = rows + (size_t)counts[3] * row_len;
    long long absorbed = 0;
    if (t < kMaxTags)
        for (int k = 0; k < n_species; ++k) absorbed += st->absorbed[t][k];
    for (int o = 16; o > 0; o >>= 1) absorbed += __shfl_down_sync(0xffffffffu, absorbed, o);
    if ((t & 31) == 0) part[t >> 5] = absorbed;
    if (t < n_obj) {
        const int64_t tag = tags[t];
        double cur = 0.0;
        if (tag > 0 && tag < kMaxTags)
            for (int sp = 0; sp < n_species; ++sp) cur += (double)st->absorbed[tag][sp] * q[sp];
        const double charge = obj[4 * t + 0] + cur, rate = cur / dt;
        obj[4 * t + 0] = charge;
        obj[4 * t + 1] = rate;
        r[6 + 3 * t] = rate;
        r[7 + 3 * t] = charge;
        r[8 + 3 * t] = obj[4 * t + 2];
    }
    __syncthreads();
    if (t != 0) return;
    long long total = 0;
    for (int w = 0; w < 8; ++w) total += part[w];
    int64_t live = 0, kept = 0;
    for (int k = 0; k < n_species; ++k) live += st->live[k];
    for (int k = 0; k < kMaxSpecies; ++k) kept += st->injected[k];
    r[0] = *ke;
    r[1] = (double)live;
    r[2] = (double)total;
    r[3] = (double)kept;
    r[4] = pcg_i ? (double)pcg_i[0] : 0.0;
    r[5] = pcg_d ? sqrt(pcg_d[0]) : 0.0;
    const int64_t appended = injected ? st->inject_total : 0;
    counts[0] += appended;
    counts[1] += appended;
    counts[2] += 1;
    counts[3] += 1;
}

__global__ void k_set_count(int64_t *counts, const int64_t *cursor, int32_t nc) { counts[0] = cursor[nc]; }

}  // namespace

void launch_circuit_pre(const double *isrc, int n_isrc, double circ_dt, int n_obj, double *obj, double *obj_pot,
                        cudaStream_t s) {
    count_launches(1);
    k_circuit_pre<<<1, 1, 0, s>>>(isrc, n_isrc, circ_dt, n_obj, obj, obj_pot);
}
void launch_circuit_post(const CircuitDev &c, const double *img, double *obj, double *obj_pot, cudaStream_t s) {
    count_launches(1);
    const int threads = c.n <= 16 ? 32 : (c.n <= 128 ? 256 : 512);
    k_circuit_post<<<1, threads, 0, s>>>(c, img, obj, obj_pot);
}
void launch_superpose_dev(const double *phi0, const double *lap, const double *pot, const int32_t *rng, int n_obj,
                         int32_t n, double *out, cudaStream_t s) {
    count_launches(1);
    k_superpose_dev<<<(n + 255) / 256, 256, 0, s>>>(phi0, lap, pot, rng, n_obj, n, out);
}
void launch_step_finish(double *rows, int row_len, int64_t *counts, const double *ke, const DevState *st, const double *q,
                        int n_species, int injected, const int32_t *pcg_i, const double *pcg_d, const int64_t *tags,
                        double *obj, int n_obj, double dt, cudaStream_t s) {
    count_launches(1);
    k_step_finish<<<1, 256, 0, s>>>(rows, row_len, counts, ke, st, q, n_species, injected, pcg_i, pcg_d, tags, obj, n_obj,
                                    dt);
}
void launch_set_count(int64_t *counts, const int64_t *cursor, int32_t nc, cudaStream_t s) {
    count_launches(1);
    k_set_count<<<1, 1, 0, s>>>(counts, cursor, nc);
}

}  // namespace pg
