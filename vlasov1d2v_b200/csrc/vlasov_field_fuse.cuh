// The field solve and the loop bookkeeping at the start of a stage kernel (sm_100a).
//
// In its convolution form (vlasov_field_conv.cuh) a solve at one x element is n sums over the nx n
// nodes, so every CTA of a stage kernel forms E at its own x element before its tiles: the partials of
// all nodes, their mean, n dot products with the element's rows of KE (read from L2 by each CTA, once).
// The loop then has three launches a step and no field kernel between them; the first tile's copies
// travel meanwhile.  The CTA with blockIdx.x = 0 of each x element writes the step's last E and phi.
//
// The step's first stage also does the bookkeeping of the step before it (energy and max |a E| of its
// field, dt, time, the history entry, whether this step runs): every CTA repeats it, from the control
// record of the previous step, and the grid's first CTA writes the next record.  Records alternate
// between two places, and so do the moment partials a kernel reads and the ones it writes, because
// the CTAs of one kernel do not wait for each other; field_close_kernel brings the loop state up to
// date at the end of a batch.
//
// Bound by latency: partials, two block reductions, the dot products, 2 to 4 us where a separate solve and
// the gap before it cost 6 to 8.  Per step, separate solves against this (whose stages are also launched as
// the one before ends): 64 -> 52.5 us at 16x20x20 n = 6, 68 -> 53.5 at 16^3 n = 8, 32 -> 22.6 at 8x12x12 n = 4,
// 585 -> 575 at 32x50x50 n = 8 (FP64).  Not in FP32 at n = 2, whose small CTAs sum the partials slowly
// (24x30x30 45 -> 52 us); a called instead of an inlined prologue costs the n = 8 stage 7 us of 160 in stack
// frames.
#pragma once

#include "vlasov_field_conv.cuh"
#include "vlasov_kernels.cuh"

namespace vl {

// shared values of the prologue
template <int N, int NT>
struct FuseShared {
    double E[N];               // E at the x nodes of the CTA's element
    double dt;
    dd rho[NT / 32], en[NT / 32];
    double mx[NT / 32];
    int go;
};

// doubles of scratch: the density at every x node, rows of n | 1
__host__ __device__ constexpr size_t field_fuse_scratch(int nx, int n) { return sizeof(double) * (size_t)nx * (n | 1); }

// the record of the step that follows `c`: bookkeeping of the step that ran with c (energy, max |a E| of
// its field), then the promotion to the next step
__device__ __forceinline__ void fuse_close_step(const FieldFuse &f, vl_run_state &c, double energy, double max_e,
                                                double accel, double bfield, bool keeper) {
    const double dtn = adapted_dt(f, accel, bfield, max_e);
    c.steps += 1;
    c.time += dtn;
    c.dt_next = dtn;
    const bool finite = isfinite(energy) && isfinite(dtn);
    c.active_next = (c.time < f.st->final_time) && (c.steps < f.st->max_steps) && finite;
    if (!keeper) return;
    const int cap = f.st->hist_capacity;
    if (cap > 0) {
        const int slot = (int)((c.steps - 1) % cap);
        if (f.st->energy_hist) f.st->energy_hist[slot] = energy;
        if (f.st->time_hist) f.st->time_hist[slot] = c.time;
        if (f.st->dt_hist) f.st->dt_hist[slot] = dtn;
    }
    if (!finite) atomicOr(&f.st->status, 1);
}

__device__ __forceinline__ void fuse_load(vl_run_state &c, const vl_run_state *s) {
    c.dt = s->dt;
    c.dt_next = s->dt_next;
    c.time = s->time;
    c.steps = s->steps;
    c.active = s->active;
    c.active_next = s->active_next;
}

__device__ __forceinline__ void fuse_store(vl_run_state *s, const vl_run_state &c) {
    s->dt = c.dt;
    s->dt_next = c.dt_next;
    s->time = c.time;
    s->steps = c.steps;
    s->active = c.active;
    s->active_next = c.active_next;
}

// E at x element e into sh.E, dt into sh.dt; false when the step does not run (all threads of the grid
// agree).  scratch: field_fuse_scratch bytes of shared memory.
// CONTROL: the step's first stage (FUSE_FIRST, FUSE_STEP), which keeps the books; the others are FUSE_FIELD.
template <int N, int NT, bool CONTROL>
__device__ __forceinline__ bool field_prologue(const StageArgs &a, int e, double *scratch, FuseShared<N, NT> &sh) {
    constexpr int NW = NT / 32, RS = N | 1, S = field_conv_stride(N);
    const FieldFuse &f = a.ff;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nx = a.nx, nn = nx * N;
    const bool close = CONTROL && f.mode == FUSE_STEP;
    vl_run_state c;
    if (CONTROL && tid == 0) fuse_load(c, f.ctl_in);
    // a step after the loop's end (the one that finds the end closes the last step, below): its record is the
    // last one's.  Read beside the field and tested after it, the word costs a running step nothing (32 steps
    // after the end at 20x27x29 n = 7 FP32 436 -> 200 us, 352 with separate solves)
    const int ran = close ? f.ctl_in->active : 1;
    dd loc = {0.0, 0.0}, en = {0.0, 0.0};
    double mx = 0.0;
    if (close) {
        for (int p = tid; p < nn; p += NT) {
            const double ev = f.E_prev[N + p];
            en = dd_gather(en, dd{f.xw[p % N] * (ev * ev), 0.0});
            mx = fmax(mx, fabs(a.accel * ev));
        }
        if (ran == 0) {
            if (tid == 0 && blockIdx.x == 0 && blockIdx.y == 0) fuse_store(f.ctl_out, c);
            return false;
        }
    }
    for (int p = tid; p < nn; p += NT) {
        const int e2 = p / N, i = p - e2 * N;
        const double *src = f.partials + (size_t)e2 * f.G * N + i;
        dd s = {0.0, 0.0};
#pragma unroll 8
        for (int g = 0; g < f.G; ++g) s = dd_gather(s, dd{src[(size_t)g * N], 0.0});
        const double rho = s.hi + s.lo;
        scratch[e2 * RS + i] = rho;
        loc = dd_gather(loc, dd{rho, 0.0});
    }
    for (int off = 16; off > 0; off >>= 1) loc = dd_gather(loc, dd_shfl_xor(loc, off));
    if (close) {
        for (int off = 16; off > 0; off >>= 1) {
            en = dd_gather(en, dd_shfl_xor(en, off));
            mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, off));
        }
    }
    if (lane == 0) {
        sh.rho[warp] = loc;
        if constexpr (CONTROL) {
            sh.en[warp] = en;
            sh.mx[warp] = mx;
        }
    }
    __syncthreads();
    dd t = sh.rho[0];
#pragma unroll
    for (int w = 1; w < NW; ++w) t = dd_gather(t, sh.rho[w]);
    const double mean = (t.hi + t.lo) / (double)nn;
    if (tid == 0) {
        if constexpr (CONTROL) {
            const bool keeper = blockIdx.x == 0 && blockIdx.y == 0;
            if (close && c.active) {
                dd es = sh.en[0];
                double m = sh.mx[0];
#pragma unroll
                for (int w = 1; w < NW; ++w) {
                    es = dd_gather(es, sh.en[w]);
                    m = fmax(m, sh.mx[w]);
                }
                fuse_close_step(f, c, 0.5 * (es.hi + es.lo), m, a.accel, a.bfield, keeper);
            }
            c.active = c.active_next;
            if (c.active) c.dt = c.dt_next;
            if (keeper) fuse_store(f.ctl_out, c);
            sh.go = c.active;
            sh.dt = c.dt;
        } else {
            sh.go = 1;
            sh.dt = *a.dt;
        }
    }
    // E[e, j] = kappa sum K[e - e'][j][.] . (mean - rho[e']): `parts` neighbouring lanes a node
    constexpr int parts = 32 * N <= NT ? 32 : 16 * N <= NT ? 16 : 8 * N <= NT ? 8 : 4 * N <= NT ? 4 : 2 * N <= NT ? 2 : 1;
    const int j = tid / parts, part = tid % parts;
    const bool in = j < N;
    const bool writer = f.E_out != nullptr && blockIdx.x == 0;   // CTA-uniform
    auto dot = [&](const double *__restrict__ K) {
        double s0 = 0.0, s1 = 0.0;
        if (in) {
            for (int e2 = part; e2 < nx; e2 += parts) {
                int d = e - e2;
                if (d < 0) d += nx;
                const double *kr = K + d * S + j * N;
                const double *rr = scratch + e2 * RS;
#pragma unroll
                for (int m = 0; m < N; m += 2) {
                    s0 = fma(__ldg(kr + m), mean - rr[m], s0);
                    if (m + 1 < N) s1 = fma(__ldg(kr + m + 1), mean - rr[m + 1], s1);
                }
            }
        }
        double s = s0 + s1;
        for (int off = 1; off < parts; off *= 2) s += __shfl_xor_sync(0xffffffffu, s, off);
        return a.ff.kappa * s;
    };
    const double er = dot(f.KE);
    const double pr = writer && f.phi_out != nullptr ? dot(f.KP) : 0.0;
    if (in && part == 0) sh.E[j] = er;
    __syncthreads();
    if (sh.go == 0) return false;
    if (in && part == 0 && !isfinite(er)) atomicOr(f.status, 1);
    if (writer && in && part == 0) {
        const int p = e * N + j;
        f.E_out[N + p] = er;
        if (e == nx - 1) f.E_out[j] = er;        // E[0] = E[-2]
        if (e == 0) f.E_out[nn + N + j] = er;    // E[-1] = E[1]
        if (f.phi_out != nullptr) f.phi_out[p] = pr;
    }
    return true;
}

// end of a batch: the bookkeeping of its last step and the loop state
static __global__ void __launch_bounds__(256) field_close_kernel(const FieldFuse f, int nx, int n, double accel,
                                                                 double bfield) {
    __shared__ dd s_en[8];
    __shared__ double s_mx[8];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nn = nx * n;
    vl_run_state c;
    fuse_load(c, f.ctl_in);
    dd en = {0.0, 0.0};
    double mx = 0.0;
    for (int p = tid; p < nn; p += 256) {
        const double ev = f.E_prev[n + p];
        en = dd_gather(en, dd{f.xw[p % n] * (ev * ev), 0.0});
        mx = fmax(mx, fabs(accel * ev));
    }
    for (int off = 16; off > 0; off >>= 1) {
        en = dd_gather(en, dd_shfl_xor(en, off));
        mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, off));
    }
    if (lane == 0) {
        s_en[warp] = en;
        s_mx[warp] = mx;
    }
    __syncthreads();
    if (tid != 0) return;
    if (c.active) {
        dd es = s_en[0];
        double m = s_mx[0];
        for (int w = 1; w < 8; ++w) {
            es = dd_gather(es, s_en[w]);
            m = fmax(m, s_mx[w]);
        }
        fuse_close_step(f, c, 0.5 * (es.hi + es.lo), m, accel, bfield, true);
    }
    fuse_store(f.st, c);
}

}  // namespace vl
