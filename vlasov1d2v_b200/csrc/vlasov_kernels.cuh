// Device kernels of the 1D2V DG Vlasov-Poisson hot path (sm_100a).
//
// State layout in HBM: the reference's ghost-inclusive C-order array
//     f[X][n][U][n][V][n]   X = nx+2, U = nu+2, V = nv+2      (main/grid.py:262-268)
// i.e. a plain 3-D node grid (X n) x (U n) x (V n) whose innermost axis (v) is contiguous.
// A DG element is an n^3 block; its six face traces are the adjacent node planes.
//
// Kernels
//   stage kernel    (vlasov_stage.cuh) one fused SSP-RK stage or a bare RHS.
//   moment_kernel   standalone zeroth velocity moment, one CTA per (x element, x node).
//   field_kernel    one CTA: moment partials -> density -> mean-subtracted charge -> forward
//                   high-order DFT -> spectral E and phi -> inverse DFT at the LGL nodes ->
//                   periodic ghosts; optionally energy, adaptive dt and the loop bookkeeping.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "vlasov1d2v.h"

namespace vl {

constexpr int NMAX = 10;

enum StageKind : int { KIND_EULER = 0, KIND_COMBINE = 1, KIND_RHS = 2 };

// Per-order coefficient tables passed by value as kernel parameters: the contraction loops are
// fully unrolled, so every table entry is a compile-time offset into the parameter constant
// bank and becomes an FMA operand without a load instruction.
template <typename T>
struct StageTables {
    T up[NMAX * NMAX];     // up[i][j]        (main/basis.py:176-188)
    T xi[NMAX * 2];        // xi[i][face]     (main/basis.py:110)
    double qw[NMAX * NMAX];  // w_j w_k / (J_u J_v)  (main/grid.py:297-301)
    // up with the own-trace lift folded in, per upwind direction:
    //   speed >= 0: d = sum_m upP[i][m] f[m] + xi[i][0] * (left neighbour trace)
    //   speed <  0: d = sum_m upM[i][m] f[m] - xi[i][1] * (right neighbour trace)
    T upP[NMAX * NMAX];
    T upM[NMAX * NMAX];
    // the velocity weights factored: w_j w_k / (J_u J_v) = (w_j / J_u) (w_k / J_v)
    double wu[NMAX];
    double wv[NMAX];
};

// Field solve and loop bookkeeping inside a stage kernel (vlasov_field_fuse.cuh)
enum FuseMode : int {
    FUSE_NONE = 0,    // E is given
    FUSE_FIELD = 1,   // E from the moment partials of the stage's input
    FUSE_FIRST = 2,   // the same, first stage of a batch's first step: promotes the loop state
    FUSE_STEP = 3,    // the same, first stage of a later step: closes the step before it first
};
struct FieldFuse {
    int mode;
    int G;                       // partials per x node
    const double *partials;      // [nx][G][n] of the stage's input (not the buffer the stage writes)
    const double *KE, *KP;       // convolution tables
    double kappa;
    double *E_out, *phi_out;     // written by the CTAs with blockIdx.x = 0, or null
    int *status;                 // bit 0: non-finite E
    const vl_run_state *ctl_in;  // control record of the step before (FUSE_FIRST: the loop state)
    vl_run_state *ctl_out;       // control record of this step
    vl_run_state *st;            // the loop state: limits, history ring, status
    const double *E_prev;        // the field of the step before (its last solve)
    const double *xw;
    double dx, du, dv, umax, vmax, courant;
};

struct StageArgs {
    const void *in;        // stage input (ghost-inclusive)
    const void *fn;        // f^n for KIND_COMBINE
    void *out;             // output (interior written)
    void *ghost_out;       // when not null (KIND_EULER on f): periodic x-ghost refresh of f
    const double *E;       // [(nx+2) n]
    const double *dt;      // device scalar
    const vl_run_state *state;  // when not null, the kernel returns if !state->active
    const double *u_nodes; // [(nu+2) n]
    const void *usv;       // [(nu+2) n] pairs (u, a (-B u)) in the state precision: the x and v
                           // flux speeds per u node (n = 8 kernel)
    const double *v_nodes; // [(nv+2) n]
    double *partials;      // [nx][G][n] moment partials of out, or null
    const double *tables;  // device copy: up [n n], xi [n 2], qw [n n] (per-lane indexed reads)
    int *err;              // device error word: bit 1 = a bounded wait timed out
    int nx, nu, nv;
    int xhalo;
    int kind;
    double c0, c1, c2;
    double accel, bfield, jx, ju, jv;
    // Background split (FP32 mixed form): when bg_rb is not null the state holds the deviation
    // from an x-independent background f0(u, v), and the RHS of f0 is added per node:
    //   r0 = E_i * bg_eu + bg_rb,
    // tables in the velocity-slab layout [U][n][V][n] (index a sA + j sJ + v column).
    const float *bg_rb;
    const float *bg_eu;
    // FP32 n = 8 kernel: its per-u-node speed table holds u J_x and a (-B u) J_v with the
    // context's Jacobians; a call with other direction weights (jx, jv above) scales them by
    // jx / J_x and jv / J_v (the RHS kind only; the RK stages use the context's Jacobians)
    double sx, sv;
    FieldFuse ff;
    int grid_g;  // CTAs per x element (0: the context's own choice; host side)
    int pdl;     // launched while the kernel before it still runs (stage_gate)
    int never;   // line-form kernel: a value that no tile index takes (-1)
};


// Start of a stage kernel, before its first read of what other kernels write (and after the set-up that
// needs none of it): with `pdl` the kernel is launched as the last CTAs of the one before exit, so wait
// until that one is complete and its writes are visible.  Every CTA waits, so kernels complete in order.
// Hides the launch and the set-up: 24.1 -> 22.2 us per step at 8x12x12 n = 4, 55.7 -> 53.5 at 16^3 n = 8,
// 583 -> 578 at 32x50x50 n = 8.  The next kernel is not let in earlier: its CTAs then take slots as they
// free up, unevenly over the SMs (597 us there, 509 against 497 at 32x62x62 n = 6).
// Returns false when the loop has ended.
__device__ __forceinline__ bool stage_gate(const StageArgs &a) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    return a.pdl == 0 || a.state == nullptr || a.state->active != 0;
}

// Without `pdl` the loop's state is up to date when the kernel starts: a stage of a loop that has ended
// returns before its set-up (the generic kernel clears 95 KB of shared memory per CTA: 32 steps after
// the end at 64^3 n = 9 1.09 ms with the test at the gate, 0.88 before the set-up).
__device__ __forceinline__ bool stage_skipped(const StageArgs &a) {
    return a.pdl == 0 && a.state != nullptr && a.state->active == 0;
}

// SSP-RK combination stage c0 f^n + c1 s + (c2 dt) r with c0 + c1 = 1 (main/timestep.py:157-163,
// :174-182).  FP64 evaluates the reference's expression as written; FP32 evaluates
// f^n + c1 (s - f^n) + (c2 dt) r, whose weights of f^n and s sum to exactly 1: with rounded
// weights, float(1/3) + float(2/3) = 1 + 3e-8 would amplify every mode by 3e-8 per step.
template <typename T>
__device__ __forceinline__ T rk_combine(T c0, T c1, T c2dt, T fn, T s, T r) {
    if constexpr (sizeof(T) == 4)
        return fma(c2dt, r, fma(c1, s - fn, fn));
    else
        return fma(c2dt, r, fma(c1, s, c0 * fn));
}

// launch configuration of a stage kernel; `attr` is the caller's storage
inline cudaLaunchConfig_t stage_config(const StageArgs &a, dim3 grid, int threads, size_t smem, cudaStream_t s,
                                       cudaLaunchAttribute *attr) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    if (a.pdl) {
        attr->id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr->val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
    }
    return cfg;
}

// ----------------------------------------------------------------------------------------------
// error-free transformation helpers for the FP64 moment reductions
// ----------------------------------------------------------------------------------------------
struct dd {
    double hi, lo;
};

__device__ __forceinline__ dd two_sum(double a, double b) {
    double s = a + b;
    double bp = s - a;
    double e = (a - (s - bp)) + (b - bp);
    return {s, e};
}

__device__ __forceinline__ dd dd_add(dd a, dd b) {
    dd s = two_sum(a.hi, b.hi);
    double lo = s.lo + a.lo + b.lo;
    dd r = two_sum(s.hi, lo);
    return r;
}

// compensated sum: the high part is one addition per term, the rounding errors are gathered beside it
// (dd_add renormalises each term: four more additions on the chain)
__device__ __forceinline__ dd dd_gather(dd a, dd b) {
    const double s = a.hi + b.hi;
    const double bp = s - a.hi;
    return {s, ((a.hi - (s - bp)) + (b.hi - bp)) + (a.lo + b.lo)};
}

__device__ __forceinline__ dd dd_shfl_xor(dd v, int off) {
    return {__shfl_xor_sync(0xffffffffu, v.hi, off), __shfl_xor_sync(0xffffffffu, v.lo, off)};
}

__device__ __forceinline__ dd shfl_down_dd(dd v, int off) {
    dd r;
    r.hi = __shfl_down_sync(0xffffffffu, v.hi, off);
    r.lo = __shfl_down_sync(0xffffffffu, v.lo, off);
    return r;
}

// Stepper.adapt_time_step of get_max_speeds (main/timestep.py:231-242): dt from the largest |a E|; `a` has
// the set-up's umax, vmax, dx, du, dv and courant
template <typename A>
__device__ __forceinline__ double adapted_dt(const A &a, double accel, double bfield, double max_e) {
    const double ab = accel * bfield;
    const double s0 = fabs(a.umax);
    const double s1 = fabs(max_e + fabs(ab * a.vmax));
    const double s2 = fabs(accel * fabs(bfield * a.umax));
    return a.courant / (((s0 / a.dx) + (s1 / a.du)) + (s2 / a.dv));
}

// block-wide double-double sum (all threads call); result valid in every thread
__device__ __forceinline__ double block_sum_dd_rt(double v, double c, dd *scratch) {
    dd s = {v, c};
    for (int off = 16; off > 0; off >>= 1) s = dd_add(s, shfl_down_dd(s, off));
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    __syncthreads();
    if (lane == 0) scratch[warp] = s;
    __syncthreads();
    dd t = scratch[0];
    for (int w = 1; w < (int)(blockDim.x >> 5); ++w) t = dd_add(t, scratch[w]);
    return t.hi + t.lo;
}

struct MomentArgs {
    const void *f;
    double *out;
    int G;
    int nx, nu, nv;
    double qw[NMAX * NMAX];
};

// ----------------------------------------------------------------------------------------------
// standalone moment: grid (G, nx).  CTA (g, e) sums its share of the nu nv velocity elements of x slab e
// for every x node i and writes out[(e G + g) n + i] -- the layout of the stage kernels' moment partials.
// A share is a run of columns (u element, v node) of the slab; columns go to threads with a stride that
// is a multiple of n, so each thread sees one v node k and keeps its row of weights w_j w_k / (J_u J_v)
// in registers.  Bound by HBM on large grids (with the reduction over CTAs, 32x50x50 n = 8: FP64 66 us with
// shares of whole u elements, 56 now; FP32 45 -> 34; 64^3 n = 9 279 -> 237), by latency on small ones, where
// the sums over the threads were most of the time: node by node, each five shuffles, two barriers and a
// chain over the warps; now a warp per node over all threads' sums at once (16^3 n = 8 15.5 -> 5.9 us,
// 16x20x20 n = 6 13.4 -> 6.0).
// ----------------------------------------------------------------------------------------------
constexpr int MOMENT_THREADS = 256;
// 2 resident CTAs per SM leave 128 registers per thread, room for most of a column's n x n loads
// in flight at once (at 4 CTAs, 64 registers, the loads issued a few at a time and the kernel ran
// at half the HBM rate, bound by load latency)
constexpr int MOMENT_CTAS_PER_SM = 2;

template <int N, typename T>
__global__ void __launch_bounds__(MOMENT_THREADS, MOMENT_CTAS_PER_SM) moment_kernel(const MomentArgs a) {
    const T *__restrict__ f = static_cast<const T *>(a.f);
    constexpr int CT = (MOMENT_THREADS / N) * N;   // column threads (stride keeps k fixed)
    constexpr int NW = MOMENT_THREADS / 32;
    __shared__ double part[N][MOMENT_THREADS];
    const int g = blockIdx.x, Gn = gridDim.x, e = blockIdx.y;
    const int nu = a.nu, nv = a.nv;
    const int U = nu + 2, V = nv + 2;
    const int sJ = V * N, sA = sJ * N, sI = sA * U;
    const int ncol = nv * N, cells = nu * nv;
    const int lo = (int)(((long long)g * cells) / Gn) * N, hi = (int)(((long long)(g + 1) * cells) / Gn) * N;
    const T *const slab = f + (size_t)(e + 1) * ((size_t)sI * N) + sA + N;   // first interior column
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int k = tid % N;
    double w[N];
#pragma unroll
    for (int j = 0; j < N; ++j) w[j] = a.qw[j * N + k];
    double acc[N];
#pragma unroll
    for (int i = 0; i < N; ++i) acc[i] = 0.0;
    if (tid < CT) {
        for (int q = lo + tid; q < hi; q += CT) {
            const int au = q / ncol;
            const T *pi = slab + (size_t)au * sA + (q - au * ncol);
            // the row strides are opaque here: kept across columns, the offsets of the n x n rows take the
            // registers that the loads in flight need (32x50x50 n = 8 100 us)
            int si = sI, sj = sJ;
            asm volatile("" : "+r"(si), "+r"(sj));
#pragma unroll
            for (int i = 0; i < N; ++i) {
                double s = 0.0;
#pragma unroll
                for (int j = 0; j < N; ++j) s = fma(w[j], (double)pi[i * si + j * sj], s);
                acc[i] += s;
            }
        }
    }
#pragma unroll
    for (int i = 0; i < N; ++i) part[i][tid] = acc[i];
    __syncthreads();
    for (int i = warp; i < N; i += NW) {
        dd s = {part[i][lane], 0.0};
#pragma unroll
        for (int m = 1; m < NW; ++m) s = dd_gather(s, dd{part[i][lane + 32 * m], 0.0});
        for (int off = 16; off > 0; off >>= 1) s = dd_gather(s, dd_shfl_xor(s, off));
        if (lane == 0) a.out[((size_t)e * Gn + g) * N + i] = s.hi + s.lo;
    }
}

// rho[e][i] = sum over g of the partials [e][g][i] (double-double, fixed order)
static __global__ void moment_reduce_kernel(const double *__restrict__ partials, double *__restrict__ rho,
                                     int nx, int G, int n) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= nx * n) return;
    const int e = p / n, i = p - e * n;
    const double *src = partials + (size_t)e * G * n + i;
    dd s = {0.0, 0.0};
#pragma unroll 8
    for (int g = 0; g < G; ++g) s = dd_gather(s, dd{src[(size_t)g * n], 0.0});
    rho[p] = s.hi + s.lo;
}

// ----------------------------------------------------------------------------------------------
// field solve (the kernel itself is vlasov_field.cuh): arguments, loop gating, reductions
// ----------------------------------------------------------------------------------------------
enum FieldMode : int {
    FIELD_REQUIRE_ACTIVE = 1,  // return if !state->active
    FIELD_PROMOTE = 2,         // start of a step: active <- active_next, dt <- dt_next
    FIELD_RECORD = 4,          // after stage 2: energy, dt_next, time, steps, history
};

struct FieldArgs {
    const double *partials;   // [nx][G][n] (rho = sum over g), or null when charge_in is used
    int G;
    const double *charge_in;  // [nx][n] mean-subtracted charge density (vl_poisson), or null
    double *E;                // [(nx+2) n]
    double *phi;              // [nx n] or null
    vl_run_state *state;      // or null
    int mode;
    const double2 *ell;       // [n][M]   T[e, j, m] = phase[e, m] ell[j, m]
    const double2 *phase;     // [nx][M]  exp(-i k_m mid_e)
    const double2 *qnode;     // [n][M]   exp(i k_m x_{e,j}) = conj(phase[e, m]) qnode[j, m]
    const double *k;          // [M]
    const double *xw;         // [n]
    int nx, n, M;
    double kappa, dx, length, accel, bfield, umax, vmax, du, dv, courant;
    // 1: each CTA first copies the phase-table entries it reads in its loops into shared memory
    // (field_prefetch_bytes more dynamic shared memory; the arithmetic is unchanged)
    int prefetch;
    // convolution form (vlasov_field_conv.cuh): [nx][field_conv_stride(n)] tables, or null
    const double *KE, *KP;
};

constexpr int SCALAR_THREADS = 256;           // threads of the single-CTA scalar kernel
constexpr int FIELD_MAX_NODES = 64 * NMAX;    // nx * n capacity of the shared buffers
constexpr int FIELD_MAX_MODES = 2 * 160 + 1;  // M capacity

__device__ __forceinline__ double block_sum_dd(double v, double c, dd *scratch) {
    return block_sum_dd_rt(v, c, scratch);
}

__device__ __forceinline__ double block_max(double v, double *scratch) {
    for (int off = 16; off > 0; off >>= 1) v = fmax(v, __shfl_down_sync(0xffffffffu, v, off));
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    __syncthreads();
    if (lane == 0) scratch[warp] = v;
    __syncthreads();
    double t = scratch[0];
    for (int w = 1; w < (int)(blockDim.x >> 5); ++w) t = fmax(t, scratch[w]);
    return t;
}

// returns false when this step is inactive (all threads agree)
__device__ __forceinline__ bool field_gate(const FieldArgs &a, bool first_cta) {
    vl_run_state *st = a.state;
    if (st == nullptr) return true;
    if (a.mode & FIELD_PROMOTE) {
        const int go = st->active_next;
        if (first_cta && threadIdx.x == 0) {
            st->active = go;
            if (go) st->dt = st->dt_next;
        }
        return go != 0;
    }
    if (a.mode & FIELD_REQUIRE_ACTIVE) return st->active != 0;
    return true;
}

// energy + dt from a given E (vl_field_energy / vl_adapt_dt / vl_run_state_init)
struct ScalarArgs {
    const double *E;
    const double *xw;
    int nx, n;
    double accel, bfield, umax, vmax, dx, du, dv, courant;
    double *energy;      // or null
    double *dt;          // or null
    vl_run_state *init;  // or null: initialise the loop state
    double final_time;
    int64_t max_steps;
    double *eh, *th, *dh;
    int cap;
};

// Latency: a few terms a thread, then one sum and one maximum over the CTA, both in one pass (two serial
// passes over 32 warps' parts took 8.3 us, this 2.4)
static __global__ void __launch_bounds__(SCALAR_THREADS) scalars_kernel(const ScalarArgs a) {
    constexpr int NW = SCALAR_THREADS / 32;
    __shared__ dd s_sum[NW];
    __shared__ double s_max[NW];
    const int nn = a.nx * a.n;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    dd esq = {0.0, 0.0};
    double emax = 0.0;
    // energy over the interior rows E[1:-1]; max |a E| over all rows incl. ghosts
    for (int p = threadIdx.x; p < nn + 2 * a.n; p += SCALAR_THREADS) {
        const double er = a.E[p];
        emax = fmax(emax, fabs(a.accel * er));
        if (p >= a.n && p < nn + a.n) esq = dd_gather(esq, dd{a.xw[p % a.n] * (er * er), 0.0});
    }
    for (int off = 16; off > 0; off >>= 1) {
        esq = dd_gather(esq, dd_shfl_xor(esq, off));
        emax = fmax(emax, __shfl_xor_sync(0xffffffffu, emax, off));
    }
    if (lane == 0) {
        s_sum[warp] = esq;
        s_max[warp] = emax;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        dd t = s_sum[0];
        double maxE = s_max[0];
#pragma unroll
        for (int w = 1; w < NW; ++w) {
            t = dd_gather(t, s_sum[w]);
            maxE = fmax(maxE, s_max[w]);
        }
        const double energy = 0.5 * (t.hi + t.lo);
        const double dtn = adapted_dt(a, a.accel, a.bfield, maxE);
        if (a.energy) *a.energy = energy;
        if (a.dt) *a.dt = dtn;
        if (a.init) {
            vl_run_state *st = a.init;
            st->dt = dtn;
            st->dt_next = dtn;
            st->time = 0.0;
            st->final_time = a.final_time;
            st->steps = 0;
            st->max_steps = a.max_steps;
            st->active = 0;
            const bool finite = isfinite(energy) && isfinite(dtn);
            st->status = finite ? 0 : 1;
            st->active_next = (0.0 < a.final_time) && (0 < a.max_steps) && finite;
            st->hist_capacity = a.cap;
            st->energy_hist = a.eh;
            st->time_hist = a.th;
            st->dt_hist = a.dh;
        }
    }
}

}  // namespace vl
