// Spectral Poisson solve (main/elliptic.py:117-145) as one real block convolution (sm_100a).
//
// The solve is linear in the charge, and on the uniform periodic x grid the element phases of the
// forward and inverse high-order DFT (main/basis.py:204-228) combine to conj(ph[e, m]) ph[e', m],
// which depends on d = (e - e') mod nx only.  So with rhs = kappa (mean rho - rho)
//   E[e, j]   = sum_{e', j'} KE[e - e'][j][j'] rhs[e', j'],
//   KE[d][j][j'] = Re sum_{k_m != 0} (dx / L) (i / k_m) conj(ph[d, m]) ph[0, m] q[j, m] ell[j', m],
// phi likewise with -1 / k_m^2.  The tables of nx n^2 values are built on the device when the
// context is created (field_conv_table_kernel; only for phases that pass the host's check of the
// uniform periodic grid -- other tables keep the transform form of vlasov_field.cuh).
//
// A solve is then nx n products and sums per node (6.6e4 at 32 elements of n = 8, where the two
// transforms over M = 159 modes take 1.6e5 and a cluster barrier between them), with no exchange
// between the CTAs: CTA r sums the moment partials of every node, then forms E at its elements.
// Solves without bookkeeping launch one CTA per x element; the step's last solve (energy, dt, loop
// state) is one cluster of FC CTAs that sends its energies and maxima to rank 0 through distributed
// shared memory.  Both are bound by the latency of their chain: loop state and partials, the mean,
// the products, the store.  A standalone solve takes 3.2 us at 32 x 50 x 50, n = 8 and 4.1 us at 64^3,
// n = 9 (graph of repeated solves), against 8.3 us and 15.7 us in the transform form.
#pragma once

#include <cooperative_groups.h>

#include "vlasov_field.cuh"
#include "vlasov_kernels.cuh"

namespace vl {

constexpr int FV_THREADS = 256;

// values per element distance d, an odd number: the parts of a sum, lanes of a warp at consecutive d,
// read distinct shared-memory banks
__host__ __device__ constexpr int field_conv_stride(int n) { return (n * n) | 1; }
__host__ __device__ constexpr int field_conv_elems(int nx, int n) { return (nx * field_conv_stride(n) + 1) & ~1; }
__host__ __device__ constexpr size_t field_conv_smem(int nx, int n, bool phi) {
    return sizeof(double) * (size_t)(phi ? 2 : 1) * field_conv_elems(nx, n);
}

// KE and KP: 8 lanes share a value's sum over the modes (compensated; 40 us with one thread per value
// at 16 elements of n = 8, 11 us now)
static __global__ void __launch_bounds__(256) field_conv_table_kernel(double *KE, double *KP, const double2 *ell,
                                                                      const double2 *phase, const double2 *qnode,
                                                                      const double *k, int nx, int n, int M, double dx,
                                                                      double length) {
    constexpr int LANES = 8;
    const int p = (blockIdx.x * blockDim.x + threadIdx.x) / LANES, lane = threadIdx.x % LANES;
    const int S = field_conv_stride(n);
    const int d = p / S, jj = p - d * S;
    dd se = {0.0, 0.0}, sp = {0.0, 0.0};
    if (d < nx && jj < n * n) {
        const int j = jj / n, j2 = jj - j * n;
        for (int m = lane; m < M; m += LANES) {
            const double km = k[m];
            if (km == 0.0) continue;
            const double2 a = phase[(size_t)d * M + m], b = phase[m];
            const double2 h = make_double2(a.x * b.x + a.y * b.y, a.x * b.y - a.y * b.x);   // conj(a) b
            const double2 q = qnode[(size_t)j * M + m], l = ell[(size_t)j2 * M + m];
            const double2 g = make_double2(q.x * l.x - q.y * l.y, q.x * l.y + q.y * l.x);
            const double re = h.x * g.x - h.y * g.y, im = h.x * g.y + h.y * g.x;
            const double ik = 1.0 / km;
            se = dd_gather(se, dd{-(im * ik), 0.0});          // Re (i z / k)
            sp = dd_gather(sp, dd{-(re * ik) * ik, 0.0});     // Re (-z / k^2)
        }
    }
    for (int off = 1; off < LANES; off *= 2) {
        se = dd_gather(se, dd_shfl_xor(se, off));
        sp = dd_gather(sp, dd_shfl_xor(sp, off));
    }
    if (lane == 0 && p < field_conv_elems(nx, n)) {
        KE[p] = ((se.hi + se.lo) * dx) / length;
        KP[p] = ((sp.hi + sp.lo) * dx) / length;
    }
}

// sum over e' = part, part + parts, ... of K[e - e'][j][.] . rhs[e'][.]
template <int N>
__device__ __forceinline__ double conv_dot(const double *K, const double *rhs, int nx, int e, int j, int part,
                                           int parts) {
    constexpr int S = field_conv_stride(N), RS = N | 1;
    double s0 = 0.0, s1 = 0.0;
    for (int e2 = part; e2 < nx; e2 += parts) {
        int d = e - e2;
        if (d < 0) d += nx;
        const double *kr = K + d * S + j * N;
        const double *rr = rhs + e2 * RS;
#pragma unroll
        for (int m = 0; m < N; m += 2) {
            s0 = fma(kr[m], rr[m], s0);
            if (m + 1 < N) s1 = fma(kr[m + 1], rr[m + 1], s1);
        }
    }
    return s0 + s1;
}

__device__ __forceinline__ double conv_dot_n(int n, const double *K, const double *rhs, int nx, int e, int j, int part,
                                             int parts) {
    switch (n) {
        case 1: return conv_dot<1>(K, rhs, nx, e, j, part, parts);
        case 2: return conv_dot<2>(K, rhs, nx, e, j, part, parts);
        case 3: return conv_dot<3>(K, rhs, nx, e, j, part, parts);
        case 4: return conv_dot<4>(K, rhs, nx, e, j, part, parts);
        case 5: return conv_dot<5>(K, rhs, nx, e, j, part, parts);
        case 6: return conv_dot<6>(K, rhs, nx, e, j, part, parts);
        case 7: return conv_dot<7>(K, rhs, nx, e, j, part, parts);
        case 8: return conv_dot<8>(K, rhs, nx, e, j, part, parts);
        case 9: return conv_dot<9>(K, rhs, nx, e, j, part, parts);
        default: return conv_dot<10>(K, rhs, nx, e, j, part, parts);
    }
}

// CTA `rank` of R: E at the elements [rank nx / R, (rank + 1) nx / R).  RECORD: the R = FC CTAs form
// a cluster, and rank 0 keeps the loop state.  FV_THREADS threads.
template <bool RECORD>
__device__ __forceinline__ void field_conv_body(const FieldArgs &a, int rank, int R) {
    namespace cg = cooperative_groups;
    constexpr int NW = FV_THREADS / 32;
    __shared__ double s_rhs[2 * FIELD_MAX_NODES];   // [e][n | 1]
    __shared__ double s_out[FIELD_MAX_NODES];   // E at this CTA's nodes
    __shared__ dd s_red[NW];
    __shared__ dd s_rank_energy[FC];            // rank 0: every rank's energy, max |a E|, non-finite flag
    __shared__ double s_rank_max[FC];
    __shared__ int s_rank_bad[FC];
    extern __shared__ __align__(16) double fv_dyn[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int n = a.n, nx = a.nx, nn = nx * n, RS = n | 1;
    const bool want_phi = a.phi != nullptr;
    const int kelems = field_conv_elems(nx, n);
    double *sKE = fv_dyn, *sKP = fv_dyn + kelems;
    for (int q = tid; q < kelems / 2; q += FV_THREADS) {
        field_cp16(sKE + 2 * q, a.KE + 2 * q);
        if (want_phi) field_cp16(sKP + 2 * q, a.KP + 2 * q);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    if constexpr (RECORD) cg::this_cluster().barrier_arrive();   // (waited for before the remote stores)

    // loop state of the bookkeeping, read early by its one thread
    vl_run_state *st = a.state;
    const bool keeper = RECORD && rank == 0 && tid == 0;
    int64_t st_steps = 0, st_max = 0;
    double st_time = 0.0, st_final = 0.0;
    if (keeper) {
        st_steps = st->steps;
        st_max = st->max_steps;
        st_time = st->time;
        st_final = st->final_time;
    }

    // charge: every CTA, identical (the partials of one node are summed in the order of the CTAs)
    dd loc = {0.0, 0.0};
    if (a.charge_in != nullptr) {
        for (int p = tid; p < nn; p += FV_THREADS) {
            const int e = p / n;
            s_rhs[e * RS + (p - e * n)] = a.kappa * a.charge_in[p];
        }
    } else {
        for (int p = tid; p < nn; p += FV_THREADS) {
            const int e = p / n, i = p - e * n;
            const double *src = a.partials + (size_t)e * a.G * n + i;
            dd s = {0.0, 0.0};
#pragma unroll 8
            for (int g = 0; g < a.G; ++g) s = dd_gather(s, dd{src[(size_t)g * n], 0.0});
            const double rho = s.hi + s.lo;
            s_rhs[e * RS + i] = rho;
            loc = dd_gather(loc, dd{rho, 0.0});
        }
    }
    // every CTA takes the same decision: rank 0 writes only active and dt here, a promoting solve
    // reads active_next (written by the step's last solve)
    bool go = true;
    if (st != nullptr) {
        if (a.mode & FIELD_PROMOTE) {
            go = st->active_next != 0;
            if (rank == 0 && tid == 0) {
                st->active = go ? 1 : 0;
                if (go) st->dt = st->dt_next;
            }
        } else if (a.mode & FIELD_REQUIRE_ACTIVE) {
            go = st->active != 0;
        }
    }
    if (!go) {   // the whole grid returns: no copy is left in flight, no barrier waiting
        asm volatile("cp.async.wait_all;" ::: "memory");
        if constexpr (RECORD) cg::this_cluster().barrier_wait();
        return;
    }
    if (a.charge_in == nullptr) {
        for (int off = 16; off > 0; off >>= 1) loc = dd_gather(loc, dd_shfl_xor(loc, off));
        if (lane == 0) s_red[warp] = loc;
        __syncthreads();
        dd t = s_red[0];
#pragma unroll
        for (int w = 1; w < NW; ++w) t = dd_gather(t, s_red[w]);
        const double mean = (t.hi + t.lo) / (double)nn;
        for (int p = tid; p < nn; p += FV_THREADS) {   // (each thread's own nodes)
            const int e = p / n, q = e * RS + (p - e * n);
            s_rhs[q] = a.kappa * (mean - s_rhs[q]);
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();   // charge and tables

    // E (and phi) at this CTA's nodes: `parts` neighbouring lanes share a node's sum
    const int e0 = rank * nx / R, e1 = (rank + 1) * nx / R;
    const int count = (e1 - e0) * n;
    int parts = 1;
    while (2 * parts * count <= FV_THREADS && parts < 32) parts *= 2;
    bool bad = false;
    for (int o0 = 0; o0 < count; o0 += FV_THREADS / parts) {
        const int o = o0 + tid / parts, part = tid & (parts - 1);
        const bool in = o < count;
        const int e = e0 + (in ? o / n : 0), j = in ? o % n : 0;
        double er = in ? conv_dot_n(n, sKE, s_rhs, nx, e, j, part, parts) : 0.0;
        double pr = in && want_phi ? conv_dot_n(n, sKP, s_rhs, nx, e, j, part, parts) : 0.0;
        for (int off = 1; off < parts; off *= 2) {
            er += __shfl_xor_sync(0xffffffffu, er, off);
            if (want_phi) pr += __shfl_xor_sync(0xffffffffu, pr, off);
        }
        if (in && part == 0) {
            const int p = e * n + j;
            a.E[n + p] = er;
            if (e == nx - 1) a.E[j] = er;        // E[0] = E[-2]
            if (e == 0) a.E[nn + n + j] = er;    // E[-1] = E[1]
            if (want_phi) a.phi[p] = pr;
            s_out[o] = er;
            bad |= !isfinite(er);
        }
    }
    const int any_bad = __syncthreads_or(bad ? 1 : 0);
    if constexpr (!RECORD) {
        if (st != nullptr && any_bad && tid == 0) atomicOr(&st->status, 1);
    } else {
        // energy and max |a E| of this CTA's nodes, to rank 0
        cg::cluster_group cluster = cg::this_cluster();
        dd part_e = {0.0, 0.0};
        double part_max = 0.0;
        if (warp == 0) {
            for (int o = lane; o < count; o += 32) {
                const double ev = s_out[o];
                part_e = dd_gather(part_e, dd{a.xw[o % n] * (ev * ev), 0.0});
                part_max = fmax(part_max, fabs(a.accel * ev));
            }
            for (int off = 16; off > 0; off >>= 1) {
                part_e = dd_gather(part_e, dd_shfl_xor(part_e, off));
                part_max = fmax(part_max, __shfl_xor_sync(0xffffffffu, part_max, off));
            }
        }
        cluster.barrier_wait();   // every CTA of the cluster has started
        if (tid == 0) {
            cluster.map_shared_rank(s_rank_energy, 0)[rank] = part_e;
            cluster.map_shared_rank(s_rank_max, 0)[rank] = part_max;
            cluster.map_shared_rank(s_rank_bad, 0)[rank] = any_bad;
        }
        cluster.sync();   // rank 0 holds every rank's values
        if (!keeper) return;
        dd etot = s_rank_energy[0];
        double maxE = s_rank_max[0];
        int bad_any = s_rank_bad[0];
#pragma unroll
        for (int r = 1; r < FC; ++r) {
            etot = dd_gather(etot, s_rank_energy[r]);
            maxE = fmax(maxE, s_rank_max[r]);
            bad_any |= s_rank_bad[r];
        }
        const double energy = 0.5 * (etot.hi + etot.lo);
        const double dtn = adapted_dt(a, a.accel, a.bfield, maxE);
        const int64_t steps = st_steps + 1;
        const double time = st_time + dtn;
        st->dt_next = dtn;
        st->time = time;
        st->steps = steps;
        const int cap = st->hist_capacity;
        if (cap > 0) {
            const int slot = (int)((steps - 1) % cap);
            if (st->energy_hist) st->energy_hist[slot] = energy;
            if (st->time_hist) st->time_hist[slot] = time;
            if (st->dt_hist) st->dt_hist[slot] = dtn;
        }
        const bool finite = isfinite(energy) && isfinite(dtn) && !bad_any;
        if (!finite) st->status |= 1;
        st->active_next = (time < st_final) && (steps < st_max) && finite;
    }
}

static __global__ void __launch_bounds__(FV_THREADS) field_conv_kernel(const FieldArgs a) {
    field_conv_body<false>(a, blockIdx.x, gridDim.x);
}

static __global__ void __launch_bounds__(FV_THREADS) field_conv_record_kernel(const FieldArgs a) {
    field_conv_body<true>(a, blockIdx.x, FC);
}

}  // namespace vl
