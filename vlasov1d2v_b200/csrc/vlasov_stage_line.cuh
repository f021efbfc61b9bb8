// Fused SSP-RK stage kernel in line form (sm_100a): each direction's contraction is done by the
// thread that holds the whole node line, with compile-time coefficients.
//
// Tile = (x element e, u element a, EPT consecutive v elements): COLS = EPT n v-node columns, n x n
// (i, j) rows, n COLS lines of n nodes in each direction, L of them per thread and direction:
//   v lines   (row r = (i, j), element b)    d_k = sum_m up[k][m] F[i][j][b n + m]
//   x lines   (j, column c)                  d_i = sum_m up[i][m] F[m][j][c]
//   u lines   (i, column c)                  d_j = sum_m up[j][m] F[i][m][c]
// A line's n outputs take n loads of the tile (against n loads per output when a thread holds one
// output per line), and every coefficient is a kernel-parameter operand that serves L lines: an FP64
// FMA with a parameter operand runs at half rate when each serves one line (31.6 against 61 FMA per
// clock and SM with two, measured), and in FP32 two lines share the addresses and tile arithmetic
// (n = 9 at 64^3: 16% less per Euler stage than with one).
//
// Per tile:
//   barrier -> v lines (terms to RV), x lines (terms to RX), meanwhile the next tile's nodes travel
//   from global memory into registers (lanes along the contiguous v columns) and then into the other
//   tile buffer, and f^n by cp.async into its own (each thread reads what it copied itself; held in
//   registers, f^n made the combination stage spill: 8% slower at 64^3 n = 9) -> barrier -> u lines, RK
//   combination, store (lanes along the columns)
// Plain loads take any row alignment: one form serves every order and grid in both precisions (the
// tensor-copy forms need rows, or pairs of rows, of 16-byte multiples).
//
// Row strides in shared memory are an odd number of vectors, so the v phase's loads (lanes along
// rows) fall in distinct banks; the x and u phases' lanes run along the columns.
//
// What bounds it: FP32 instruction issue and the next tile's loads (n = 9: 88 / 97 instructions per value in
// an Euler / combination stage, 58% issue active) at 16 resident warps, 128 registers each; more warps at
// fewer registers spill (n = 9 at 5 CTAs per SM 40% slower).  FP64 the latency of loads and shared-memory
// results at 12 warps.  Measured, Euler / combination stage in us, against the form that would serve the case
// otherwise: FP32 n = 9 at 64^3 717 / 854 (paired-row TMA form 872 / 914), with the background split
// 782 / 899 (931 / 994), n = 7 at 24x31x33 33 / 40 (register-pencil kernel 55 / 63); FP64 n = 7 at 24x31x33
// 64 / 90 (generic kernel's cp.async form 117 / 144).
#pragma once

#include <cuda_runtime.h>

#include "vlasov_field_fuse.cuh"
#include "vlasov_kernels.cuh"

namespace vl {

// coefficient tables (kernel parameters)
template <int N, typename T>
struct LineTables {
    T up[N * N];
    T xl[N];        // xi[.][0]:  lift of the left trace
    T xr[N];        // -xi[.][1]: lift of the right trace
    double wu[N];   // w_j / J_u
    double wv[N];   // w_k / J_v
};

// v elements per tile: about 256 lines per direction
template <int N>
struct LineEpt {
    static constexpr int value =
        N == 1 ? 128 : N == 2 ? 64 : N == 3 ? 28 : N == 4 ? 16 : N == 5 ? 10 : N == 6 ? 7 : N == 7 ? 5 : N == 8 ? 4 : N == 9 ? 3 : 2;
};

template <int N, typename T>
struct LineGeom {
    static constexpr int EPT = LineEpt<N>::value;
    static constexpr int COLS = EPT * N;
    static constexpr int LINES = N * COLS;
    static constexpr int L = 2;   // lines per thread and direction
    static constexpr int THREADS = ((LINES + L - 1) / L + 31) / 32 * 32;
    static constexpr int NW = THREADS / 32;
    // elements per vector access of a v line
    static constexpr int VEC = sizeof(T) == 4 ? (N % 4 == 0 ? 4 : N % 2 == 0 ? 2 : 1) : (N % 2 == 0 ? 2 : 1);
    static constexpr int W = ((COLS + VEC - 1) / VEC | 1) * VEC;   // row stride: an odd number of vectors
    static constexpr int BUF = N * N * W;                          // one shared array (elements)
    static constexpr size_t al(size_t b) { return (b + 127) & ~(size_t)127; }
    static constexpr size_t BUF_B = al(sizeof(T) * (size_t)BUF);
    static constexpr size_t HALO_B = al(sizeof(T) * (size_t)N * N);
    static constexpr size_t STAGE_B = 5 * BUF_B + 2 * HALO_B;
    static constexpr size_t RED_B = sizeof(double) * (size_t)LINES;
    static constexpr size_t smem_bytes() { return STAGE_B > RED_B ? STAGE_B : RED_B; }
    // resident CTAs per SM the registers are sized for: a thread holds about 3 L lines
    static constexpr int REGS = (3 * L * N * (int)sizeof(T)) / 4 + 44;
    static constexpr int MINB_R = 65536 / ((REGS + 7) / 8 * 8 * THREADS);
    static constexpr int MINB_S = (int)((227 * 1024) / (smem_bytes() + 1024));
    static constexpr int MINB = MINB_R < MINB_S ? (MINB_R < 1 ? 1 : MINB_R) : MINB_S;
    static_assert(N * N <= THREADS, "one thread per row for the v traces");
    static_assert(MINB_S >= 1, "the tile fits an SM");
};

template <int BYTES>
struct LineVec;
template <>
struct LineVec<4> {
    using V = float;
};
template <>
struct LineVec<8> {
    using V = double;
};
template <>
struct LineVec<16> {
    using V = float4;
};

// n contiguous elements of a v line, VEC at a time
template <int N, int VEC, typename T>
__device__ __forceinline__ void line_load(const T *p, T (&x)[N]) {
    using V = typename LineVec<VEC * (int)sizeof(T)>::V;
    if constexpr (VEC == 1) {
#pragma unroll
        for (int m = 0; m < N; ++m) x[m] = p[m];
    } else {
#pragma unroll
        for (int m = 0; m < N; m += VEC) {
            union {
                V v;
                T s[VEC];
            } u;
            u.v = *reinterpret_cast<const V *>(p + m);
#pragma unroll
            for (int s = 0; s < VEC; ++s) x[m + s] = u.s[s];
        }
    }
}

template <int N, int VEC, typename T>
__device__ __forceinline__ void line_store(T *p, const T (&x)[N]) {
    using V = typename LineVec<VEC * (int)sizeof(T)>::V;
    if constexpr (VEC == 1) {
#pragma unroll
        for (int m = 0; m < N; ++m) p[m] = x[m];
    } else {
#pragma unroll
        for (int m = 0; m < N; m += VEC) {
            union {
                V v;
                T s[VEC];
            } u;
#pragma unroll
            for (int s = 0; s < VEC; ++s) u.s[s] = x[m + s];
            *reinterpret_cast<V *>(p + m) = u.v;
        }
    }
}

// d = up x + lifts of the left trace tl and the right trace tr, for L lines that share each
// coefficient.  z is 0 in a form the compiler cannot see through (FP64): it keeps the coefficient
// loads inside the tile loop, where each serves L FMAs, instead of in registers across it.
template <int N, int L, typename T>
__device__ __forceinline__ void line_contract(const LineTables<N, T> &tb, int z, const T (&x)[L][N], const T (&tl)[L],
                                              const T (&tr)[L], T (&d)[L][N]) {
#pragma unroll
    for (int m = 0; m < N; ++m)
#pragma unroll
        for (int k = 0; k < N; ++k) {
            const T u = tb.up[z + k * N + m];
#pragma unroll
            for (int s = 0; s < L; ++s) d[s][k] = m ? fma(u, x[s][m], d[s][k]) : u * x[s][m];
        }
#pragma unroll
    for (int k = 0; k < N; ++k) {
        const T l = tb.xl[z + k], r = tb.xr[z + k];
#pragma unroll
        for (int s = 0; s < L; ++s) d[s][k] = fma(r, tr[s], fma(l, tl[s], d[s][k]));
    }
}

// Element of the tile (nb elements) that v line b reads: its own, or the first for a line past the last one
// (of a ragged tile, or of the CTA), whose values are dropped.
__host__ __device__ constexpr int line_elem(int b, int nb) { return b < nb ? b : 0; }
// Whether the upwind trace of the tile's element b is the one kept beside the tile, not a neighbour's node
__host__ __device__ constexpr bool line_trace_beside(int b, int nb, bool pos) { return pos ? b == 0 : b == nb - 1; }

template <typename T>
struct LinePair;
template <>
struct LinePair<double> {
    using V = double2;
};
template <>
struct LinePair<float> {
    using V = float2;
};

template <int BYTES>
__device__ __forceinline__ void line_cp(void *dst, const void *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)),
                 "l"(src), "n"(BYTES)
                 : "memory");
}

template <typename T>
__device__ __forceinline__ T line_ld(const char *base, uint32_t off) {
    return *reinterpret_cast<const T *>(base + off);
}

// KIND: stage kind; BG 1: with the background-split RHS tables (FP32).  Global addresses are a
// uniform base plus a 32-bit byte offset inside one x slab (the launch checks the slab's size).
template <int N, typename T, int KIND, int BG>
__global__ void __launch_bounds__(LineGeom<N, T>::THREADS, LineGeom<N, T>::MINB)
stage_line_kernel(const StageArgs a, const __grid_constant__ LineTables<N, T> tb) {
    using G = LineGeom<N, T>;
    using V2 = typename LinePair<T>::V;
    constexpr int EPT = G::EPT, COLS = G::COLS, W = G::W, L = G::L, NN = N * N;
    constexpr uint32_t ES = sizeof(T);
    static_assert(BG == 0 || sizeof(T) == 4, "the background split is a form of FP32 states");
    if (stage_skipped(a)) return;

    extern __shared__ __align__(128) unsigned char line_smem[];
    T *const sTile = reinterpret_cast<T *>(line_smem);   // two tile buffers
    constexpr int TB = (int)(G::BUF_B / sizeof(T));      // elements between them
    T *const sRV = sTile + 2 * TB;
    T *const sRX = sTile + 3 * TB;
    T *const sFn = sTile + 4 * TB;                       // f^n of the tile (combination stages)
    T *const sHalo = sTile + 5 * TB;                     // upwind v trace of every row, two buffers
    constexpr int HB = (int)(G::HALO_B / sizeof(T));
    __shared__ float sE[N];
    __shared__ FuseShared<N, G::THREADS> sFuse;

    const int tid = threadIdx.x;
    const int nx = a.nx, nu = a.nu, nv = a.nv;
    const int V = nv + 2;
    const uint32_t sJ = (uint32_t)(V * N) * ES, sA = sJ * N, sI = sA * (uint32_t)(nu + 2);   // bytes
    const size_t sE_ = (size_t)sI * N;
    const int e = blockIdx.y, Eg = e + 1;
    int El, Er;
    if (a.xhalo == VL_XHALO_PERIODIC) {
        El = (e == 0) ? nx : e;
        Er = (e == nx - 1) ? 1 : e + 2;
    } else {
        El = e;
        Er = e + 2;
    }
    const char *const in = static_cast<const char *>(a.in);
    const char *const inE = in + (size_t)Eg * sE_;
    const char *const fnE = static_cast<const char *>(a.fn) + (size_t)Eg * sE_;
    char *const outE = static_cast<char *>(a.out) + (size_t)Eg * sE_;
    const char *const xL = in + (size_t)El * sE_ + (size_t)sI * (N - 1);   // left neighbour's last node
    const char *const xR = in + (size_t)Er * sE_;                          // right neighbour's first node
    const bool ghost = KIND == KIND_EULER && a.ghost_out != nullptr && (e == 0 || e == nx - 1);   // CTA-uniform
    const V2 *const usv = static_cast<const V2 *>(a.usv);

    // x and u lines (q, c): q the row j of an x line and the x node i of a u line; v lines (row r, b)
    int q[L], c[L], r[L], b[L];
    uint32_t own[L], xrow[L];
    double Ei[L];
#pragma unroll
    for (int s = 0; s < L; ++s) {
        const int l = tid + s * G::THREADS;
        const bool has = l < G::LINES;
        q[s] = has ? l / COLS : 0;
        c[s] = has ? l - q[s] * COLS : 1 << 20;   // (a line past the last: never inside a tile)
        r[s] = has ? l % NN : 0;
        b[s] = has ? l / NN : 1 << 20;
        own[s] = (uint32_t)q[s] * sI + (uint32_t)(c[s] & 0xfffff) * ES;
        xrow[s] = (uint32_t)q[s] * sJ + (uint32_t)(c[s] & 0xfffff) * ES;
    }
    const int hj = tid % N;                                                    // v trace of row tid
    const uint32_t hrow = (uint32_t)(tid / N % N) * sI + (uint32_t)hj * sJ;

    const int nbt = (nv + EPT - 1) / EPT;
    const int GX = gridDim.x;
    const int da = GX / nbt, db = GX - da * nbt;   // tile step of the CTA
    int au = blockIdx.x / nbt, bt = blockIdx.x - au * nbt;
    auto tile_off = [&](int ta, int tb_) { return (uint32_t)(ta + 1) * sA + (uint32_t)((tb_ * EPT + 1) * N) * ES; };
    auto tile_cols = [&](int tb_) { return min(EPT, nv - tb_ * EPT) * N; };

    T F[L][N];
    T halo = (T)0;
    auto load_tile = [&](int ta, int tb_) {
        const uint32_t off = tile_off(ta, tb_);
        const int ncol = tile_cols(tb_);
#pragma unroll
        for (int s = 0; s < L; ++s)
            if (c[s] < ncol) {
                const char *o = inE + (off + own[s]);
#pragma unroll
                for (int m = 0; m < N; ++m, o += sJ) F[s][m] = *reinterpret_cast<const T *>(o);
            }
        if (tid < NN) {
            const bool vpos = usv[(ta + 1) * N + hj].y >= (T)0;
            halo = line_ld<T>(inE, off + hrow + (vpos ? (uint32_t)-(int)ES : (uint32_t)ncol * ES));
        }
    };
    auto store_tile = [&](int p, int ncol) {
#pragma unroll
        for (int s = 0; s < L; ++s)
            if (c[s] < ncol) {
                T *d = sTile + p * TB + q[s] * (N * W) + c[s];
#pragma unroll
                for (int m = 0; m < N; ++m) d[m * W] = F[s][m];
            }
        if (tid < NN) sHalo[p * HB + tid] = halo;
    };
    double mk[L];   // sum over a line's outputs of (w_j / J_u) out
#pragma unroll
    for (int s = 0; s < L; ++s) mk[s] = 0.0;

    int cur = 0;
    if (!stage_gate(a)) return;
    if (au < nu) load_tile(au, bt);
    if (KIND != KIND_RHS && a.ff.mode != FUSE_NONE) {
        // E at this x element while the first tile travels; the tile buffers are the scratch
        if (!field_prologue<N, G::THREADS, KIND == KIND_EULER>(a, e, reinterpret_cast<double *>(line_smem), sFuse)) return;
    }
    const double accel = a.accel, bfield = a.bfield;
    const double dtd = (KIND == KIND_RHS) ? 0.0 : a.ff.mode != FUSE_NONE ? sFuse.dt : *a.dt;
    const T dtT = (T)dtd, c0 = (T)a.c0, c1 = (T)a.c1, c2dt = (T)(a.c2 * dtd);
    const T jx = (T)a.jx, ju = (T)a.ju, jv = (T)a.jv;
    if constexpr (BG == 1) {
        if (tid < N) sE[tid] = (float)(a.ff.mode != FUSE_NONE ? sFuse.E[tid] : a.E[Eg * N + tid]);   // (read after the first barrier)
    }
#pragma unroll
    for (int s = 0; s < L; ++s) Ei[s] = a.ff.mode != FUSE_NONE ? sFuse.E[q[s]] : a.E[Eg * N + q[s]];
    if (au < nu) store_tile(0, tile_cols(bt));

    while (au < nu) {
        const int ncol = tile_cols(bt), nb = ncol / N;
        const uint32_t toff = tile_off(au, bt);
        int an = au + da, bn = bt + db;   // next tile
        if (bn >= nbt) {
            bn -= nbt;
            ++an;
        }
        if constexpr (KIND == KIND_COMBINE) {   // each thread copies the values that it reads itself
#pragma unroll
            for (int s = 0; s < L; ++s)
                if (c[s] < ncol) {
                    const char *o = fnE + (toff + own[s]);
                    T *d = sFn + q[s] * (N * W) + c[s];
#pragma unroll
                    for (int m = 0; m < N; ++m, o += sJ) line_cp<sizeof(T)>(d + m * W, o);
                }
            asm volatile("cp.async.commit_group;" ::: "memory");
        }
        if (an < nu) load_tile(an, bn);
        const int z0 = sizeof(T) == 8 ? (bt == a.never ? 1 : 0) : 0;
        const int z1 = sizeof(T) == 8 ? (au == a.never ? 1 : 0) : 0;
        const int z2 = sizeof(T) == 8 ? (bn == a.never ? 1 : 0) : 0;
        // speeds and neighbour traces
        T ux[L], svl[L], xn[L], un[L];
        double sd[L];
        float beu[L], brb[L];
#pragma unroll
        for (int s = 0; s < L; ++s) {
            ux[s] = usv[(au + 1) * N + q[s]].x;
            svl[s] = usv[(au + 1) * N + r[s] % N].y;
            xn[s] = un[s] = (T)0;
            sd[s] = 0.0;
            beu[s] = brb[s] = 0.0f;
            if (c[s] < ncol) {
                if (ux[s] >= (T)0)
                    xn[s] = line_ld<T>(xL, toff + xrow[s]);
                else
                    xn[s] = line_ld<T>(xR, toff + xrow[s]);
                sd[s] = accel * (Ei[s] + bfield * a.v_nodes[(bt * EPT + 1) * N + c[s]]);
                un[s] = line_ld<T>(inE, toff + own[s] + (sd[s] >= 0.0 ? (uint32_t)-(int)sJ : sA));
                if constexpr (BG == 1) {
                    beu[s] = line_ld<float>(reinterpret_cast<const char *>(a.bg_eu), toff + xrow[s]);
                    brb[s] = line_ld<float>(reinterpret_cast<const char *>(a.bg_rb), toff + xrow[s]);
                }
            }
        }
        const T *const sIn = sTile + cur * TB;
        const T *const sH = sHalo + cur * HB;
        __syncthreads();   // the tile is in shared memory; the previous one's terms are consumed

        T x[L][N], d[L][N], tl[L], tr[L];
        // v lines
#pragma unroll
        for (int s = 0; s < L; ++s) {
            const int bb = line_elem(b[s], nb);
            const T *p = sIn + r[s] * W + bb * N;
            line_load<N, G::VEC>(p, x[s]);
            const bool pos = svl[s] >= (T)0;
            const bool beside = line_trace_beside(bb, nb, pos);
            const int to = pos ? -1 : N;
            // FP64 selects the value (n = 7 at 24x31x33 64 us per Euler stage, 66 the other way), FP32 its
            // address (n = 9 at 64^3 852 us per combination stage, 871 the other way)
            T t;
            if constexpr (sizeof(T) == 8) {
                t = beside ? sH[r[s]] : p[to];
            } else {
                const T *pn = beside ? sH + r[s] : p + to;
                t = *pn;
            }
            tl[s] = pos ? t : x[s][0];
            tr[s] = pos ? x[s][N - 1] : t;
        }
        line_contract(tb, z0, x, tl, tr, d);
#pragma unroll
        for (int s = 0; s < L; ++s) {
            const T sv = svl[s] * jv;
#pragma unroll
            for (int k = 0; k < N; ++k) d[s][k] *= sv;
            if (b[s] < nb) line_store<N, G::VEC>(sRV + r[s] * W + b[s] * N, d[s]);
        }
        // x lines
#pragma unroll
        for (int s = 0; s < L; ++s) {
            const T *p = sIn + q[s] * W + (c[s] < ncol ? c[s] : 0);
#pragma unroll
            for (int m = 0; m < N; ++m) x[s][m] = p[m * (N * W)];
            const bool pos = ux[s] >= (T)0;
            tl[s] = pos ? xn[s] : x[s][0];
            tr[s] = pos ? x[s][N - 1] : xn[s];
        }
        line_contract(tb, z1, x, tl, tr, d);
#pragma unroll
        for (int s = 0; s < L; ++s)
            if (c[s] < ncol) {
                const T uj = ux[s] * jx;
                T *p = sRX + q[s] * W + c[s];
#pragma unroll
                for (int i = 0; i < N; ++i) {
                    if constexpr (BG == 1)   // + RHS of the x-independent background
                        p[i * (N * W)] = fmaf(uj, d[s][i], fmaf(sE[i], beu[s], brb[s]));
                    else
                        p[i * (N * W)] = uj * d[s][i];
                }
            }
        if (an < nu) store_tile(cur ^ 1, tile_cols(bn));
        __syncthreads();   // the v and x terms are complete

        // u lines, RK combination, store
        if constexpr (KIND == KIND_COMBINE) asm volatile("cp.async.wait_group 0;" ::: "memory");
#pragma unroll
        for (int s = 0; s < L; ++s) {
            const T *p = sIn + q[s] * (N * W) + (c[s] < ncol ? c[s] : 0);
#pragma unroll
            for (int m = 0; m < N; ++m) x[s][m] = p[m * W];
            const bool pos = sd[s] >= 0.0;
            tl[s] = pos ? un[s] : x[s][0];
            tr[s] = pos ? x[s][N - 1] : un[s];
        }
        line_contract(tb, z2, x, tl, tr, d);
#pragma unroll
        for (int s = 0; s < L; ++s)
            if (c[s] < ncol) {
                const T sp = (T)sd[s] * ju;
                const int w = q[s] * (N * W) + c[s];
                char *o = outE + (toff + own[s]);
#pragma unroll
                for (int j = 0; j < N; ++j, o += sJ) {
                    const T rr = fma(sp, d[s][j], sRX[w + j * W]) + sRV[w + j * W];
                    T v;
                    if constexpr (KIND == KIND_RHS)
                        v = rr;
                    else if constexpr (KIND == KIND_EULER)
                        v = fma(dtT, rr, x[s][j]);
                    else
                        v = rk_combine(c0, c1, c2dt, sFn[w + j * W], x[s][j], rr);
                    *reinterpret_cast<T *>(o) = v;
                    mk[s] = fma(tb.wu[j], (double)v, mk[s]);
                }
                if (ghost) {   // periodic x-ghost refresh of f (Distribution.swap_ghost_cells_of_array)
                    char *g0 = static_cast<char *>(a.ghost_out) + (toff + own[s]);
#pragma unroll
                    for (int j = 0; j < N; ++j) {
                        if (e == nx - 1) *reinterpret_cast<T *>(g0 + j * sJ) = x[s][j];
                        if (e == 0) *reinterpret_cast<T *>(g0 + (size_t)(nx + 1) * sE_ + j * sJ) = x[s][j];
                    }
                }
            }
        au = an;
        bt = bn;
        cur ^= 1;
    }

    if (a.partials == nullptr) return;
    // moment partial of x node i: its COLS columns, one warp per node, fixed order
    __syncthreads();
    double *sRed = reinterpret_cast<double *>(line_smem);
#pragma unroll
    for (int s = 0; s < L; ++s) {
        const int l = tid + s * G::THREADS;
        if (l < G::LINES) sRed[l] = tb.wv[c[s] % N] * mk[s];
    }
    __syncthreads();
    const int lane = tid & 31;
    for (int i = tid >> 5; i < N; i += G::NW) {
        dd s = {0.0, 0.0};
        for (int cc = lane; cc < COLS; cc += 32) s = dd_gather(s, dd{sRed[i * COLS + cc], 0.0});
        for (int off = 16; off > 0; off >>= 1) s = dd_gather(s, dd_shfl_xor(s, off));
        if (lane == 0) a.partials[((size_t)e * GX + blockIdx.x) * N + i] = s.hi + s.lo;
    }
}

}  // namespace vl
