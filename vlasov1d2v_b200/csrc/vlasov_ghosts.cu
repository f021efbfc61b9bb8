// Ghost elements of the state: the copies around the time loop and the zero ghosts of a right-hand
// side, without passes over the interior (declarations in include/vlasov1d2v.h).
//
// Every (x element, x node) is one velocity plane of (nu + 2) n rows of (nv + 2) n values.  Its
// velocity-ghost values are contiguous runs: the first n rows with the left ghost columns of the
// row after them, the last n rows with the right ghost columns before them, and between each two
// interior rows the right ghost columns of one and the left ghost columns of the next (2 n values).
// At the 32 x 50 x 50, n = 8 state they are 7.5% of the values: copying them to both stage buffers
// and f's two x-ghost slabs takes 31 us where whole-state copies took 246 us (FP64), at 64^3, n = 9 144 against 2359 us: bound by the
// latency of the short scattered runs.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <string>

#include "vlasov_ctx.cuh"

namespace {

// index in a plane of its q-th velocity-ghost value (q < ghost_count)
struct GhostPlane {
    int n, R, rows;   // order, row length (nv + 2) n, rows (nu + 2) n
    int edge;         // values of the first (and of the last) run: (n + 1 row starts) n R + n
    int count;        // velocity-ghost values of the plane
    __host__ __device__ GhostPlane(int n_, int nu, int nv)
        : n(n_), R((nv + 2) * n_), rows((nu + 2) * n_), edge(n_ * (nv + 2) * n_ + n_),
          count(2 * (n_ * (nv + 2) * n_ + n_) + (nu * n_ - 1) * 2 * n_) {}
    __device__ int at(int q) const {
        if (q < edge) return q;
        q -= edge;
        if (q < edge) return (rows - n) * R - n + q;
        q -= edge;
        const int r = q / (2 * n);
        return (n + 1 + r) * R - n + (q - r * 2 * n);
    }
};

constexpr int THREADS = 256;
constexpr int PER = 8;   // values per thread, their loads in flight together

// CTAs: slices of the velocity ghosts of every interior plane, then slices of the 2 n planes of the
// x-ghost slabs
struct GhostGrid {
    int sv, sx;       // slices of a plane's velocity ghosts, of an x-ghost plane
    unsigned ctas;
    explicit GhostGrid(const vl_config &c) {
        const GhostPlane g(c.n, c.nu, c.nv);
        const int64_t per = THREADS * PER;
        sv = (int)((g.count + per - 1) / per);
        sx = (int)(((int64_t)g.rows * g.R + per - 1) / per);
        ctas = (unsigned)(c.nx * c.n * sv + 2 * c.n * sx);
    }
};

// The CTA's values of f: body(position to read, position to write, velocity ghost or x-ghost slab).
// ZERO: every ghost position (the position to read is unused); otherwise the velocity ghosts in
// place and f[nx] -> f[0], f[1] -> f[nx + 1].
template <typename T, bool ZERO>
__global__ void __launch_bounds__(THREADS) ghosts_kernel(T *f, T *sa, T *sb, int nx, int n, int nu, int nv, int sv,
                                                         int sx) {
    const GhostPlane g(n, nu, nv);
    const size_t plane = (size_t)g.rows * g.R;
    const int nint = nx * n * sv;
    const bool vel = (int)blockIdx.x < nint;   // CTA-uniform
    const int k = vel ? blockIdx.x / sv : (blockIdx.x - nint) / sx;
    const int slice = vel ? blockIdx.x - k * sv : (blockIdx.x - nint) - k * sx;
    const int total = vel ? g.count : (int)plane;
    const int i = k % n;
    const size_t dst = (vel ? (size_t)(n + k) : (size_t)((k < n ? 0 : nx + 1) * n + i)) * plane;
    const size_t src = vel ? dst : (size_t)((k < n ? nx : 1) * n + i) * plane;
    int p[PER];
    T v[PER];
#pragma unroll
    for (int u = 0; u < PER; ++u) {
        const int q = slice * (THREADS * PER) + u * THREADS + threadIdx.x;
        p[u] = q < total ? (vel ? g.at(q) : q) : -1;
        if constexpr (!ZERO) {
            if (p[u] >= 0) v[u] = f[src + p[u]];
        }
    }
#pragma unroll
    for (int u = 0; u < PER; ++u) {
        if (p[u] < 0) continue;
        if constexpr (ZERO) {
            f[dst + p[u]] = (T)0;
        } else if (vel) {
            sa[dst + p[u]] = v[u];
            sb[dst + p[u]] = v[u];
        } else {
            f[dst + p[u]] = v[u];
        }
    }
}

template <bool ZERO>
void launch(const vl_config &c, void *f, void *sa, void *sb, cudaStream_t s) {
    const GhostGrid g(c);
    if (c.precision == VL_FP64)
        ghosts_kernel<double, ZERO><<<g.ctas, THREADS, 0, s>>>(static_cast<double *>(f), static_cast<double *>(sa),
                                                               static_cast<double *>(sb), c.nx, c.n, c.nu, c.nv, g.sv,
                                                               g.sx);
    else
        ghosts_kernel<float, ZERO><<<g.ctas, THREADS, 0, s>>>(static_cast<float *>(f), static_cast<float *>(sa),
                                                              static_cast<float *>(sb), c.nx, c.n, c.nu, c.nv, g.sv,
                                                              g.sx);
}

int launched(const char *where) {
    const cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) return VL_OK;
    vl_internal_set_error((std::string(where) + ": " + cudaGetErrorString(e)).c_str());
    return VL_ERR_CUDA;
}

int invalid(const char *msg) {
    vl_internal_set_error(msg);
    return VL_ERR_INVALID;
}

}  // namespace

extern "C" {

VL_API int vl_sync_stage_ghosts(vl_ctx *c, void *f, void *stage_a, void *stage_b, void *stream) {
    if (!c || !f || !stage_a || !stage_b) return invalid("null argument");
    launch<false>(c->cfg, f, stage_a, stage_b, static_cast<cudaStream_t>(stream));
    return launched("ghosts_kernel");
}

VL_API int vl_rhs_whole(vl_ctx *c, const void *f, const double *E, void *out, int xhalo, const double *weights,
                        void *stream) {
    if (!c || !f || !E || !out) return invalid("null argument");
    const int rc = weights ? vl_rhs_weighted(c, f, E, out, xhalo, weights, stream) : vl_rhs(c, f, E, out, xhalo, stream);
    if (rc) return rc;
    launch<true>(c->cfg, out, nullptr, nullptr, static_cast<cudaStream_t>(stream));
    return launched("ghosts_kernel");
}

}  // extern "C"
