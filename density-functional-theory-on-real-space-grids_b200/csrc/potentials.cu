// (c2, d, s1) The Kohn--Sham potentials on the device (src/cdft/scf/step.py:224-313): the Hartree
// split n = sum_a c_a exp(-2 Z_a s_a) + n_s, the pointwise XC kernels, the node- and grid-side
// assembly of the lumped weights omega~ (quadrature.py:711-753) fused with the functional, and the
// deterministic row sums and finite-difference gradient the energies need.

#include "common.cuh"
#include "xc_device.cuh"

namespace cdftb {

namespace {

constexpr int MAX_ATOMS = 8;

inline unsigned blocks_for(int64_t n, int threads) {
    const int64_t b = ceil_div(n, threads);
    return static_cast<unsigned>(b < 148 * 32 ? b : 148 * 32);
}

#define GRID_STRIDE(i, n) \
    for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < (n); i += static_cast<int64_t>(gridDim.x) * blockDim.x)

// k -> (system g, point i) of a (batch, np) array; 32-bit division when the whole index fits.
__device__ __forceinline__ void split_index(int64_t k, int64_t np, bool narrow, int64_t& g, int64_t& i) {
    if (narrow) {
        const unsigned uk = static_cast<unsigned>(k), un = static_cast<unsigned>(np), ug = uk / un;
        g = ug;
        i = uk - ug * un;
    } else {
        g = k / np;
        i = k - g * np;
    }
}

__global__ void xc_lda_kernel(const double* __restrict__ n, int64_t p, double* __restrict__ e, double* __restrict__ v) {
    GRID_STRIDE(i, p) {
        double ei, vi;
        xc::lda_vwn(n[i], ei, vi);
        e[i] = ei;
        v[i] = vi;
    }
}

__global__ void xc_pbe_kernel(const double* __restrict__ n, const double* __restrict__ sigma, int64_t p,
                              double* __restrict__ e, double* __restrict__ v, double* __restrict__ vs) {
    GRID_STRIDE(i, p) {
        double ei, vi, vsi;
        xc::pbe(n[i], sigma[i], ei, vi, vsi);
        e[i] = ei;
        v[i] = vi;
        vs[i] = vsi;
    }
}

// c = S^{-1} (nucleus_f2 * rho(R_a)) by Gaussian elimination with partial pivoting, one system per
// thread (step.py:240-242; n_atoms <= MAX_ATOMS). rho_at_nuclei and coef: the system's own na values.
__device__ void solve_cusp_coefficients(const double* rho_at_nuclei, const double* __restrict__ nucleus_f2,
                                        const double* __restrict__ overlap, int na, double* coef) {
    double a[MAX_ATOMS][MAX_ATOMS + 1];
    for (int i = 0; i < na; ++i) {
        for (int j = 0; j < na; ++j) a[i][j] = overlap[i * na + j];
        a[i][na] = nucleus_f2[i] * rho_at_nuclei[i];
    }
    for (int c = 0; c < na; ++c) {
        int piv = c;
        for (int r = c + 1; r < na; ++r)
            if (fabs(a[r][c]) > fabs(a[piv][c])) piv = r;
        if (piv != c)
            for (int k = 0; k <= na; ++k) {
                const double t = a[c][k];
                a[c][k] = a[piv][k];
                a[piv][k] = t;
            }
        for (int r = c + 1; r < na; ++r) {
            const double f = a[r][c] / a[c][c];
            for (int k = c; k <= na; ++k) a[r][k] -= f * a[c][k];
        }
    }
    for (int r = na - 1; r >= 0; --r) {
        double v = a[r][na];
        for (int k = r + 1; k < na; ++k) v -= a[r][k] * coef[k];
        coef[r] = v / a[r][r];
    }
}

__global__ void cusp_coefficients_kernel(const double* __restrict__ rho_at_nuclei, const double* __restrict__ nucleus_f2,
                                         const double* __restrict__ overlap, int na, int batch,
                                         double* __restrict__ coef) {
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g < batch)
        solve_cusp_coefficients(rho_at_nuclei + int64_t(g) * na, nucleus_f2, overlap, na, coef + int64_t(g) * na);
}

// The same from the density: rho(R_a) = L_a (n / f^2) over the 8^3 points around each nucleus, a CTA per
// system, two points per thread. Only these 512 quotients are needed: forming rho on the grid first, to
// interpolate it, took a pass over all points (32 systems at 65^3: 60 us for the three launches; this
// kernel 5 us).
__global__ void __launch_bounds__(256) cusp_coefficients_density_kernel(
    const double* __restrict__ n, const double* __restrict__ f2, const int* __restrict__ base,
    const double* __restrict__ w1d, const double* __restrict__ nucleus_f2, const double* __restrict__ overlap, int na,
    int64_t np, int ny, int nz, double* __restrict__ coef) {
    __shared__ double red[8][MAX_ATOMS], rho[MAX_ATOMS];
    const int64_t g = blockIdx.x;
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    const int a = t >> 6, b = (t >> 3) & 7, c = t & 7;  // taps (a and a + 4, b, c)
    for (int k = 0; k < na; ++k) {
        const double* w = w1d + k * 24;
        const int64_t bx = base[k * 3] - 3 + a, by = base[k * 3 + 1] - 3 + b, bz = base[k * 3 + 2] - 3 + c;
        const int64_t i0 = (bx * ny + by) * nz + bz, i1 = i0 + 4 * int64_t(ny) * nz;
        double v = (w[8 + b] * w[16 + c]) * fma(w[a], n[g * np + i0] / f2[i0], w[a + 4] * (n[g * np + i1] / f2[i1]));
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
        if (lane == 0) red[warp][k] = v;
    }
    __syncthreads();
    if (t < na) {
        double v = 0.0;
        for (int w = 0; w < 8; ++w) v += red[w][t];
        rho[t] = v;
    }
    __syncthreads();
    if (t == 0) solve_cusp_coefficients(rho, nucleus_f2, overlap, na, coef + g * na);
}

// rho = n / f^2 and n_smooth = n - sum_a c_a exp(-2 Z_a s_a) (step.py:235-244).
__global__ void hartree_split_kernel(const double* __restrict__ n, const double* __restrict__ f2,
                                     const double* __restrict__ cusp_grid, const double* __restrict__ coef, int na,
                                     int64_t np, int batch, double* __restrict__ rho, double* __restrict__ n_smooth) {
    const bool narrow = np * batch <= 0xffffffffll;
    GRID_STRIDE(k, np * batch) {
        int64_t g, i;
        split_index(k, np, narrow, g, i);
        const double nv = n[k];
        rho[k] = nv / f2[i];
        double cusp = 0.0;
        for (int a = 0; a < na; ++a) {
            const double t = coef[g * na + a] * cusp_grid[a * np + i];
            cusp = (a == 0) ? t : cusp + t;
        }
        n_smooth[k] = nv - cusp;
    }
}

// Node side of potentials(), LDA, at node i of system g: x_H = w f2 vH, x_xc = w f2 v_xc (the lift inputs
// of the lumped Hartree and XC weights, x [batch][2][m]); returns e_w = w e_xc (the node part of the XC
// energy). fields: rho_node (batch x m) followed by vsmooth_node (batch x m).
__device__ __forceinline__ double node_lda(const double* __restrict__ fields, int64_t m,
                                           const double* __restrict__ weights, const double* __restrict__ f2n,
                                           const double* __restrict__ v1s_node, const double* __restrict__ coef, int na,
                                           int batch, int64_t g, int64_t i, double* __restrict__ x) {
    const double rho_node = fields[g * m + i];
    double vh = 0.0;
    for (int a = 0; a < na; ++a) {
        const double t = coef[g * na + a] * v1s_node[a * m + i];
        vh = (a == 0) ? t : vh + t;
    }
    vh = vh + fields[(batch + g) * m + i];
    const double f2 = f2n[i];
    const double nn = f2 * rho_node;
    double e, v;
    xc::lda_vwn(nn, e, v);
    const double w = weights[i];
    x[g * 2 * m + i] = w * (f2 * vh);
    x[g * 2 * m + m + i] = w * (f2 * v);
    return w * e;
}

__global__ void node_lda_kernel(const double* __restrict__ fields, int64_t m, const double* __restrict__ weights,
                                const double* __restrict__ f2n, const double* __restrict__ v1s_node,
                                const double* __restrict__ coef, int na, int batch, double* __restrict__ x,
                                double* __restrict__ e_w) {
    const bool narrow = m * batch <= 0xffffffffll;
    GRID_STRIDE(k, m * batch) {
        int64_t g, i;
        split_index(k, m, narrow, g, i);
        e_w[g * m + i] = node_lda(fields, m, weights, f2n, v1s_node, coef, na, batch, g, i, x);
    }
}

// Grid side, LDA, at point i of system g: hartree_w = L_H + far_w (f2 vH), xc_w = L_xc + far_w (f2 v_xc),
// effective = (hartree_w + xc_w) / omega (step.py:249-303); terms = (hartree_w rho, xc_w rho,
// far_w e_xc) for the energy sums; v_hartree = sum_a c_a v1s_a + v_smooth.
struct GridLda {
    const double *n, *rho, *f2, *far_w, *mass, *v_smooth, *v1s_grid, *coef;
    int na;
    const double* lifted;
    int64_t np;
    double *effective, *v_hartree, *v_xc;
};

__device__ __forceinline__ void grid_lda(const GridLda& p, int64_t g, int64_t i, double terms[3]) {
    const int64_t np = p.np, k = g * np + i;
    double vh = 0.0;
    for (int a = 0; a < p.na; ++a) {
        const double t = p.coef[g * p.na + a] * p.v1s_grid[a * np + i];
        vh = (a == 0) ? t : vh + t;
    }
    vh = vh + p.v_smooth[k];
    double e, v;
    xc::lda_vwn(p.n[k], e, v);
    const double fw = p.far_w[i];
    const double f = p.f2[i];
    const double hw = p.lifted[g * 2 * np + i] + fw * (f * vh);
    const double xw = p.lifted[g * 2 * np + np + i] + fw * (f * v);
    const double r = p.rho[k];
    p.effective[k] = (hw + xw) / p.mass[i];
    p.v_hartree[k] = vh;
    if (p.v_xc) p.v_xc[k] = v;
    terms[0] = hw * r;
    terms[1] = xw * r;
    terms[2] = fw * e;
}

__global__ void grid_lda_kernel(const GridLda p, int batch, double* __restrict__ terms) {
    const bool narrow = p.np * batch <= 0xffffffffll;
    GRID_STRIDE(k, p.np * batch) {
        int64_t g, i;
        split_index(k, p.np, narrow, g, i);
        double t[3];
        grid_lda(p, g, i, t);
#pragma unroll
        for (int j = 0; j < 3; ++j) terms[(g * 3 + j) * p.np + i] = t[j];
    }
}

// Both sides with their energy sums: a CTA takes sum_points points of one system and leaves one partial
// per sum, lda_energies_kernel adds a system's partials in order. The terms never reach memory, where
// writing them and summing the rows took 48 of a point's 112 bytes; what is left is bound by the FP64 issue
// of the functional (32 systems at 65^3: 196 us with the sums, 193 and 50 us apart).
constexpr int kSumThreads = 256;

// Points of a CTA: one per thread until the launch has 16 CTAs per SM, then up to 8 (the sums over the
// block and the partials are then a small part).
int64_t sum_points(int64_t n, int64_t batch) {
    const int64_t k = n * batch / (int64_t(kSumThreads) * 148 * 16);
    return kSumThreads * (k < 1 ? 1 : k > 8 ? 8 : k);
}

template <int N>
__device__ __forceinline__ void block_sums(double v[N], double* sums) {
    __shared__ double red[kSumThreads / 32][N];
#pragma unroll
    for (int j = 0; j < N; ++j) {
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) v[j] += __shfl_down_sync(0xffffffffu, v[j], off);
        if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5][j] = v[j];
    }
    __syncthreads();
    if (threadIdx.x < N) {
        double t = 0.0;
        for (int w = 0; w < kSumThreads / 32; ++w) t += red[w][threadIdx.x];
        sums[threadIdx.x] = t;
    }
}

__global__ void __launch_bounds__(kSumThreads) node_lda_sums_kernel(
    const double* __restrict__ fields, int64_t m, int64_t points, int64_t chunks, const double* __restrict__ weights,
    const double* __restrict__ f2n, const double* __restrict__ v1s_node, const double* __restrict__ coef, int na,
    int batch, double* __restrict__ x, double* __restrict__ partial) {
    const int64_t g = blockIdx.x / chunks, i0 = (blockIdx.x - g * chunks) * points;
    double sum[1] = {0.0};
    for (int64_t i = i0 + threadIdx.x; i < i0 + points && i < m; i += kSumThreads)
        sum[0] += node_lda(fields, m, weights, f2n, v1s_node, coef, na, batch, g, i, x);
    block_sums<1>(sum, partial + blockIdx.x);
}

__global__ void __launch_bounds__(kSumThreads) grid_lda_sums_kernel(const GridLda p, int64_t points, int64_t chunks,
                                                                    double* __restrict__ partial) {
    const int64_t g = blockIdx.x / chunks, i0 = (blockIdx.x - g * chunks) * points;
    double sum[3] = {0.0, 0.0, 0.0};
    for (int64_t i = i0 + threadIdx.x; i < i0 + points && i < p.np; i += kSumThreads) {
        double t[3];
        grid_lda(p, g, i, t);
#pragma unroll
        for (int j = 0; j < 3; ++j) sum[j] += t[j];
    }
    block_sums<3>(sum, partial + int64_t(blockIdx.x) * 3);
}

// energies [batch][3] = (Hartree energy, XC double counting, XC energy), a CTA per system.
__global__ void __launch_bounds__(kSumThreads) lda_energies_kernel(const double* __restrict__ node, int64_t node_chunks,
                                                                   const double* __restrict__ grid, int64_t grid_chunks,
                                                                   double* __restrict__ energies) {
    __shared__ double sums[4];
    const int64_t g = blockIdx.x;
    double v[4] = {0.0, 0.0, 0.0, 0.0};
    for (int64_t c = threadIdx.x; c < grid_chunks; c += kSumThreads)
#pragma unroll
        for (int j = 0; j < 3; ++j) v[j] += grid[(g * grid_chunks + c) * 3 + j];
    for (int64_t c = threadIdx.x; c < node_chunks; c += kSumThreads) v[3] += node[g * node_chunks + c];
    block_sums<4>(v, sums);
    __syncthreads();
    if (threadIdx.x == 0) {
        energies[g * 3] = 0.5 * sums[0];
        energies[g * 3 + 1] = sums[1];
        energies[g * 3 + 2] = sums[3] + sums[2];
    }
}

// Deterministic row sums: pass 1 sums fixed chunks, pass 2 sums the chunk partials in order.
constexpr int RS_THREADS = 256;

__global__ void row_partial_kernel(const double* __restrict__ a, int64_t len, int64_t chunk, int chunks,
                                   double* __restrict__ partial) {
    const int r = blockIdx.y;
    const int c = blockIdx.x;
    const int64_t p0 = static_cast<int64_t>(c) * chunk;
    const int64_t p1 = (p0 + chunk < len) ? p0 + chunk : len;
    double s = 0.0;
    for (int64_t p = p0 + threadIdx.x; p < p1; p += RS_THREADS) s += a[static_cast<int64_t>(r) * len + p];
    __shared__ double red[RS_THREADS / 32];
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) s += __shfl_down_sync(0xffffffffu, s, off);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int w = 0; w < RS_THREADS / 32; ++w) t += red[w];
        partial[static_cast<int64_t>(r) * chunks + c] = t;
    }
}

__global__ void row_final_kernel(const double* __restrict__ partial, int rows, int chunks, double* __restrict__ out) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= rows) return;
    double t = 0.0;
    for (int c = 0; c < chunks; ++c) t += partial[static_cast<int64_t>(r) * chunks + c];
    out[r] = t;
}

void row_shape(int rows, int64_t len, int64_t& chunk, int& chunks) {
    int64_t want = ceil_div(2 * 148, rows);
    const int64_t max_chunks = ceil_div(len, 4096);
    if (want > max_chunks) want = max_chunks;
    if (want < 1) want = 1;
    chunk = ceil_div(len, want);
    chunks = static_cast<int>(ceil_div(len, chunk));
}

// Order-8 (or any even order <= 8) central first derivative along `axis`, zero halo
// (src/cdft/operators/laplacian.py:111-130; grid.py:745-758).
__global__ void fd_derivative_kernel(const double* __restrict__ in, double* __restrict__ out, int nx, int ny, int nz,
                                     int axis, int half, const double* __restrict__ coeffs_dev, double scale,
                                     int64_t batch, int accumulate, double sign) {
    const int64_t np = static_cast<int64_t>(nx) * ny * nz;
    const bool narrow = np * batch <= 0xffffffffll;  // 32-bit index arithmetic suffices
    GRID_STRIDE(k, np * batch) {
        int64_t g, i;
        int ix, iy, iz;
        if (narrow) {
            const unsigned uk = static_cast<unsigned>(k), unp = static_cast<unsigned>(np);
            const unsigned ug = uk / unp, ui = uk - ug * unp;
            const unsigned uyz = static_cast<unsigned>(ny) * static_cast<unsigned>(nz);
            const unsigned ux = ui / uyz, r = ui - ux * uyz;
            const unsigned uy = r / static_cast<unsigned>(nz);
            g = ug;
            i = ui;
            ix = static_cast<int>(ux);
            iy = static_cast<int>(uy);
            iz = static_cast<int>(r - uy * static_cast<unsigned>(nz));
        } else {
            g = k / np;
            i = k - g * np;
            ix = static_cast<int>(i / (static_cast<int64_t>(ny) * nz));
            iy = static_cast<int>((i / nz) % ny);
            iz = static_cast<int>(i % nz);
        }
        const int pos = axis == 0 ? ix : (axis == 1 ? iy : iz);
        const int ext = axis == 0 ? nx : (axis == 1 ? ny : nz);
        const int64_t stride = axis == 0 ? static_cast<int64_t>(ny) * nz : (axis == 1 ? nz : 1);
        double acc = 0.0;
        bool first = true;
        for (int t = 0; t <= 2 * half; ++t) {
            const double c = coeffs_dev[t];
            if (c == 0.0) continue;
            const int off = t - half;
            const int q = pos + off;
            const double val = (q >= 0 && q < ext) ? in[g * np + i + off * stride] : 0.0;
            const double term = val * (c * scale);
            acc = first ? term : acc + term;
            first = false;
        }
        if (accumulate)
            out[k] += sign * acc;
        else
            out[k] = sign * acc;
    }
}

// The three partial derivatives of a batch of fields at once, out[g][axis][i] (the (..., 3, N)
// gradient): per point the same sums, in the same order, as three fd_derivative_kernel calls, so the
// result is theirs bit for bit, with the field read once and no stacking copy.
__global__ void gradient_kernel(const double* __restrict__ in, double* __restrict__ out, int nx, int ny, int nz,
                                int half, const double* __restrict__ coeffs_dev, double scale, int64_t batch) {
    const int64_t np = static_cast<int64_t>(nx) * ny * nz;
    const int64_t plane = static_cast<int64_t>(ny) * nz;
    GRID_STRIDE(k, np * batch) {
        const int64_t g = k / np, i = k - g * np;
        const int ix = static_cast<int>(i / plane);
        const int iy = static_cast<int>((i / nz) % ny);
        const int iz = static_cast<int>(i % nz);
        const double* src = in + g * np + i;
#pragma unroll
        for (int axis = 0; axis < 3; ++axis) {
            const int pos = axis == 0 ? ix : (axis == 1 ? iy : iz);
            const int ext = axis == 0 ? nx : (axis == 1 ? ny : nz);
            const int64_t stride = axis == 0 ? plane : (axis == 1 ? nz : 1);
            double acc = 0.0;
            bool first = true;
            for (int t = 0; t <= 2 * half; ++t) {
                const double c = coeffs_dev[t];
                if (c == 0.0) continue;
                const int off = t - half;
                const int q = pos + off;
                const double val = (q >= 0 && q < ext) ? src[off * stride] : 0.0;
                const double term = val * (c * scale);
                acc = first ? term : acc + term;
                first = false;
            }
            out[(g * 3 + axis) * np + i] = 1.0 * acc;
        }
    }
}

// The output density and the density residual of one SCF iteration, per system g and point i
// (src/cdft/scf/step.py:366-370 output_density; src/cdft/scf/loop.py:298-301 and 375-376, the
// residual norm):
//   rho_out = sum_k occ_k v_k^2,  n_out = rho_out f^2,  res = mass |n_out - n_in| / f^2.
// Products and sums are rounded one at a time (no contraction), in the order of those lines.
__global__ void density_residual_kernel(const double* __restrict__ vectors, const double* __restrict__ occ, int k,
                                        int64_t np, int batch, const double* __restrict__ f2,
                                        const double* __restrict__ mass, const double* __restrict__ n_in,
                                        double* __restrict__ rho_out, double* __restrict__ n_out,
                                        double* __restrict__ res) {
    const bool narrow = np * batch <= 0xffffffffll;
    GRID_STRIDE(idx, np * batch) {
        int64_t g, i;
        split_index(idx, np, narrow, g, i);
        const double* v = vectors + g * k * np + i;
        double r = __dmul_rn(occ[0], __dmul_rn(v[0], v[0]));
        for (int j = 1; j < k; ++j) r = __dadd_rn(r, __dmul_rn(occ[j], __dmul_rn(v[j * np], v[j * np])));
        const double f = f2[i];
        const double n = __dmul_rn(r, f);
        rho_out[idx] = r;
        n_out[idx] = n;
        res[idx] = __dmul_rn(mass[i], __ddiv_rn(fabs(__dsub_rn(n, n_in[idx])), f));
    }
}

// Grid half of the external energy parts (hamiltonian.py:360-378), per system g and point i:
//   out[g][0][i] = far_w (weight ((g0 u0 + g1 u1) + g2 u2)),  out[g][1][i] = far_w ((weight rho) W),
// with grad (batch, 3, np) the density gradient, u the cusp exponent's gradient (3, np) and W the
// transformed potential; rounded one operation at a time in that order.
__global__ void external_grid_kernel(const double* __restrict__ grad, const double* __restrict__ rho,
                                     const double* __restrict__ weight, const double* __restrict__ grad_u,
                                     const double* __restrict__ tpot, const double* __restrict__ far_w, int64_t np,
                                     int batch, double* __restrict__ out) {
    const bool narrow = np * batch <= 0xffffffffll;
    GRID_STRIDE(idx, np * batch) {
        int64_t g, i;
        split_index(idx, np, narrow, g, i);
        const double* gr = grad + g * 3 * np + i;
        const double dot = __dadd_rn(__dadd_rn(__dmul_rn(gr[0], grad_u[i]), __dmul_rn(gr[np], grad_u[np + i])),
                                     __dmul_rn(gr[2 * np], grad_u[2 * np + i]));
        const double w = weight[i], fw = far_w[i];
        out[g * 2 * np + i] = __dmul_rn(fw, __dmul_rn(w, dot));
        out[g * 2 * np + np + i] = __dmul_rn(fw, __dmul_rn(__dmul_rn(w, rho[idx]), tpot[i]));
    }
}

}  // namespace

}  // namespace cdftb

using namespace cdftb;

extern "C" int cdftb_xc_lda_vwn_f64(const double* n, int64_t p, double* e, double* v, cdftb_stream_t stream) {
    if (p < 0 || (p > 0 && (!n || !e || !v))) return CDFTB_ERR_ARGUMENT;
    if (p == 0) return CDFTB_OK;
    xc_lda_kernel<<<blocks_for(p, 256), 256, 0, as_stream(stream)>>>(n, p, e, v);
    return check_launch();
}

extern "C" int cdftb_xc_pbe_f64(const double* n, const double* sigma, int64_t p, double* e, double* v, double* vs,
                                cdftb_stream_t stream) {
    if (p < 0 || (p > 0 && (!n || !sigma || !e || !v || !vs))) return CDFTB_ERR_ARGUMENT;
    if (p == 0) return CDFTB_OK;
    xc_pbe_kernel<<<blocks_for(p, 256), 256, 0, as_stream(stream)>>>(n, sigma, p, e, v, vs);
    return check_launch();
}

extern "C" int cdftb_cusp_coefficients_f64(const double* rho_at_nuclei, const double* nucleus_f2, const double* overlap,
                                           int n_atoms, int batch, double* coefficients, cdftb_stream_t stream) {
    if (n_atoms < 1 || n_atoms > MAX_ATOMS || batch < 1 || !rho_at_nuclei || !nucleus_f2 || !overlap || !coefficients)
        return CDFTB_ERR_ARGUMENT;
    cusp_coefficients_kernel<<<static_cast<unsigned>(ceil_div(batch, 64)), 64, 0, as_stream(stream)>>>(
        rho_at_nuclei, nucleus_f2, overlap, n_atoms, batch, coefficients);
    return check_launch();
}

extern "C" int cdftb_hartree_split_f64(const double* density, const double* f2, const double* cusp_grid,
                                       const double* coefficients, int n_atoms, int64_t n_points, int batch, double* rho,
                                       double* n_smooth, cdftb_stream_t stream) {
    if (n_atoms < 0 || n_atoms > MAX_ATOMS || n_points <= 0 || batch < 1 || !density || !f2 || !rho || !n_smooth ||
        (n_atoms > 0 && (!cusp_grid || !coefficients)))
        return CDFTB_ERR_ARGUMENT;
    hartree_split_kernel<<<blocks_for(n_points * batch, 256), 256, 0, as_stream(stream)>>>(
        density, f2, cusp_grid, coefficients, n_atoms, n_points, batch, rho, n_smooth);
    return check_launch();
}

extern "C" int cdftb_potentials_node_lda_f64(const double* fields, int64_t m, const double* weights, const double* f2_node,
                                             const double* v1s_node, const double* coefficients, int n_atoms, int batch,
                                             double* lift_inputs, double* xc_energy_density, cdftb_stream_t stream) {
    if (m < 0 || n_atoms < 0 || n_atoms > MAX_ATOMS || batch < 1) return CDFTB_ERR_ARGUMENT;
    if (m == 0) return CDFTB_OK;
    if (!fields || !weights || !f2_node || !lift_inputs || !xc_energy_density || (n_atoms > 0 && (!v1s_node || !coefficients)))
        return CDFTB_ERR_ARGUMENT;
    node_lda_kernel<<<blocks_for(m * batch, 256), 256, 0, as_stream(stream)>>>(fields, m, weights, f2_node, v1s_node,
                                                                                coefficients, n_atoms, batch, lift_inputs,
                                                                                xc_energy_density);
    return check_launch();
}

extern "C" int cdftb_potentials_grid_lda_f64(const double* density, const double* rho, const double* f2,
                                             const double* far_weights, const double* mass_weights,
                                             const double* v_smooth, const double* v1s_grid, const double* coefficients,
                                             int n_atoms, const double* lifted, int64_t n_points, int batch,
                                             double* effective, double* v_hartree, double* terms, double* v_xc,
                                             cdftb_stream_t stream) {
    if (n_points <= 0 || batch < 1 || n_atoms < 0 || n_atoms > MAX_ATOMS) return CDFTB_ERR_ARGUMENT;
    if (!density || !rho || !f2 || !far_weights || !mass_weights || !v_smooth || !lifted || !effective || !v_hartree ||
        !terms || (n_atoms > 0 && (!v1s_grid || !coefficients)))
        return CDFTB_ERR_ARGUMENT;
    const GridLda p{density,  rho,     f2,     far_weights, mass_weights, v_smooth,  v1s_grid,
                    coefficients, n_atoms, lifted, n_points,    effective,    v_hartree, v_xc};
    grid_lda_kernel<<<blocks_for(n_points * batch, 256), 256, 0, as_stream(stream)>>>(p, batch, terms);
    return check_launch();
}

extern "C" int cdftb_cusp_coefficients_density_f64(const double* density, const double* f2, const int* nuclei_base,
                                                   const double* nuclei_w1d, const double* nucleus_f2,
                                                   const double* overlap, int n_atoms, int nx, int ny, int nz, int batch,
                                                   double* coefficients, cdftb_stream_t stream) {
    if (n_atoms < 1 || n_atoms > MAX_ATOMS || batch < 1 || nx < 1 || ny < 1 || nz < 1 || !density || !f2 ||
        !nuclei_base || !nuclei_w1d || !nucleus_f2 || !overlap || !coefficients)
        return CDFTB_ERR_ARGUMENT;
    cusp_coefficients_density_kernel<<<static_cast<unsigned>(batch), 256, 0, as_stream(stream)>>>(
        density, f2, nuclei_base, nuclei_w1d, nucleus_f2, overlap, n_atoms, int64_t(nx) * ny * nz, ny, nz, coefficients);
    return check_launch();
}

extern "C" int64_t cdftb_potentials_lda_work_bytes(int64_t m, int64_t n_points, int batch) {
    if (m < 0 || n_points <= 0 || batch < 1) return 0;
    return (ceil_div(m, sum_points(m, batch)) + 3 * ceil_div(n_points, sum_points(n_points, batch))) * batch * 8;
}

extern "C" int cdftb_potentials_node_lda_sums_f64(const double* fields, int64_t m, int64_t n_points,
                                                  const double* weights, const double* f2_node, const double* v1s_node,
                                                  const double* coefficients, int n_atoms, int batch,
                                                  double* lift_inputs, void* work, int64_t work_bytes,
                                                  cdftb_stream_t stream) {
    if (m < 0 || n_points <= 0 || n_atoms < 0 || n_atoms > MAX_ATOMS || batch < 1 || !work ||
        work_bytes < cdftb_potentials_lda_work_bytes(m, n_points, batch))
        return CDFTB_ERR_ARGUMENT;
    if (m == 0) return CDFTB_OK;
    if (!fields || !weights || !f2_node || !lift_inputs || (n_atoms > 0 && (!v1s_node || !coefficients)))
        return CDFTB_ERR_ARGUMENT;
    const int64_t points = sum_points(m, batch), chunks = ceil_div(m, points);
    if (chunks * batch > 0x7fffffffll) return CDFTB_ERR_CAPACITY;
    node_lda_sums_kernel<<<static_cast<unsigned>(chunks * batch), kSumThreads, 0, as_stream(stream)>>>(
        fields, m, points, chunks, weights, f2_node, v1s_node, coefficients, n_atoms, batch, lift_inputs,
        static_cast<double*>(work));
    return check_launch();
}

extern "C" int cdftb_potentials_grid_lda_sums_f64(const double* density, const double* rho, const double* f2,
                                                  const double* far_weights, const double* mass_weights,
                                                  const double* v_smooth, const double* v1s_grid,
                                                  const double* coefficients, int n_atoms, const double* lifted,
                                                  int64_t m, int64_t n_points, int batch, double* effective,
                                                  double* v_hartree, double* v_xc, double* energies, void* work,
                                                  int64_t work_bytes, cdftb_stream_t stream) {
    if (m < 0 || n_points <= 0 || batch < 1 || n_atoms < 0 || n_atoms > MAX_ATOMS || !work ||
        work_bytes < cdftb_potentials_lda_work_bytes(m, n_points, batch))
        return CDFTB_ERR_ARGUMENT;
    if (!density || !rho || !f2 || !far_weights || !mass_weights || !v_smooth || !lifted || !effective || !v_hartree ||
        !energies || (n_atoms > 0 && (!v1s_grid || !coefficients)))
        return CDFTB_ERR_ARGUMENT;
    const int64_t node_chunks = ceil_div(m, sum_points(m, batch));
    const int64_t points = sum_points(n_points, batch), chunks = ceil_div(n_points, points);
    if (chunks * batch > 0x7fffffffll) return CDFTB_ERR_CAPACITY;
    double* node = static_cast<double*>(work);
    double* grid = node + node_chunks * batch;
    const GridLda p{density,  rho,     f2,     far_weights, mass_weights, v_smooth,  v1s_grid,
                    coefficients, n_atoms, lifted, n_points,    effective,    v_hartree, v_xc};
    cudaStream_t s = as_stream(stream);
    grid_lda_sums_kernel<<<static_cast<unsigned>(chunks * batch), kSumThreads, 0, s>>>(p, points, chunks, grid);
    const int st = check_launch();
    if (st != CDFTB_OK) return st;
    lda_energies_kernel<<<static_cast<unsigned>(batch), kSumThreads, 0, s>>>(node, node_chunks, grid, chunks, energies);
    return check_launch();
}

extern "C" int64_t cdftb_row_sums_scratch_bytes(int rows, int64_t len) {
    if (rows <= 0 || len <= 0) return 0;
    int64_t chunk;
    int chunks;
    row_shape(rows, len, chunk, chunks);
    return static_cast<int64_t>(rows) * chunks * 8;
}

extern "C" int cdftb_density_residual_f64(const double* vectors, const double* occupations, int k, int64_t n_points,
                                          int batch, const double* f2, const double* mass_weights,
                                          const double* n_in, double* rho_out, double* n_out, double* residual_terms,
                                          cdftb_stream_t stream) {
    if (!vectors || !occupations || !f2 || !mass_weights || !n_in || !rho_out || !n_out || !residual_terms || k < 1 ||
        n_points <= 0 || batch < 1)
        return CDFTB_ERR_ARGUMENT;
    density_residual_kernel<<<blocks_for(n_points * batch, 256), 256, 0, as_stream(stream)>>>(
        vectors, occupations, k, n_points, batch, f2, mass_weights, n_in, rho_out, n_out, residual_terms);
    return check_launch();
}

extern "C" int cdftb_external_grid_terms_f64(const double* grad, const double* rho, const double* weight,
                                             const double* grad_u, const double* transformed_potential,
                                             const double* far_weights, int64_t n_points, int batch, double* out,
                                             cdftb_stream_t stream) {
    if (!grad || !rho || !weight || !grad_u || !transformed_potential || !far_weights || !out || n_points <= 0 ||
        batch < 1)
        return CDFTB_ERR_ARGUMENT;
    external_grid_kernel<<<blocks_for(n_points * batch, 256), 256, 0, as_stream(stream)>>>(
        grad, rho, weight, grad_u, transformed_potential, far_weights, n_points, batch, out);
    return check_launch();
}

extern "C" int cdftb_row_sums_f64(const double* a, int rows, int64_t len, double* out, void* scratch,
                                  int64_t scratch_bytes, cdftb_stream_t stream) {
    if (!a || !out || rows <= 0 || rows > 65535 || len <= 0) return CDFTB_ERR_ARGUMENT;
    if (!scratch || scratch_bytes < cdftb_row_sums_scratch_bytes(rows, len)) return CDFTB_ERR_ARGUMENT;
    int64_t chunk;
    int chunks;
    row_shape(rows, len, chunk, chunks);
    cudaStream_t s = as_stream(stream);
    double* partial = static_cast<double*>(scratch);
    row_partial_kernel<<<dim3(chunks, rows), RS_THREADS, 0, s>>>(a, len, chunk, chunks, partial);
    int st = check_launch();
    if (st != CDFTB_OK) return st;
    row_final_kernel<<<static_cast<unsigned>(ceil_div(rows, 64)), 64, 0, s>>>(partial, rows, chunks, out);
    return check_launch();
}

extern "C" int cdftb_gradient_f64(const double* in, double* out, int nx, int ny, int nz, int accuracy,
                                  const double* coefficients, double spacing, int64_t batch, cdftb_stream_t stream) {
    if (!in || !out || !coefficients || accuracy < 2 || accuracy > 8 || accuracy % 2 || !(spacing > 0.0) || batch < 1 ||
        nx <= 0 || ny <= 0 || nz <= 0)
        return CDFTB_ERR_ARGUMENT;
    const int64_t np = static_cast<int64_t>(nx) * ny * nz;
    gradient_kernel<<<blocks_for(np * batch, 256), 256, 0, as_stream(stream)>>>(in, out, nx, ny, nz, accuracy / 2,
                                                                              coefficients, 1.0 / spacing, batch);
    return check_launch();
}

extern "C" int cdftb_fd_derivative_f64(const double* in, double* out, int nx, int ny, int nz, int axis, int accuracy,
                                       const double* coefficients, double spacing, int64_t batch, int accumulate,
                                       double sign, cdftb_stream_t stream) {
    if (!in || !out || !coefficients || axis < 0 || axis > 2 || accuracy < 2 || accuracy > 8 || accuracy % 2 ||
        !(spacing > 0.0) || batch < 1)
        return CDFTB_ERR_ARGUMENT;
    const int64_t np = static_cast<int64_t>(nx) * ny * nz;
    fd_derivative_kernel<<<blocks_for(np * batch, 256), 256, 0, as_stream(stream)>>>(
        in, out, nx, ny, nz, axis, accuracy / 2, coefficients, 1.0 / spacing, batch, accumulate, sign);
    return check_launch();
}
