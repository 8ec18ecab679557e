// (c) The Coulomb-cutoff Poisson solve (src/cdft/operators/poisson.py:21-107) as five pruned
// axis-wise FFT passes on the device, with the truncated kernel K(G) fused into the x pass.
//
// The definition pads the box to N = fft_friendly(ceil(pad n)) points per axis and multiplies by K(G)
// there. The density fills the first n points and only the first n outputs are kept, so the product is
// the linear convolution with K's inverse transform at the offsets -(n-1) .. n-1, which a circular
// transform of any length M >= 2n - 1 gives too. The plan therefore carries K over to the shortest
// such length that the kernels below take (reduce_kernel_table: 135 instead of 180 points per axis at
// 65^3, 0.41 of the work), and the passes are
//   pass 1  z, real -> half complex      rho[x][y][z]        -> A[x][y][kz]    (x < nx, y < ny)
//   pass 2  y, forward                   A[x][y][kz]         -> B[x][ky][kz]   (x < nx)
//   pass 3  x, forward, * K, inverse     B[x][ky][kz]        -> B[x][ky][kz]   (in place, x < nx)
//   pass 4  y, inverse                   B[x][ky][kz]        -> A[x][y][kz]    (y < ny)
//   pass 5  z, half complex -> real      A[x][y][kz]         -> v[x][y][z]     (z < nz)
// with the 1 / (Mx My Mz) of the inverse in K's table.
// Only lines that can be non-zero are transformed, and only the outputs a later pass reads are kept.
// Every pass is one CTA per 8 lines staged in shared memory as [element][line] (row stride 9, so that
// the steps and the transposed loads and stores avoid bank conflicts): the four-step register kernels
// for lengths up to 320, a mixed-radix Stockham FFT (radices 4, 2, 3, 5) beyond.

#include <math.h>

#include <algorithm>

#include "common.cuh"

namespace cdftb {

namespace {

struct cplx {
    double re, im;
};

__device__ __forceinline__ cplx operator+(cplx a, cplx b) { return {a.re + b.re, a.im + b.im}; }
__device__ __forceinline__ cplx operator-(cplx a, cplx b) { return {a.re - b.re, a.im - b.im}; }
__device__ __forceinline__ cplx scale(cplx a, double s) { return {a.re * s, a.im * s}; }
__device__ __forceinline__ cplx cmul(cplx a, cplx b) { return {a.re * b.re - a.im * b.im, a.re * b.im + a.im * b.re}; }
__device__ __forceinline__ cplx cmulc(cplx a, cplx b) { return {a.re * b.re + a.im * b.im, a.im * b.re - a.re * b.im}; }
// i * sign * a
__device__ __forceinline__ cplx rot(cplx a, int sign) { return sign < 0 ? cplx{a.im, -a.re} : cplx{-a.im, a.re}; }

constexpr int MAX_STAGES = 16;

// One axis: N = product of radix[0..nst); stage st has stride s (product of the earlier radices),
// m = N / (s * radix) and twiddles tw[tw_off + p * (radix - 1) + k - 1] = exp(-2 pi i p k / (N / s)).
struct FftPlan {
    int n;
    int nst;
    int radix[MAX_STAGES];
    int stride[MAX_STAGES];
    int m[MAX_STAGES];
    int tw_off[MAX_STAGES];
    const cplx* tw;
};

// Radix-R DFT with the rotation exp(sign 2 pi i / R) (sign -1 forward, +1 inverse).
template <int R>
__device__ __forceinline__ void dft_radix(cplx* a, int sign);

template <>
__device__ __forceinline__ void dft_radix<2>(cplx* a, int) {
    const cplx t = a[0] - a[1];
    a[0] = a[0] + a[1];
    a[1] = t;
}

template <>
__device__ __forceinline__ void dft_radix<4>(cplx* a, int sign) {
    const cplx t0 = a[0] + a[2], t1 = a[0] - a[2], t2 = a[1] + a[3], t3 = rot(a[1] - a[3], sign);
    a[0] = t0 + t2;
    a[1] = t1 + t3;
    a[2] = t0 - t2;
    a[3] = t1 - t3;
}

// sqrt(3)/2 a. The double nearest to sqrt(3)/2 is off by almost half a unit in its last place, the
// same way in every butterfly; the remainder is added.
__device__ __forceinline__ cplx scale_half_sqrt3(cplx a) {
    constexpr double hi = 0.86602540378443864676, lo = 5.0175422e-17;
    return {fma(a.re, hi, a.re * lo), fma(a.im, hi, a.im * lo)};
}

template <>
__device__ __forceinline__ void dft_radix<3>(cplx* a, int sign) {
    const cplx t = a[1] + a[2];
    const cplx v = rot(scale_half_sqrt3(a[1] - a[2]), sign);
    const cplx h = {a[0].re - 0.5 * t.re, a[0].im - 0.5 * t.im};
    a[0] = a[0] + t;
    a[1] = h + v;
    a[2] = h - v;
}

template <>
__device__ __forceinline__ void dft_radix<5>(cplx* a, int sign) {
    constexpr double c1 = 0.30901699437494742410;   // cos(2 pi / 5)
    constexpr double c2 = -0.80901699437494742410;  // cos(4 pi / 5)
    constexpr double s1 = 0.95105651629515357212;   // sin(2 pi / 5)
    constexpr double s2 = 0.58778525229247312917;   // sin(4 pi / 5)
    const cplx t1 = a[1] + a[4], t2 = a[2] + a[3], t3 = a[1] - a[4], t4 = a[2] - a[3];
    const cplx x1 = {a[0].re + c1 * t1.re + c2 * t2.re, a[0].im + c1 * t1.im + c2 * t2.im};
    const cplx x2 = {a[0].re + c2 * t1.re + c1 * t2.re, a[0].im + c2 * t1.im + c1 * t2.im};
    const cplx y1 = rot({s1 * t3.re + s2 * t4.re, s1 * t3.im + s2 * t4.im}, sign);
    const cplx y2 = rot({s2 * t3.re - s1 * t4.re, s2 * t3.im - s1 * t4.im}, sign);
    a[0] = a[0] + t1 + t2;
    a[1] = x1 + y1;
    a[2] = x2 + y2;
    a[3] = x2 - y2;
    a[4] = x1 - y1;
}

template <int R>
__device__ __forceinline__ void stage_radix(const cplx* __restrict__ x, cplx* __restrict__ y, int s, int m,
                                            const cplx* __restrict__ tw, int sign, int lp, int lane, int ty, int nty,
                                            int nb) {
    for (int b = ty; b < nb; b += nty) {
        const int p = b / s;
        const int q = b - p * s;
        cplx a[R];
#pragma unroll
        for (int j = 0; j < R; ++j) a[j] = x[(q + s * (p + j * m)) * lp + lane];
        dft_radix<R>(a, sign);
        const cplx* w = tw + p * (R - 1);
        y[(q + s * R * p) * lp + lane] = a[0];
#pragma unroll
        for (int k = 1; k < R; ++k) {
            const cplx wk = w[k - 1];
            y[(q + s * (R * p + k)) * lp + lane] = sign < 0 ? cmul(a[k], wk) : cmulc(a[k], wk);
        }
    }
}

// The FFT of the lines held in x ([N][lp]); y is scratch of the same size. Returns the buffer that
// holds the result. Called by every thread of the CTA (it synchronises after each stage).
__device__ cplx* fft_lines(cplx* x, cplx* y, const FftPlan& P, int sign, int lp, int lane, int ty, int nty) {
    for (int st = 0; st < P.nst; ++st) {
        const int R = P.radix[st];
        const int s = P.stride[st];
        const int m = P.m[st];
        const cplx* tw = P.tw + P.tw_off[st];
        const int nb = P.n / R;
        switch (R) {
            case 4: stage_radix<4>(x, y, s, m, tw, sign, lp, lane, ty, nty, nb); break;
            case 2: stage_radix<2>(x, y, s, m, tw, sign, lp, lane, ty, nty, nb); break;
            case 3: stage_radix<3>(x, y, s, m, tw, sign, lp, lane, ty, nty, nb); break;
            default: stage_radix<5>(x, y, s, m, tw, sign, lp, lane, ty, nty, nb); break;
        }
        __syncthreads();
        cplx* t = x;
        x = y;
        y = t;
    }
    return x;
}

// ---------------------------------------------------------------------------------------------
// Four-step transforms in registers, for line lengths N = A B with A, B in {4, 6, 8, 9, 10, 12, 15, 16,
// 18, 20}. For n = B n1 + n2 and k = k1 + A k2:
//   X[k1 + A k2] = sum_n2 W_B^(n2 k2) W_N^(n2 k1) sum_n1 x[B n1 + n2] W_A^(n1 k1),
// so a thread does one A-point DFT (over n1, fixed n2) and, after an in-place exchange through
// shared memory, one B-point DFT (over n2, fixed k1), each entirely in registers. The small DFTs
// are nested radix 2/3/4/5 butterflies with their internal twiddles from a constant table of the
// 720th roots of unity (every size here divides 720); W_N comes from a per-axis table.

__constant__ cplx kUnit720[720];  // exp(-2 pi i j / 720)

template <int R>
__device__ __forceinline__ cplx unit_root(int m, int sign) {
    const cplx w = kUnit720[(m % R) * (720 / R)];
    return sign < 0 ? w : cplx{w.re, -w.im};
}

template <int R>
struct FirstFactor {
    static constexpr int value = R % 4 == 0 ? 4 : (R % 2 == 0 ? 2 : (R % 3 == 0 ? 3 : 5));
};

// In-place DFT of R values held in registers (natural order in and out), sign -1 forward.
template <int R>
__device__ __forceinline__ void small_dft(cplx* a, int sign) {
    if constexpr (R == 2 || R == 3 || R == 4 || R == 5) {
        dft_radix<R>(a, sign);
    } else {
        constexpr int P = FirstFactor<R>::value;
        constexpr int Q = R / P;
        static_assert(P * Q == R && 720 % R == 0, "small DFT sizes divide 720");
        cplx b[R];
#pragma unroll
        for (int n2 = 0; n2 < Q; ++n2) {
            cplx c[P];
#pragma unroll
            for (int n1 = 0; n1 < P; ++n1) c[n1] = a[Q * n1 + n2];
            small_dft<P>(c, sign);
#pragma unroll
            for (int k1 = 0; k1 < P; ++k1) b[k1 * Q + n2] = (n2 * k1 == 0) ? c[k1] : cmul(c[k1], unit_root<R>(n2 * k1, sign));
        }
#pragma unroll
        for (int k1 = 0; k1 < P; ++k1) {
            cplx c[Q];
#pragma unroll
            for (int n2 = 0; n2 < Q; ++n2) c[n2] = b[k1 * Q + n2];
            small_dft<Q>(c, sign);
#pragma unroll
            for (int k2 = 0; k2 < Q; ++k2) a[k1 + P * k2] = c[k2];
        }
    }
}

// The same DFTs of R values of which only the first CNT are non-zero (the others are not read).
template <int R, int CNT>
__device__ __forceinline__ void dft_radix_lead(cplx* a, int sign) {
    static_assert(CNT >= 1 && CNT <= R, "at least one input");
    if constexpr (CNT == R) {
        dft_radix<R>(a, sign);
    } else if constexpr (CNT == 1) {
#pragma unroll
        for (int k = 1; k < R; ++k) a[k] = a[0];
    } else if constexpr (R == 3) {
        const cplx v = rot(scale_half_sqrt3(a[1]), sign);
        const cplx h = {a[0].re - 0.5 * a[1].re, a[0].im - 0.5 * a[1].im};
        a[0] = a[0] + a[1];
        a[1] = h + v;
        a[2] = h - v;
    } else if constexpr (R == 4 && CNT == 2) {
        const cplx t = a[0], r = rot(a[1], sign);
        a[0] = t + a[1];
        a[2] = t - a[1];
        a[1] = t + r;
        a[3] = t - r;
    } else if constexpr (R == 4) {
        const cplx t0 = a[0] + a[2], t1 = a[0] - a[2], r = rot(a[1], sign);
        a[0] = t0 + a[1];
        a[2] = t0 - a[1];
        a[1] = t1 + r;
        a[3] = t1 - r;
    } else {
#pragma unroll
        for (int k = CNT; k < R; ++k) a[k] = cplx{0.0, 0.0};
        dft_radix<R>(a, sign);
    }
}

template <int R, int CNT>
__device__ __forceinline__ void small_dft_lead(cplx* a, int sign);

// The first stage of small_dft_lead for n2 = N2, N2 + 1, ...: the P-point DFTs over n1.
template <int R, int CNT, int N2>
__device__ __forceinline__ void lead_stage(const cplx* a, cplx* b, int sign) {
    constexpr int P = FirstFactor<R>::value, Q = R / P;
    if constexpr (N2 < Q) {
        constexpr int LEAD = (CNT - N2 + Q - 1) / Q;  // inputs Q n1 + N2 below CNT
        cplx c[P];
#pragma unroll
        for (int n1 = 0; n1 < LEAD; ++n1) c[n1] = a[Q * n1 + N2];
        dft_radix_lead<P, LEAD>(c, sign);
#pragma unroll
        for (int k1 = 0; k1 < P; ++k1) b[k1 * Q + N2] = (N2 * k1 == 0) ? c[k1] : cmul(c[k1], unit_root<R>(N2 * k1, sign));
        lead_stage<R, CNT, N2 + 1>(a, b, sign);
    }
}

template <int R, int CNT>
__device__ __forceinline__ void small_dft_lead(cplx* a, int sign) {
    if constexpr (CNT == R) {
        small_dft<R>(a, sign);
    } else if constexpr (R == 2 || R == 3 || R == 4 || R == 5) {
        dft_radix_lead<R, CNT>(a, sign);
    } else {
        constexpr int P = FirstFactor<R>::value, Q = R / P;
        static_assert(CNT >= Q, "every first-stage DFT has an input");
        cplx b[R];
        lead_stage<R, CNT, 0>(a, b, sign);
#pragma unroll
        for (int k1 = 0; k1 < P; ++k1) {
            cplx c[Q];
#pragma unroll
            for (int n2 = 0; n2 < Q; ++n2) c[n2] = b[k1 * Q + n2];
            small_dft<Q>(c, sign);
#pragma unroll
            for (int k2 = 0; k2 < Q; ++k2) a[k1 + P * k2] = c[k2];
        }
    }
}

// Measured: 8 systems of 81 x 81 x 91 points 495 us per solve; with the definition's lengths, complex z
// transforms of real lines on the Stockham kernels and no pruning it was 1015 us. One He 65^3 system
// 39 us, was 75. The error against long double is 2.1e-16 at 65^3 as before (2.1e-16): roots of unity
// made in double angles and sqrt(3)/2 as one double would have cost 3.3e-16.
constexpr int kLines4 = 8;     // lines per CTA of the four-step kernels
constexpr int kThreads4 = 128;

// What a transform of length A B needs to handle when only the first (A B + 1) / 2 elements of its
// input, or of its output, count (the box of a convolution).
template <int A, int B>
struct FourStep {
    static constexpr int N = A * B;
    static constexpr int BOX = (N + 1) / 2;
    static constexpr int IN = (BOX + B - 1) / B;    // first-step inputs n1 < IN hold every n = B n1 + n2 < BOX
    static constexpr int OUT = (BOX + A - 1) / A;   // second-step outputs k2 < OUT hold every k1 + A k2 < BOX
    static constexpr int ROWS = B * IN;             // staged elements of a box input
    static_assert(A * kLines4 <= kThreads4, "one second-step task per thread");
};

// Step 1 of a forward (sign -1) or inverse (+1) transform of the L lines in buf ([N][L+1]): per
// (line, n2), the A-point DFT over n1 of x[B n1 + n2] (non-zero for n1 < LEAD), times W_N^(+-n2 k1),
// back in place.
template <int A, int B, int LEAD>
__device__ __forceinline__ void fourstep_first(cplx* buf, const cplx* __restrict__ twn, int sign) {
    constexpr int N = A * B, L = kLines4, LP = L + 1;
    for (int task = threadIdx.x; task < B * L; task += kThreads4) {
        const int line = task % L, n2 = task / L;
        cplx v[A];
#pragma unroll
        for (int n1 = 0; n1 < LEAD; ++n1) v[n1] = buf[(B * n1 + n2) * LP + line];
        small_dft_lead<A, LEAD>(v, sign);
#pragma unroll
        for (int k1 = 0; k1 < A; ++k1) {
            const cplx w = twn[(n2 * k1) % N];
            buf[(B * k1 + n2) * LP + line] = sign < 0 ? cmul(v[k1], w) : cmulc(v[k1], w);
        }
    }
}

// Pass 3, four-step: the x lines of one system ([nx][inner]) -- forward, times K, inverse -- with
// the K multiply and the first inverse step on the registers of the second forward step. The first
// step reads and the last one forms only the box's elements.
template <int A, int B>
__global__ void __launch_bounds__(kThreads4) fft_x_fourstep_kernel(cplx* __restrict__ data, int nx, int64_t inner,
                                                                  const double* __restrict__ kernel,
                                                                  const cplx* __restrict__ twn) {
    using F = FourStep<A, B>;
    constexpr int N = F::N, L = kLines4, LP = L + 1;
    __shared__ cplx buf[N * LP];
    const int64_t c0 = int64_t(blockIdx.x) * L;
    cplx* col = data + int64_t(blockIdx.y) * nx * inner + c0;
#pragma unroll 4
    for (int idx = threadIdx.x; idx < F::ROWS * L; idx += kThreads4) {
        const int line = idx % L, x = idx / L;
        buf[x * LP + line] = (x < nx && c0 + line < inner) ? col[int64_t(x) * inner + line] : cplx{0.0, 0.0};
    }
    __syncthreads();
    fourstep_first<A, B, F::IN>(buf, twn, -1);
    __syncthreads();
    for (int task = threadIdx.x; task < A * L; task += kThreads4) {
        const int line = task % L, k1 = task / L;
        const bool live = c0 + line < inner;
        cplx v[B];
#pragma unroll
        for (int n2 = 0; n2 < B; ++n2) v[n2] = buf[(B * k1 + n2) * LP + line];
        small_dft<B>(v, -1);  // X[k1 + A k2] = v[k2]
#pragma unroll
        for (int k2 = 0; k2 < B; ++k2)
            v[k2] = scale(v[k2], live ? kernel[int64_t(k1 + A * k2) * inner + c0 + line] : 0.0);
        small_dft<B>(v, +1);  // inverse, first step: Z[k1][n2] = v[n2]
#pragma unroll
        for (int n2 = 0; n2 < B; ++n2) buf[(B * k1 + n2) * LP + line] = cmulc(v[n2], twn[(n2 * k1) % N]);
    }
    __syncthreads();
    for (int task = threadIdx.x; task < B * L; task += kThreads4) {
        const int line = task % L, n2 = task / L;
        cplx v[A];
#pragma unroll
        for (int k1 = 0; k1 < A; ++k1) v[k1] = buf[(B * k1 + n2) * LP + line];
        small_dft<A>(v, +1);
        if (c0 + line < inner) {
#pragma unroll
            for (int n1 = 0; n1 < F::IN; ++n1) {
                const int x = B * n1 + n2;
                if (x < nx) col[int64_t(x) * inner + line] = v[n1];
            }
        }
    }
}

// Passes 2 and 4, four-step: middle-axis lines of [outer][n][inner]. Forward (SIGN -1): n_in elements
// per line in (zero beyond), all N out; inverse (+1): all N in, the first n_out out.
template <int A, int B, int SIGN>
__global__ void __launch_bounds__(kThreads4) fft_middle_fourstep_kernel(const cplx* __restrict__ in,
                                                                       int64_t in_outer_stride, int n_in,
                                                                       cplx* __restrict__ out,
                                                                       int64_t out_outer_stride, int n_out,
                                                                       int64_t inner, const cplx* __restrict__ twn) {
    using F = FourStep<A, B>;
    constexpr int N = F::N, L = kLines4, LP = L + 1;
    constexpr int ROWS = SIGN < 0 ? F::ROWS : N, LEAD = SIGN < 0 ? F::IN : A, KEEP = SIGN < 0 ? B : F::OUT;
    __shared__ cplx buf[N * LP];
    const int64_t o = blockIdx.x;
    const int64_t c0 = int64_t(blockIdx.y) * L;
    const cplx* src = in + o * in_outer_stride + c0;
#pragma unroll 4
    for (int idx = threadIdx.x; idx < ROWS * L; idx += kThreads4) {
        const int line = idx % L, j = idx / L;
        buf[j * LP + line] = (j < n_in && c0 + line < inner) ? src[int64_t(j) * inner + line] : cplx{0.0, 0.0};
    }
    __syncthreads();
    fourstep_first<A, B, LEAD>(buf, twn, SIGN);
    __syncthreads();
    cplx* dst = out + o * out_outer_stride + c0;
    for (int task = threadIdx.x; task < A * L; task += kThreads4) {
        const int line = task % L, k1 = task / L;
        cplx v[B];
#pragma unroll
        for (int n2 = 0; n2 < B; ++n2) v[n2] = buf[(B * k1 + n2) * LP + line];
        small_dft<B>(v, SIGN);
        if (c0 + line < inner) {
#pragma unroll
            for (int k2 = 0; k2 < KEEP; ++k2) {
                const int k = k1 + A * k2;
                if (k < n_out) dst[int64_t(k) * inner + line] = v[k2];
            }
        }
    }
}

// Pass 1, four-step: the z lines (contiguous, nz real values) of system blockIdx.y -> half spectrum kz < nk.
// Two real lines a, b share one complex transform of a + i b: with Z its spectrum,
// A[k] = (Z[k] + conj Z[N-k]) / 2 and B[k] = (Z[k] - conj Z[N-k]) / 2i. Rounding errors of one line, and its
// NaN, reach the other one, so the two are always lines of one system (an odd last line has zeros beside it).
template <int A, int B>
__global__ void __launch_bounds__(kThreads4) fft_z_forward_fourstep_kernel(const double* __restrict__ rho,
                                                                          int64_t lines, int nz,
                                                                          cplx* __restrict__ out, int nk,
                                                                          const cplx* __restrict__ twn) {
    using F = FourStep<A, B>;
    constexpr int N = F::N, L = kLines4, LP = L + 1;
    __shared__ cplx buf[N * LP];
    const int64_t l0 = blockIdx.y * lines + int64_t(blockIdx.x) * (2 * L);
    lines *= blockIdx.y + 1;  // the end of the system's lines
#pragma unroll 4
    for (int idx = threadIdx.x; idx < 2 * L * F::ROWS; idx += kThreads4) {
        const int line = idx / F::ROWS, z = idx % F::ROWS;
        const double v = (z < nz && l0 + line < lines) ? rho[(l0 + line) * nz + z] : 0.0;
        reinterpret_cast<double*>(buf + z * LP + (line >> 1))[line & 1] = v;
    }
    __syncthreads();
    fourstep_first<A, B, F::IN>(buf, twn, -1);
    __syncthreads();
    const int line = threadIdx.x % L, k1 = threadIdx.x / L;
    cplx v[B];
    if (k1 < A) {
#pragma unroll
        for (int n2 = 0; n2 < B; ++n2) v[n2] = buf[(B * k1 + n2) * LP + line];
        small_dft<B>(v, -1);
    }
    __syncthreads();
    if (k1 < A) {
#pragma unroll
        for (int k2 = 0; k2 < B; ++k2) buf[(k1 + A * k2) * LP + line] = v[k2];
    }
    __syncthreads();
    for (int idx = threadIdx.x; idx < L * nk; idx += kThreads4) {
        const int pair = idx / nk, k = idx - pair * nk;
        const cplx p = buf[k * LP + pair], q = buf[(k == 0 ? 0 : N - k) * LP + pair];
        const int64_t row = l0 + 2 * pair;
        if (row < lines) out[row * nk + k] = {0.5 * (p.re + q.re), 0.5 * (p.im - q.im)};
        if (row + 1 < lines) out[(row + 1) * nk + k] = {0.5 * (p.im + q.im), 0.5 * (q.re - p.re)};
    }
}

// Pass 5, four-step: half spectra -> real z lines (z < nz) of system blockIdx.y, two lines per
// complex transform of A + i B (both Hermitian-extended; irfft drops the imaginary parts of the k = 0
// and Nyquist terms, which would leak into the other line here).
template <int A, int B>
__global__ void __launch_bounds__(kThreads4) fft_z_inverse_fourstep_kernel(const cplx* __restrict__ in, int64_t lines,
                                                                          int nk, double* __restrict__ out, int nz,
                                                                          const cplx* __restrict__ twn) {
    using F = FourStep<A, B>;
    constexpr int N = F::N, L = kLines4, LP = L + 1;
    __shared__ cplx buf[N * LP];
    const int64_t l0 = blockIdx.y * lines + int64_t(blockIdx.x) * (2 * L);
    lines *= blockIdx.y + 1;  // the end of the system's lines
#pragma unroll 2
    for (int idx = threadIdx.x; idx < L * nk; idx += kThreads4) {
        const int pair = idx / nk, k = idx - pair * nk;
        const int64_t row = l0 + 2 * pair;
        cplx a = row < lines ? in[row * nk + k] : cplx{0.0, 0.0};
        cplx b = row + 1 < lines ? in[(row + 1) * nk + k] : cplx{0.0, 0.0};
        if (k == 0 || 2 * k == N) a.im = b.im = 0.0;
        buf[k * LP + pair] = {a.re - b.im, a.im + b.re};
        if (k > 0 && N - k >= nk) buf[(N - k) * LP + pair] = {a.re + b.im, b.re - a.im};
    }
    __syncthreads();
    fourstep_first<A, B, A>(buf, twn, +1);
    __syncthreads();
    const int line = threadIdx.x % L, k1 = threadIdx.x / L;
    cplx v[B];
    if (k1 < A) {
#pragma unroll
        for (int n2 = 0; n2 < B; ++n2) v[n2] = buf[(B * k1 + n2) * LP + line];
        small_dft<B>(v, +1);
    }
    __syncthreads();
    if (k1 < A) {
#pragma unroll
        for (int k2 = 0; k2 < F::OUT; ++k2) buf[(k1 + A * k2) * LP + line] = v[k2];
    }
    __syncthreads();
    for (int idx = threadIdx.x; idx < 2 * L * nz; idx += kThreads4) {
        const int l = idx / nz, z = idx - l * nz;
        if (l0 + l < lines)
            out[(l0 + l) * nz + z] = reinterpret_cast<const double*>(buf + z * LP + (l >> 1))[l & 1];
    }
}

int fft_friendly(int n) {
    for (int c = n;; ++c) {
        int r = c;
        for (int p : {2, 3, 5})
            while (r % p == 0) r /= p;
        if (r == 1) return c;
    }
}

// The factor pair (A, B) of a length the four-step kernels take, A * B = n; false otherwise.
bool fourstep_pair(int n, int* a, int* b) {
    static const int pairs[][3] = {{36, 4, 9},    {48, 6, 8},    {64, 8, 8},    {72, 8, 9},    {80, 8, 10},
                                   {90, 9, 10},   {96, 8, 12},   {100, 10, 10}, {108, 9, 12},
                                   {120, 10, 12}, {128, 8, 16},  {135, 9, 15},  {144, 12, 12}, {150, 10, 15},
                                   {160, 10, 16}, {162, 9, 18},  {180, 12, 15}, {192, 12, 16}, {200, 10, 20},
                                   {216, 12, 18}, {225, 15, 15}, {240, 15, 16}, {256, 16, 16}, {270, 15, 18},
                                   {288, 16, 18}, {300, 15, 20}, {320, 16, 20}};
    for (const auto& q : pairs)
        if (q[0] == n) {
            *a = q[1];
            *b = q[2];
            return true;
        }
    return false;
}

#define CDFTB_FOURSTEP_PAIRS(X)                                                                                   \
    X(4, 9) X(6, 8) X(8, 8) X(8, 9) X(8, 10) X(9, 10) X(8, 12) X(10, 10) X(9, 12) X(10, 12) X(8, 16)      \
        X(9, 15) X(12, 12) X(10, 15) X(10, 16) X(9, 18) X(12, 15) X(12, 16) X(10, 20) X(12, 18) X(15, 15)         \
            X(15, 16) X(16, 16) X(15, 18) X(16, 18) X(15, 20) X(16, 20)

// The shortest length of at least 2n - 1 points that the four-step kernels take, else the next 2,3,5-smooth one.
int convolution_length(int n) {
    int best = 0, a, b;
    for (int len = 2 * n - 1; len <= 320 && !best; ++len)
        if (fourstep_pair(len, &a, &b)) best = len;
    return best ? best : fft_friendly(2 * n - 1);
}

// Pass 1: z lines (contiguous, nz real values zero-padded to N) -> half spectrum kz < nk.
template <int L>
__global__ void __launch_bounds__(256) fft_z_forward_kernel(const double* __restrict__ rho, int64_t lines, int nz,
                                                            cplx* __restrict__ out, int nk, const FftPlan P) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr int LP = L + 1;
    cplx* b0 = reinterpret_cast<cplx*>(smem_raw);
    cplx* b1 = b0 + P.n * LP;
    const int tid = threadIdx.y * L + threadIdx.x;
    const int nthreads = L * blockDim.y;
    const int64_t l0 = int64_t(blockIdx.x) * L;
    for (int idx = tid; idx < L * P.n; idx += nthreads) {
        const int line = idx / P.n;
        const int z = idx - line * P.n;
        const double v = (z < nz && l0 + line < lines) ? rho[(l0 + line) * nz + z] : 0.0;
        b0[z * LP + line] = {v, 0.0};
    }
    __syncthreads();
    const cplx* r = fft_lines(b0, b1, P, -1, LP, threadIdx.x, threadIdx.y, blockDim.y);
    for (int idx = tid; idx < L * nk; idx += nthreads) {
        const int line = idx / nk;
        const int k = idx - line * nk;
        if (l0 + line < lines) out[(l0 + line) * nk + k] = r[k * LP + line];
    }
}

// Passes 2 and 4: middle-axis lines of data viewed as [outer][n][inner], inner contiguous; reads
// n_in elements per line (zero beyond), transforms with length P.n, writes n_out elements.
template <int L>
__global__ void __launch_bounds__(256) fft_middle_kernel(const cplx* __restrict__ in, int64_t in_outer_stride, int n_in,
                                                         cplx* __restrict__ out, int64_t out_outer_stride, int n_out,
                                                         int64_t inner, const FftPlan P, int sign) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr int LP = L + 1;
    cplx* b0 = reinterpret_cast<cplx*>(smem_raw);
    cplx* b1 = b0 + P.n * LP;
    const int64_t o = blockIdx.x;
    const int64_t c = int64_t(blockIdx.y) * L + threadIdx.x;
    const bool live = c < inner;
    const cplx* src = in + o * in_outer_stride + c;
    for (int j = threadIdx.y; j < P.n; j += blockDim.y)
        b0[j * LP + threadIdx.x] = (j < n_in && live) ? src[int64_t(j) * inner] : cplx{0.0, 0.0};
    __syncthreads();
    const cplx* r = fft_lines(b0, b1, P, sign, LP, threadIdx.x, threadIdx.y, blockDim.y);
    if (!live) return;
    cplx* dst = out + o * out_outer_stride + c;
    for (int j = threadIdx.y; j < n_out; j += blockDim.y) dst[int64_t(j) * inner] = r[j * LP + threadIdx.x];
}

// Pass 3: x lines of one system ([nx][inner], inner = N1 * nk contiguous): forward FFT of the nx
// non-zero values, times K[kx][ky][kz], inverse FFT, the first nx values written back in place.
template <int L>
__global__ void __launch_bounds__(256) fft_x_fused_kernel(cplx* __restrict__ data, int nx, int64_t inner,
                                                          const double* __restrict__ kernel, const FftPlan P) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr int LP = L + 1;
    cplx* b0 = reinterpret_cast<cplx*>(smem_raw);
    cplx* b1 = b0 + P.n * LP;
    const int64_t c = int64_t(blockIdx.x) * L + threadIdx.x;
    const bool live = c < inner;
    cplx* col = data + int64_t(blockIdx.y) * nx * inner + c;
    for (int j = threadIdx.y; j < P.n; j += blockDim.y)
        b0[j * LP + threadIdx.x] = (j < nx && live) ? col[int64_t(j) * inner] : cplx{0.0, 0.0};
    __syncthreads();
    cplx* r = fft_lines(b0, b1, P, -1, LP, threadIdx.x, threadIdx.y, blockDim.y);
    for (int j = threadIdx.y; j < P.n; j += blockDim.y) {
        const double kv = live ? kernel[int64_t(j) * inner + c] : 0.0;
        r[j * LP + threadIdx.x] = scale(r[j * LP + threadIdx.x], kv);
    }
    __syncthreads();
    const cplx* v = fft_lines(r, r == b0 ? b1 : b0, P, +1, LP, threadIdx.x, threadIdx.y, blockDim.y);
    if (!live) return;
    for (int j = threadIdx.y; j < nx; j += blockDim.y) col[int64_t(j) * inner] = v[j * LP + threadIdx.x];
}

// Pass 5: half spectrum -> real z lines (z < nz). The full
// spectrum is the Hermitian extension X[N-k] = conj(X[k]); the real part of its inverse is irfft
// (the imaginary parts of the k = 0 and Nyquist terms drop out, as in irfft).
template <int L>
__global__ void __launch_bounds__(256) fft_z_inverse_kernel(const cplx* __restrict__ in, int64_t lines, int nk,
                                                            double* __restrict__ v, int nz, const FftPlan P) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr int LP = L + 1;
    cplx* b0 = reinterpret_cast<cplx*>(smem_raw);
    cplx* b1 = b0 + P.n * LP;
    const int tid = threadIdx.y * L + threadIdx.x;
    const int nthreads = L * blockDim.y;
    const int64_t l0 = int64_t(blockIdx.x) * L;
    const int N = P.n;
    for (int idx = tid; idx < L * nk; idx += nthreads) {
        const int line = idx / nk;
        const int k = idx - line * nk;
        const cplx a = (l0 + line < lines) ? in[(l0 + line) * nk + k] : cplx{0.0, 0.0};
        b0[k * LP + line] = a;
        if (k > 0 && N - k >= nk) b0[(N - k) * LP + line] = {a.re, -a.im};
    }
    __syncthreads();
    const cplx* r = fft_lines(b0, b1, P, +1, LP, threadIdx.x, threadIdx.y, blockDim.y);
    for (int idx = tid; idx < L * nz; idx += nthreads) {
        const int line = idx / nz;
        const int z = idx - line * nz;
        if (l0 + line < lines) v[(l0 + line) * nz + z] = r[z * LP + line].re;
    }
}

// The truncated kernel K(G) = 4 pi (1 - cos(G R)) / G^2, K(0) = 2 pi R^2 (poisson.py:43-64) at the
// frequencies f (cycles per bohr).
__device__ __forceinline__ double cutoff_kernel(double f0, double f1, double f2, double radius) {
    const double two_pi = 6.283185307179586;
    const double kx = two_pi * f0, ky = two_pi * f1, kz = two_pi * f2;
    const double g_sq = kx * kx + ky * ky + kz * kz;
    if (!(g_sq > 0.0)) return 2.0 * 3.141592653589793 * radius * radius;
    const double g = sqrt(g_sq);
    return 4.0 * 3.141592653589793 * (1.0 - cos(g * radius)) / g_sq;
}

// K on the half-spectrum grid (Nx, Ny, Nz/2+1), laid out [kx][ky][kz].
__global__ void kernel_table_kernel(double* __restrict__ out, int n0, int n1, int n2, int nk2, double spacing,
                                    double radius) {
    const int64_t total = static_cast<int64_t>(n0) * n1 * nk2;
    for (int64_t idx = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; idx < total;
         idx += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        const int i2 = static_cast<int>(idx % nk2);
        const int i1 = static_cast<int>((idx / nk2) % n1);
        const int i0 = static_cast<int>(idx / (static_cast<int64_t>(nk2) * n1));
        // fftfreq: i / (n d) for i < ceil(n/2), (i - n) / (n d) above; times 2 pi.
        const double f0 = (i0 < (n0 + 1) / 2 ? i0 : i0 - n0) / (n0 * spacing);
        const double f1 = (i1 < (n1 + 1) / 2 ? i1 : i1 - n1) / (n1 * spacing);
        const double f2 = i2 / (n2 * spacing);
        out[idx] = cutoff_kernel(f0, f1, f2, radius);
    }
}

// ---- K carried over to the lengths M = 2n - 1 or a little more (reduce_kernel_table). K is even along every
// axis, so per axis K_M = T K_N on the half spectra i <= N/2, a <= M/2 with
//   T[i][a] = (mult_i / N) sum_{|m| < n} cos(2 pi i m / N) cos(2 pi a m / M),
// mult_i = 1 for i = 0 and i = N/2, else 2. T and the sums are formed in pairs of doubles (high and low
// parts), from cosines made in long double on the host, so that K_M is K_N's rounding and no more:
// with T in plain doubles the solve's error at 65^3 grew from 2.0e-16 to 3.4e-16.
struct pair2 {
    double hi, lo;
};

// a + x y, with the rounding errors carried
__device__ __forceinline__ pair2 add_product(pair2 a, pair2 x, pair2 y) {
    const double p = __dmul_rn(x.hi, y.hi);
    const double e = fma(x.hi, y.hi, -p) + fma(x.hi, y.lo, x.lo * y.hi);
    const double s = __dadd_rn(a.hi, p), z = __dsub_rn(s, a.hi);
    const double t = __dadd_rn(__dsub_rn(a.hi, __dsub_rn(s, z)), __dsub_rn(p, z));
    return {s, a.lo + (t + e)};
}

__device__ __forceinline__ pair2 normalised(pair2 a) {
    const double s = __dadd_rn(a.hi, a.lo);
    return {s, __dsub_rn(a.lo, __dsub_rn(s, a.hi))};
}

// cosn[j] = cos(2 pi j / len_n), cosm likewise.
__global__ void transfer_kernel(int n, int len_n, int len_m, const pair2* __restrict__ cosn,
                                const pair2* __restrict__ cosm, pair2* __restrict__ t) {
    const int rows = len_n / 2 + 1, cols = len_m / 2 + 1;
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= rows * cols) return;
    const int i = k / cols, a = k % cols;
    pair2 sum{0.5, 0.0};  // half of m = 0; the terms of m and -m are equal
    int jn = 0, jm = 0;
    for (int m = 1; m < n; ++m) {
        jn += i;
        if (jn >= len_n) jn -= len_n;
        jm += a;
        if (jm >= len_m) jm -= len_m;
        sum = add_product(sum, cosn[jn], cosm[jm]);
    }
    sum = normalised(sum);
    // times mult_i 2 / len_n: a power of two over an integer, the quotient with its remainder
    const double mult = (i == 0 || 2 * i == len_n) ? 2.0 : 4.0;
    const double q = sum.hi / len_n;
    const double r = (fma(-q, static_cast<double>(len_n), sum.hi) + sum.lo) / len_n;
    t[k] = {mult * q, mult * r};
}

// K at the half-spectrum points i0 <= N0/2 and so on: [i0][i1][i2].
__global__ void kernel_octant_kernel(pair2* __restrict__ out, int n0, int n1, int n2, double spacing, double radius) {
    const int h1 = n1 / 2 + 1, h2 = n2 / 2 + 1;
    const int64_t total = int64_t(n0 / 2 + 1) * h1 * h2;
    for (int64_t idx = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; idx < total;
         idx += int64_t(gridDim.x) * blockDim.x)
        out[idx] = {cutoff_kernel(static_cast<int>(idx / (int64_t(h1) * h2)) / (n0 * spacing),
                                  static_cast<int>(idx / h2 % h1) / (n1 * spacing),
                                  static_cast<int>(idx % h2) / (n2 * spacing), radius),
                    0.0};
}

// out[o][a][r] = sum_i T[i][a] in[o][i][r] (i < rows, a < cols, r < inner).
__global__ void contract_kernel(const pair2* __restrict__ in, int64_t outer, int rows, int64_t inner,
                                const pair2* __restrict__ t, int cols, pair2* __restrict__ out) {
    const int64_t total = outer * cols * inner;
    for (int64_t idx = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; idx < total;
         idx += int64_t(gridDim.x) * blockDim.x) {
        const int64_t r = idx % inner, a = idx / inner % cols, o = idx / (inner * cols);
        const pair2* src = in + o * rows * inner + r;
        pair2 sum{0.0, 0.0};
        for (int i = 0; i < rows; ++i) sum = add_product(sum, t[int64_t(i) * cols + a], src[i * inner]);
        out[idx] = normalised(sum);
    }
}

// The half-spectrum octant unfolded to [M0][M1][M2/2+1], with the 1 / (M0 M1 M2) of the inverse transform
// (rounded with each value: as one factor of the results it would shift them all alike).
__global__ void unfold_kernel(const pair2* __restrict__ in, int m0, int m1, int nk, double points,
                              double* __restrict__ out) {
    const int64_t total = int64_t(m0) * m1 * nk;
    for (int64_t idx = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; idx < total;
         idx += int64_t(gridDim.x) * blockDim.x) {
        const int k = static_cast<int>(idx % nk), j = static_cast<int>(idx / nk % m1);
        const int i = static_cast<int>(idx / (int64_t(nk) * m1));
        const pair2 v = in[(int64_t(min(i, m0 - i)) * (m1 / 2 + 1) + min(j, m1 - j)) * nk + k];
        const double q = v.hi / points;
        out[idx] = q + (fma(-q, points, v.hi) + v.lo) / points;
    }
}

constexpr int kPoissonSmem = 200 * 1024;
constexpr int kThreads = 256;

// Lines per CTA for transforms of length n: 8 while two [n][9] complex buffers fit, else 4. (At
// n = 180, 32 systems: 8 lines 3.0 ms per solve, 16 lines 3.8 ms -- two CTAs per SM instead of
// four -- and 4 lines 3.9 ms.)
int lines_for(int n) { return size_t(2) * n * 9 * sizeof(cplx) <= size_t(kPoissonSmem) ? 8 : 4; }

size_t smem_for(int n, int L) { return size_t(2) * n * (L + 1) * sizeof(cplx); }

template <int L>
int configure_lines() {
    int st = check(cudaFuncSetAttribute(fft_z_forward_kernel<L>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        kPoissonSmem));
    if (st == CDFTB_OK)
        st = check(cudaFuncSetAttribute(fft_middle_kernel<L>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        kPoissonSmem));
    if (st == CDFTB_OK)
        st = check(cudaFuncSetAttribute(fft_x_fused_kernel<L>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        kPoissonSmem));
    if (st == CDFTB_OK)
        st = check(cudaFuncSetAttribute(fft_z_inverse_kernel<L>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        kPoissonSmem));
    return st;
}

int configure_poisson_kernels() {
    const int st = configure_lines<8>();
    return st == CDFTB_OK ? configure_lines<4>() : st;
}

// cos(2 pi j / n) in long double, the angle reduced to a small one exactly in integers.
long double cosine(int64_t j, int64_t n) {
    constexpr long double pi = 3.14159265358979323846264338327950288L;
    j %= n;
    if (2 * j > n) j = n - j;                                            // cos(2 pi - x) = cos x
    if (4 * j > n) return -cosine(n - 2 * j, 2 * n);                     // cos(pi - x) = -cos x
    return 8 * j > n ? sinl(pi * (n - 4 * j) / (2 * n)) : cosl(2 * pi * j / n);  // cos(pi/2 - x) = sin x
}

// exp(-2 pi i j / n) rounded to double.
cplx unit_root_host(int64_t j, int64_t n) {
    j %= n;
    return {static_cast<double>(cosine(j, n)), static_cast<double>(-cosine(4 * j + 3 * n, 4 * n))};  // sin x = cos(x - pi/2)
}

// Stage list and twiddle table (host, double) of a length-n transform; false if n is not 2,3,5-smooth
// or has too many stages.
bool make_fft_plan(int n, FftPlan* plan, cplx** device_tw) {
    FftPlan P{};
    P.n = n;
    int rem = n;
    int radices[MAX_STAGES];
    int count = 0;
    for (int r : {4, 2, 3, 5}) {
        while (rem % r == 0 && count < MAX_STAGES) {
            radices[count++] = r;
            rem /= r;
        }
    }
    if (rem != 1) return false;
    P.nst = count;
    int total = 0;
    int stride = 1;
    for (int st = 0; st < count; ++st) {
        const int r = radices[st];
        const int len = n / stride;
        P.radix[st] = r;
        P.stride[st] = stride;
        P.m[st] = len / r;
        P.tw_off[st] = total;
        total += P.m[st] * (r - 1);
        stride *= r;
    }
    cplx* host = new cplx[total > 0 ? total : 1];
    for (int st = 0; st < count; ++st) {
        const int r = P.radix[st];
        const int len = n / P.stride[st];
        for (int p = 0; p < P.m[st]; ++p)
            for (int k = 1; k < r; ++k) {
                host[P.tw_off[st] + p * (r - 1) + k - 1] = unit_root_host(static_cast<int64_t>(p) * k, len);
            }
    }
    cplx* dev = nullptr;
    bool ok = cudaMalloc(&dev, sizeof(cplx) * (total > 0 ? total : 1)) == cudaSuccess &&
              cudaMemcpy(dev, host, sizeof(cplx) * (total > 0 ? total : 1), cudaMemcpyHostToDevice) == cudaSuccess;
    delete[] host;
    if (!ok) {
        cudaFree(dev);
        return false;
    }
    P.tw = dev;
    *plan = P;
    *device_tw = dev;
    return true;
}

// exp(-2 pi i j / n) for j < n into device memory.
bool fill_root_table(int n, cplx* device) {
    cplx* host = new cplx[n];
    for (int j = 0; j < n; ++j) host[j] = unit_root_host(j, n);
    const bool ok = cudaMemcpy(device, host, sizeof(cplx) * n, cudaMemcpyHostToDevice) == cudaSuccess;
    delete[] host;
    return ok;
}

// cos(2 pi j / n) for j < n as pairs, into device memory.
bool fill_cosines(int n, pair2* device) {
    pair2* host = new pair2[n];
    for (int j = 0; j < n; ++j) {
        const long double c = cosine(j, n);
        host[j].hi = static_cast<double>(c);
        host[j].lo = static_cast<double>(c - host[j].hi);
    }
    const bool ok = cudaMemcpy(device, host, sizeof(pair2) * n, cudaMemcpyHostToDevice) == cudaSuccess;
    delete[] host;
    return ok;
}

// The small-DFT roots of unity in constant memory (this device's copy of the module).
int load_unit_roots() {
    cplx host[720];
    for (int j = 0; j < 720; ++j) host[j] = unit_root_host(j, 720);
    return check(cudaMemcpyToSymbol(kUnit720, host, sizeof(host)));
}

}  // namespace

}  // namespace cdftb

using namespace cdftb;

// A plan: padded shape and K there, the transform lengths with K carried over to them, the FFT plan of
// each axis, and the two transform buffers.
struct cdftb_poisson_plan {
    int n[3];
    int pad[3];
    int len[3];      // transform lengths (convolution_length)
    int nk;          // len[2]/2 + 1
    double spacing;
    double radius;
    double* kernel;  // K [pad0][pad1][pad2/2+1] (cdftb_poisson_kernel_table)
    double* table;   // K carried over, [len0][len1][nk]
    FftPlan fft[3];
    cplx* tw[3];
    cplx* twn[3];  // W_M^j, j < len[d] (the four-step kernels' outer twiddles)
    int four[3][2];  // the four-step factor pair of each axis, {0, 0} if its length has none
    cplx* a;  // [batch][n0][n1][nk]
    cplx* b;  // [batch][n0][len1][nk]
    void* memory;  // the one allocation that holds them (and, while the plan is made, the reduction's scratch)
    int max_batch;
};

static void free_plan(cdftb_poisson_plan* p) {
    cudaFree(p->memory);
    for (int d = 0; d < 3; ++d) cudaFree(p->tw[d]);
    delete p;
}

// Elements of reduce_kernel_table's two stages, matrix and cosines.
struct ReduceScratch {
    int64_t stage = 1, matrix = 0, cosines = 0;
    int64_t total() const { return 2 * stage + matrix + 2 * cosines; }
};

static ReduceScratch reduce_scratch(const cdftb_poisson_plan* p) {
    ReduceScratch r;
    for (int d = 0; d < 3; ++d) {
        const int64_t half_n = p->pad[d] / 2 + 1, half_m = p->len[d] / 2 + 1;
        r.stage *= std::max(half_n, half_m);
        r.matrix = std::max(r.matrix, half_n * half_m);
        r.cosines = std::max<int64_t>(r.cosines, std::max(p->pad[d], p->len[d]));
    }
    return r;
}

// K on the transform lengths: p->table from the definition's octant, one axis at a time.
static int reduce_kernel_table(cdftb_poisson_plan* p, pair2* scratch) {
    const ReduceScratch size = reduce_scratch(p);
    pair2 *work[2] = {scratch, scratch + size.stage}, *t = scratch + 2 * size.stage;
    pair2 *cosn = t + size.matrix, *cosm = cosn + size.cosines;
    const unsigned blocks = 148 * 16;
    kernel_octant_kernel<<<blocks, 256>>>(work[0], p->pad[0], p->pad[1], p->pad[2], p->spacing, p->radius);
    int st = check_launch();
    int at = 0, half[3];
    for (int d = 0; d < 3; ++d) half[d] = p->pad[d] / 2 + 1;
    for (int d = 2; d >= 0 && st == CDFTB_OK; --d) {
        if (p->pad[d] == p->len[d]) continue;
        const int rows = half[d], cols = p->len[d] / 2 + 1;
        // (the copies wait for the kernels before them on the default stream)
        if (!fill_cosines(p->pad[d], cosn) || !fill_cosines(p->len[d], cosm)) return CDFTB_ERR_LAUNCH;
        transfer_kernel<<<static_cast<unsigned>(ceil_div(int64_t(rows) * cols, 128)), 128>>>(p->n[d], p->pad[d],
                                                                                             p->len[d], cosn, cosm, t);
        if ((st = check_launch()) != CDFTB_OK) break;
        int64_t outer = 1, inner = 1;
        for (int e = 0; e < d; ++e) outer *= half[e];
        for (int e = d + 1; e < 3; ++e) inner *= half[e];
        contract_kernel<<<blocks, 256>>>(work[at], outer, rows, inner, t, cols, work[1 - at]);
        st = check_launch();
        half[d] = cols;
        at = 1 - at;
    }
    if (st != CDFTB_OK) return st;
    const double points = static_cast<double>(p->len[0]) * p->len[1] * p->len[2];
    unfold_kernel<<<blocks, 256>>>(work[at], p->len[0], p->len[1], p->nk, points, p->table);
    return check_launch();
}

extern "C" int cdftb_poisson_plan_create(int nx, int ny, int nz, double spacing, double pad_factor, int max_batch,
                                         void** plan_out, int* padded_shape_out, double* cutoff_radius_out) {
    if (!plan_out || nx <= 0 || ny <= 0 || nz <= 0 || !(spacing > 0.0) || pad_factor < 2.0 || max_batch < 1)
        return CDFTB_ERR_ARGUMENT;
    auto* p = new cdftb_poisson_plan{};
    p->n[0] = nx;
    p->n[1] = ny;
    p->n[2] = nz;
    for (int d = 0; d < 3; ++d) {
        p->pad[d] = fft_friendly(static_cast<int>(ceil(pad_factor * p->n[d])));
        p->len[d] = convolution_length(p->n[d]);
    }
    p->nk = p->len[2] / 2 + 1;
    p->spacing = spacing;
    double r = 1e300;
    for (int d = 0; d < 3; ++d) r = fmin(r, p->pad[d] * spacing);
    p->radius = 0.5 * r;
    p->max_batch = max_batch;
    // the sizes refused are those the definition's own lengths are refused at
    for (int d = 0; d < 3; ++d)
        if (smem_for(p->pad[d], lines_for(p->pad[d])) > size_t(kPoissonSmem)) {
            delete p;
            return CDFTB_ERR_CAPACITY;
        }
    const int nk_pad = p->pad[2] / 2 + 1;
    const int64_t nkern = static_cast<int64_t>(p->pad[0]) * p->pad[1] * nk_pad;
    const int64_t ntable = static_cast<int64_t>(p->len[0]) * p->len[1] * p->nk;
    int st = configure_poisson_kernels();
    if (st != CDFTB_OK) {
        delete p;
        return st;
    }
    const int64_t na = static_cast<int64_t>(max_batch) * nx * ny * p->nk;
    const int64_t nb = static_cast<int64_t>(max_batch) * nx * p->len[1] * p->nk;
    const int64_t buffers = std::max<int64_t>((na + nb) * sizeof(cplx), reduce_scratch(p).total() * sizeof(pair2));
    auto aligned = [](int64_t bytes) { return (bytes + 255) / 256 * 256; };
    int64_t bytes = aligned(nkern * 8) + aligned(ntable * 8) + aligned(buffers);
    for (int d = 0; d < 3; ++d) bytes += aligned(p->len[d] * sizeof(cplx));
    st = check(cudaMalloc(&p->memory, bytes));
    char* at = static_cast<char*>(p->memory);
    auto take = [&](int64_t size) {
        char* r = at;
        at += aligned(size);
        return r;
    };
    p->kernel = reinterpret_cast<double*>(take(nkern * 8));
    p->table = reinterpret_cast<double*>(take(ntable * 8));
    for (int d = 0; d < 3; ++d) p->twn[d] = reinterpret_cast<cplx*>(take(p->len[d] * sizeof(cplx)));
    p->a = reinterpret_cast<cplx*>(take(buffers));
    p->b = p->a + na;
    for (int d = 0; d < 3 && st == CDFTB_OK; ++d) {
        if (fourstep_pair(p->len[d], &p->four[d][0], &p->four[d][1])) {
            if (!fill_root_table(p->len[d], p->twn[d])) st = CDFTB_ERR_LAUNCH;
        } else if (!make_fft_plan(p->len[d], &p->fft[d], &p->tw[d])) {
            st = CDFTB_ERR_LAUNCH;
        }
    }
    if (st == CDFTB_OK) st = load_unit_roots();
    if (st == CDFTB_OK) {
        kernel_table_kernel<<<static_cast<unsigned>(ceil_div(nkern, 256)), 256>>>(p->kernel, p->pad[0], p->pad[1],
                                                                                  p->pad[2], nk_pad, spacing, p->radius);
        st = check_launch();
        if (st == CDFTB_OK) st = reduce_kernel_table(p, reinterpret_cast<pair2*>(p->a));
        if (st == CDFTB_OK) st = check(cudaDeviceSynchronize());
    }
    if (st != CDFTB_OK) {
        free_plan(p);
        return st;
    }
    if (padded_shape_out)
        for (int d = 0; d < 3; ++d) padded_shape_out[d] = p->pad[d];
    if (cutoff_radius_out) *cutoff_radius_out = p->radius;
    *plan_out = p;
    return CDFTB_OK;
}

extern "C" int cdftb_poisson_plan_destroy(void* plan) {
    auto* p = static_cast<cdftb_poisson_plan*>(plan);
    if (!p) return CDFTB_OK;
    free_plan(p);
    return CDFTB_OK;
}

extern "C" int cdftb_poisson_kernel_table(void* plan, const double** table_out) {
    auto* p = static_cast<cdftb_poisson_plan*>(plan);
    if (!p || !table_out) return CDFTB_ERR_ARGUMENT;
    *table_out = p->kernel;
    return CDFTB_OK;
}

namespace {

template <int L>
int run_passes(cdftb_poisson_plan* p, const double* density, double* potential, int batch, cudaStream_t s, int which) {
    const int nx = p->n[0], ny = p->n[1], nz = p->n[2];
    const int N0 = p->len[0], N1 = p->len[1], N2 = p->len[2], nk = p->nk;
    const int64_t lines = static_cast<int64_t>(batch) * nx * ny;
    const dim3 blk(L, kThreads / L);
    switch (which) {
        case 1:
            fft_z_forward_kernel<L><<<static_cast<unsigned>(ceil_div(lines, L)), blk, smem_for(N2, L), s>>>(
                density, lines, nz, p->a, nk, p->fft[2]);
            break;
        case 2: {
            dim3 grid(static_cast<unsigned>(batch * nx), static_cast<unsigned>(ceil_div(nk, L)));
            fft_middle_kernel<L><<<grid, blk, smem_for(N1, L), s>>>(p->a, static_cast<int64_t>(ny) * nk, ny, p->b,
                                                                   static_cast<int64_t>(N1) * nk, N1, nk, p->fft[1], -1);
            break;
        }
        case 3: {
            const int64_t inner = static_cast<int64_t>(N1) * nk;
            dim3 grid(static_cast<unsigned>(ceil_div(inner, L)), static_cast<unsigned>(batch));
            fft_x_fused_kernel<L><<<grid, blk, smem_for(N0, L), s>>>(p->b, nx, inner, p->table, p->fft[0]);
            break;
        }
        case 4: {
            dim3 grid(static_cast<unsigned>(batch * nx), static_cast<unsigned>(ceil_div(nk, L)));
            fft_middle_kernel<L><<<grid, blk, smem_for(N1, L), s>>>(p->b, static_cast<int64_t>(N1) * nk, N1, p->a,
                                                                   static_cast<int64_t>(ny) * nk, ny, nk, p->fft[1], +1);
            break;
        }
        default: {
            fft_z_inverse_kernel<L><<<static_cast<unsigned>(ceil_div(lines, L)), blk, smem_for(N2, L), s>>>(
                p->a, lines, nk, potential, nz, p->fft[2]);
            break;
        }
    }
    return check_launch();
}

// One pass with the four-step kernels (the axis length has a factor pair).
int run_fourstep(cdftb_poisson_plan* p, const double* density, double* potential, int batch, cudaStream_t s, int pass) {
    const int nx = p->n[0], ny = p->n[1], nz = p->n[2];
    const int N1 = p->len[1], nk = p->nk;
    const int d = pass == 3 ? 0 : (pass == 1 || pass == 5 ? 2 : 1);
    const int A = p->four[d][0], B = p->four[d][1];
    const cplx* twn = p->twn[d];
    const int64_t lines = static_cast<int64_t>(nx) * ny;
    const int64_t inner = static_cast<int64_t>(N1) * nk;
    const int64_t small = static_cast<int64_t>(ny) * nk;
    const dim3 grid = pass == 3 ? dim3(static_cast<unsigned>(ceil_div(inner, kLines4)), static_cast<unsigned>(batch))
                      : d == 1  ? dim3(static_cast<unsigned>(batch * nx), static_cast<unsigned>(ceil_div(nk, kLines4)))
                                : dim3(static_cast<unsigned>(ceil_div(lines, 2 * kLines4)), static_cast<unsigned>(batch));
#define CDFTB_X4(A_, B_)                                                                                              \
    if (A == A_ && B == B_) {                                                                                         \
        switch (pass) {                                                                                               \
            case 1: fft_z_forward_fourstep_kernel<A_, B_><<<grid, kThreads4, 0, s>>>(density, lines, nz, p->a, nk, twn); break; \
            case 2: fft_middle_fourstep_kernel<A_, B_, -1><<<grid, kThreads4, 0, s>>>(p->a, small, ny, p->b, inner, N1, nk, twn); break; \
            case 3: fft_x_fourstep_kernel<A_, B_><<<grid, kThreads4, 0, s>>>(p->b, nx, inner, p->table, twn); break;  \
            case 4: fft_middle_fourstep_kernel<A_, B_, +1><<<grid, kThreads4, 0, s>>>(p->b, inner, N1, p->a, small, ny, nk, twn); break; \
            default: fft_z_inverse_fourstep_kernel<A_, B_><<<grid, kThreads4, 0, s>>>(p->a, lines, nk, potential, nz, twn); break; \
        }                                                                                                             \
        return check_launch();                                                                                        \
    }
    CDFTB_FOURSTEP_PAIRS(CDFTB_X4)
#undef CDFTB_X4
    return CDFTB_ERR_ARGUMENT;
}

}  // namespace

extern "C" int cdftb_poisson_solve(void* plan, const double* density, double* potential, int batch,
                                   cdftb_stream_t stream) {
    auto* p = static_cast<cdftb_poisson_plan*>(plan);
    if (!p || !density || !potential || batch < 1 || batch > p->max_batch) return CDFTB_ERR_ARGUMENT;
    if (static_cast<int64_t>(batch) * p->n[0] > 0x7fffffff) return CDFTB_ERR_CAPACITY;
    cudaStream_t s = as_stream(stream);
    const int axis_of_pass[6] = {0, 2, 1, 0, 1, 2};
    for (int pass = 1; pass <= 5; ++pass) {
        if (p->four[axis_of_pass[pass]][0] != 0) {
            const int st = run_fourstep(p, density, potential, batch, s, pass);
            if (st != CDFTB_OK) return st;
            continue;
        }
        const int n = p->len[axis_of_pass[pass]];
        const int st = lines_for(n) == 8 ? run_passes<8>(p, density, potential, batch, s, pass)
                                         : run_passes<4>(p, density, potential, batch, s, pass);
        if (st != CDFTB_OK) return st;
    }
    return CDFTB_OK;
}
