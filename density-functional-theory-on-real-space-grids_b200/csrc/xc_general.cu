// (d) Every native semi-local functional of the reference, spin-restricted or spin-polarised, with
// its first derivatives. The reference writes each functional once as an energy density of the
// per-spin ingredients (n_up, n_dn, sigma_uu, sigma_ud, sigma_dd) and differentiates it with
// autograd (src/cdft/xc/base.py:115-189); here the same energy densities are evaluated on
// forward-mode dual numbers, so v_xc and v_sigma are exact derivatives of the energy density (to
// rounding). An LDA carries its two density partials through; a GGA is assembled from parts of two or
// three variables, each with the partials of those, which the chain rule joins (Gga below).
//
// Conventions kept from base.py:45-80, 171-189:
//   - n_spin = 1: n_up = n_dn = n/2 and sigma_uu = sigma_ud = sigma_dd = sigma/4; n_spin = 2: the
//     rows as given, sigma ordered (uu, ud, dd);
//   - a point with n_up + n_dn < 1e-14 is empty: e = v = v_sigma = 0;
//   - each density channel is clamped at 0.5e-14 and sigma_uu, sigma_dd at 1e-40 (sigma_ud is not
//     clamped); a clamped input passes no derivative (torch's clamp_min rule), and neither does a
//     clamped spin polarisation (base.py:218-226).
// The spin-restricted derivatives follow the chain rule of that split: v = (dE/dn_up + dE/dn_dn)/2,
// v_sigma = (dE/dsigma_uu + dE/dsigma_ud + dE/dsigma_dd)/4.
//
// Functionals (the name table of src/cdft/xc/dispatch.py:26-44), by cdftb_xc_id in cdftb.h:
//   LDA: Slater (lda.py:37-46), VWN5 (lda.py:113-159), PW92 in the original and modified parameter
//   sets (lda.py:49-110), PZ81 (lda.py:162-195); GGA: PBE x (gga.py:43-59), PBE c (gga.py:62-90),
//   B88 x (gga.py:93-122), LYP c (gga.py:125-159); and the combinations lda_vwn, lda_pw92,
//   lda_pw92_mod, lda_pz81, pbe, blyp.

#include "common.cuh"

namespace cdftb {
namespace {

constexpr double kPiX = 3.141592653589793;

// ---- forward-mode dual numbers with N partials
template <int N>
struct Dual {
    double v;
    double d[N];
};

template <int N>
__device__ __forceinline__ Dual<N> constant(double x) {
    Dual<N> r;
    r.v = x;
#pragma unroll
    for (int k = 0; k < N; ++k) r.d[k] = 0.0;
    return r;
}

template <int N>
__device__ __forceinline__ Dual<N> variable(double x, int k) {
    Dual<N> r = constant<N>(x);
    if (k < N) r.d[k] = 1.0;
    return r;
}

// x with every partial scaled by s (the chain rule of a unary function with derivative s)
template <int N>
__device__ __forceinline__ Dual<N> chain(double value, double s, const Dual<N>& x) {
    Dual<N> r;
    r.v = value;
#pragma unroll
    for (int k = 0; k < N; ++k) r.d[k] = s * x.d[k];
    return r;
}

template <int N>
__device__ __forceinline__ Dual<N> operator+(const Dual<N>& a, const Dual<N>& b) {
    Dual<N> r;
    r.v = a.v + b.v;
#pragma unroll
    for (int k = 0; k < N; ++k) r.d[k] = a.d[k] + b.d[k];
    return r;
}
template <int N>
__device__ __forceinline__ Dual<N> operator+(const Dual<N>& a, double b) {
    Dual<N> r = a;
    r.v = a.v + b;
    return r;
}
template <int N>
__device__ __forceinline__ Dual<N> operator+(double a, const Dual<N>& b) {
    Dual<N> r = b;
    r.v = a + b.v;
    return r;
}
template <int N>
__device__ __forceinline__ Dual<N> operator-(const Dual<N>& a) {
    Dual<N> r;
    r.v = -a.v;
#pragma unroll
    for (int k = 0; k < N; ++k) r.d[k] = -a.d[k];
    return r;
}
template <int N>
__device__ __forceinline__ Dual<N> operator-(const Dual<N>& a, const Dual<N>& b) {
    Dual<N> r;
    r.v = a.v - b.v;
#pragma unroll
    for (int k = 0; k < N; ++k) r.d[k] = a.d[k] - b.d[k];
    return r;
}
template <int N>
__device__ __forceinline__ Dual<N> operator-(const Dual<N>& a, double b) {
    Dual<N> r = a;
    r.v = a.v - b;
    return r;
}
template <int N>
__device__ __forceinline__ Dual<N> operator-(double a, const Dual<N>& b) {
    Dual<N> r;
    r.v = a - b.v;
#pragma unroll
    for (int k = 0; k < N; ++k) r.d[k] = -b.d[k];
    return r;
}
template <int N>
__device__ __forceinline__ Dual<N> operator*(const Dual<N>& a, const Dual<N>& b) {
    Dual<N> r;
    r.v = a.v * b.v;
#pragma unroll
    for (int k = 0; k < N; ++k) r.d[k] = a.d[k] * b.v + a.v * b.d[k];
    return r;
}
template <int N>
__device__ __forceinline__ Dual<N> operator*(const Dual<N>& a, double b) {
    return chain(a.v * b, b, a);
}
template <int N>
__device__ __forceinline__ Dual<N> operator*(double a, const Dual<N>& b) {
    return chain(a * b.v, a, b);
}
// Quotients through one reciprocal; the value gets the remainder's correction, so it is rounded as a
// division is. (An infinite or zero divisor makes the correction NaN: the product then stands.)
__device__ __forceinline__ double quotient(double a, double b, double inv) {
    const double q = a * inv;
    const double c = fma(fma(-q, b, a), inv, q);
    return c == c ? c : q;
}
template <int N>
__device__ __forceinline__ Dual<N> operator/(const Dual<N>& a, const Dual<N>& b) {
    Dual<N> r;
    const double inv = 1.0 / b.v;
    r.v = quotient(a.v, b.v, inv);
#pragma unroll
    for (int k = 0; k < N; ++k) r.d[k] = (a.d[k] - r.v * b.d[k]) * inv;
    return r;
}
template <int N>
__device__ __forceinline__ Dual<N> operator/(const Dual<N>& a, double b) {
    return chain(a.v / b, 1.0 / b, a);
}
template <int N>
__device__ __forceinline__ Dual<N> operator/(double a, const Dual<N>& b) {
    const double inv = 1.0 / b.v;
    const double q = quotient(a, b.v, inv);
    return chain(q, -q * inv, b);
}

template <int N>
__device__ __forceinline__ Dual<N> dsqrt(const Dual<N>& x) {
    const double s = sqrt(x.v);
    return chain(s, 0.5 / s, x);
}
template <int N>
__device__ __forceinline__ Dual<N> dlog(const Dual<N>& x) {
    return chain(log(x.v), 1.0 / x.v, x);
}
template <int N>
__device__ __forceinline__ Dual<N> dlog1p(const Dual<N>& x) {
    return chain(log1p(x.v), 1.0 / (1.0 + x.v), x);
}
template <int N>
__device__ __forceinline__ Dual<N> dexp(const Dual<N>& x) {
    const double e = exp(x.v);
    return chain(e, e, x);
}
template <int N>
__device__ __forceinline__ Dual<N> datan(const Dual<N>& x) {
    return chain(atan(x.v), 1.0 / (1.0 + x.v * x.v), x);
}
template <int N>
__device__ __forceinline__ Dual<N> dasinh(const Dual<N>& x) {
    return chain(asinh(x.v), 1.0 / sqrt(1.0 + x.v * x.v), x);
}
// x^p with autograd's rule p x^(p-1), by the cube root or products
template <int N>
__device__ __forceinline__ Dual<N> square(const Dual<N>& x) {
    return chain(x.v * x.v, 2.0 * x.v, x);
}
template <int N>
__device__ __forceinline__ Dual<N> cube(const Dual<N>& x) {
    return chain(x.v * x.v * x.v, 3.0 * (x.v * x.v), x);
}
template <int N>
__device__ __forceinline__ Dual<N> fourth(const Dual<N>& x) {
    const double x2 = x.v * x.v;
    return chain(x2 * x2, 4.0 * (x2 * x.v), x);
}
template <int N>
__device__ __forceinline__ Dual<N> pow23(const Dual<N>& x) {
    const double c = cbrt(x.v);
    return chain(c * c, (2.0 / 3.0) / c, x);
}
template <int N>
__device__ __forceinline__ Dual<N> pow43(const Dual<N>& x) {
    const double c = cbrt(x.v);
    return chain(x.v * c, fma(c, 1.0 / 3.0, c), x);
}
template <int N>
__device__ __forceinline__ Dual<N> clamp_min(const Dual<N>& x, double floor) {
    return x.v >= floor ? x : constant<N>(floor);
}
template <int N>
__device__ __forceinline__ Dual<N> clamp(const Dual<N>& x, double lo, double hi) {
    if (x.v < lo) return constant<N>(lo);
    if (x.v > hi) return constant<N>(hi);
    return x;
}

// ---- shared building blocks (base.py:196-235)
constexpr double kRsX = 0.62035049089940001667;       // (3 / (4 pi))^(1/3)
constexpr double kCbrt2X = 1.25992104989487316477;    // 2^(1/3)
constexpr double kSlaterX = 0.73855876638202240588;   // (3/4) (3/pi)^(1/3)
constexpr double kFermiX = 3.09366772628013593097;    // (3 pi^2)^(1/3)
constexpr double kSlaterSpin = 0.93052573634910002500;  // 2^(1/3) (3/4) (3/pi)^(1/3) = (3/2) (3 / (4 pi))^(1/3)
constexpr double kPbeGamma = 0.03109069086965489503;  // (1 - log 2) / pi^2

// n^(-1/3); r_s is kRsX times it
template <int N>
__device__ __forceinline__ Dual<N> inverse_cbrt(const Dual<N>& n) {
    const double c = 1.0 / cbrt(n.v);
    return chain(c, (-1.0 / 3.0) * c / n.v, n);
}
template <int N>
__device__ __forceinline__ Dual<N> wigner_seitz(const Dual<N>& n) {
    return kRsX * inverse_cbrt(n);
}
template <int N>
__device__ __forceinline__ Dual<N> polarisation(const Dual<N>& up, const Dual<N>& dn) {
    return clamp((up - dn) / (up + dn), -1.0 + 1.0e-15, 1.0 - 1.0e-15);
}
template <int N>
__device__ __forceinline__ Dual<N> f_zeta(const Dual<N>& z) {
    return (pow43(1.0 + z) + pow43(1.0 - z) - 2.0) * (1.0 / (2.0 * kCbrt2X - 2.0));
}
constexpr double kFpp0 = 4.0 / (9.0 * (kCbrt2X - 1.0));

// para + alpha f (1 - z^4) / f''(0) + (ferro - para) f z^4. (With equal channels f, f' and z are zero and the
// para part is all of it: the callers' POL = false.)
template <int N>
__device__ __forceinline__ Dual<N> interpolate_spin(const Dual<N>& para, const Dual<N>& ferro,
                                                    const Dual<N>& alpha_c, const Dual<N>& zeta, double fpp0) {
    const Dual<N> fz = f_zeta(zeta);
    const Dual<N> z4 = fourth(zeta);
    return para + alpha_c * fz * (1.0 - z4) * (1.0 / fpp0) + (ferro - para) * fz * z4;
}

template <int N>
__device__ __forceinline__ Dual<N> slater(const Dual<N>& up, const Dual<N>& dn) {
    return -kSlaterSpin * (pow43(up) + pow43(dn));
}

// ---- VWN5 (lda.py:113-159)
struct Vwn {
    double a, x0, b, c;
};
template <int N>
__device__ __forceinline__ Dual<N> vwn_aux(const Dual<N>& x, Vwn p) {
    const Dual<N> big_x = x * x + p.b * x + p.c;
    const double big_x0 = p.x0 * p.x0 + p.b * p.x0 + p.c;
    const double q = sqrt(4.0 * p.c - p.b * p.b);
    const Dual<N> at = datan(q / (2.0 * x + p.b));
    return p.a * (dlog(x * x / big_x) + (2.0 * p.b / q) * at -
                  (p.b * p.x0 / big_x0) * (dlog(square(x - p.x0) / big_x) + (2.0 * (p.b + 2.0 * p.x0) / q) * at));
}
template <bool POL, int N>
__device__ __forceinline__ Dual<N> vwn5(const Dual<N>& up, const Dual<N>& dn) {
    const Dual<N> n = up + dn;
    const Dual<N> x = dsqrt(wigner_seitz(n));
    const Dual<N> para = vwn_aux(x, Vwn{0.0310907, -0.10498, 3.72744, 12.9352});
    if constexpr (!POL) return n * para;
    const Dual<N> ferro = vwn_aux(x, Vwn{0.01554535, -0.32500, 7.06042, 18.0578});
    const Dual<N> alpha_c = vwn_aux(x, Vwn{-1.0 / (6.0 * kPiX * kPiX), -0.0047584, 1.13107, 13.0045});
    return n * interpolate_spin(para, ferro, alpha_c, polarisation(up, dn), kFpp0);
}

// ---- PW92 (lda.py:49-110)
struct Pw {
    double a, a1, b1, b2, b3, b4;
};
template <int N>
__device__ __forceinline__ Dual<N> pw92_g(const Dual<N>& rs, const Dual<N>& s, Pw p) {
    const Dual<N> den = 2.0 * p.a * (p.b1 * s + p.b2 * rs + p.b3 * rs * s + p.b4 * rs * rs);
    return -2.0 * p.a * (1.0 + p.a1 * rs) * dlog1p(1.0 / den);
}
template <bool POL, int N>
__device__ __forceinline__ Dual<N> pw92_epsilon(const Dual<N>& rs, const Dual<N>& zeta, bool modified) {
    const Pw para_p = modified ? Pw{0.0310907, 0.21370, 7.5957, 3.5876, 1.6382, 0.49294}
                               : Pw{0.031091, 0.21370, 7.5957, 3.5876, 1.6382, 0.49294};
    const Pw ferro_p = modified ? Pw{0.01554535, 0.20548, 14.1189, 6.1977, 3.3662, 0.62517}
                                : Pw{0.015545, 0.20548, 14.1189, 6.1977, 3.3662, 0.62517};
    const Pw stiff_p = modified ? Pw{0.0168869, 0.11125, 10.357, 3.6231, 0.88026, 0.49671}
                                : Pw{0.016887, 0.11125, 10.357, 3.6231, 0.88026, 0.49671};
    const double fpp0 = modified ? kFpp0 : 1.709921;
    const Dual<N> s = dsqrt(rs);
    const Dual<N> para = pw92_g(rs, s, para_p);
    if constexpr (!POL) return para;
    const Dual<N> ferro = pw92_g(rs, s, ferro_p);
    const Dual<N> alpha_c = -pw92_g(rs, s, stiff_p);
    return interpolate_spin(para, ferro, alpha_c, zeta, fpp0);
}
template <bool POL, int N>
__device__ __forceinline__ Dual<N> pw92(const Dual<N>& up, const Dual<N>& dn, bool modified) {
    const Dual<N> n = up + dn;
    return n * pw92_epsilon<POL>(wigner_seitz(n), polarisation(up, dn), modified);
}

// ---- PZ81 (lda.py:162-195)
struct Pz {
    double gamma, b1, b2, a, b, c, d;
};
template <int N>
__device__ __forceinline__ Dual<N> pz81_epsilon(const Dual<N>& rs, Pz p) {
    if (rs.v >= 1.0) return p.gamma / (1.0 + p.b1 * dsqrt(rs) + p.b2 * rs);
    const Dual<N> l = dlog(rs);
    return p.a * l + p.b + p.c * rs * l + p.d * rs;
}
template <bool POL, int N>
__device__ __forceinline__ Dual<N> pz81(const Dual<N>& up, const Dual<N>& dn) {
    const Dual<N> n = up + dn;
    const Dual<N> rs = wigner_seitz(n);
    const Dual<N> para = pz81_epsilon(rs, Pz{-0.1423, 1.0529, 0.3334, 0.0311, -0.048, 0.0020, -0.0116});
    if constexpr (!POL) return n * para;
    const Dual<N> ferro = pz81_epsilon(rs, Pz{-0.0843, 1.3981, 0.2611, 0.01555, -0.0269, 0.0007, -0.0048});
    return n * (para + f_zeta(polarisation(up, dn)) * (ferro - para));
}

// ---- GGA. Each is assembled from parts of few variables, with the partials of those only (a quantity of
// the densities alone carries two, a channel of exchange its density and its sigma), and the chain rule
// joins them. With that, powers of a third by the cube root instead of pow, and quotients sharing a
// reciprocal, spin-polarised BLYP at 275 k points takes 19 us (FP64 issue; 78 us with five partials through
// every operation and two pow per power), and every value is nearer to the multi-precision one: a pow
// with the exponent 1/3 rounded to double is off by |log x| / 3 units.
struct Gga {
    double e;
    double dn[2];  // d/dn_up, d/dn_dn
    double ds[3];  // d/dsigma_uu, _ud, _dd
};
__device__ __forceinline__ Gga operator+(const Gga& a, const Gga& b) {
    return {a.e + b.e, {a.dn[0] + b.dn[0], a.dn[1] + b.dn[1]}, {a.ds[0] + b.ds[0], a.ds[1] + b.ds[1], a.ds[2] + b.ds[2]}};
}

// a channel of exchange: variables its density (0) and its sigma (1)
__device__ __forceinline__ Dual<2> pbe_x_channel(const Dual<2>& n, const Dual<2>& s) {
    const double kappa = 0.804, mu = 0.2195149727645171;
    const Dual<2> n2 = 2.0 * n;
    const Dual<2> n43 = pow43(n2);
    const Dual<2> s2 = s / ((kFermiX * kFermiX) * square(n43));
    const Dual<2> fx = 1.0 + kappa - kappa / (1.0 + (mu / kappa) * s2);
    return (-0.5 * kSlaterX) * n43 * fx;
}
__device__ __forceinline__ Dual<2> b88_x_channel(const Dual<2>& n, const Dual<2>& s) {
    const double beta = 0.0042;
    const Dual<2> n43 = pow43(n);
    const Dual<2> x2 = s / square(n43);
    const Dual<2> x = dsqrt(x2);
    return -(n43 * (kSlaterSpin + beta * x2 / (1.0 + 6.0 * beta * x * dasinh(x))));
}
// E(n_up, sigma_uu) + E(n_dn, sigma_dd)
__device__ __forceinline__ Gga both_channels(const Dual<2>& u, const Dual<2>& d) {
    return {u.v + d.v, {u.d[0], d.d[0]}, {u.d[1], 0.0, d.d[1]}};
}

// ---- PBE correlation (gga.py:62-90): n (eps + H(eps, phi, t^2)); eps, phi and t^2 / sigma are functions
// of the densities, H carries its own three partials
template <bool POL>
__device__ __forceinline__ Gga pbe_c(const Dual<2>& up, const Dual<2>& dn, double suu, double sud, double sdd) {
    const double beta = 0.06672455060314922;
    const Dual<2> n = up + dn;
    const Dual<2> n_m13 = inverse_cbrt(n);
    const Dual<2> zeta = polarisation(up, dn);
    const Dual<2> eps = pw92_epsilon<POL>(kRsX * n_m13, zeta, true);
    Dual<2> phi = constant<2>(1.0);
    if constexpr (POL) phi = 0.5 * (pow23(1.0 + zeta) + pow23(1.0 - zeta));
    const double sigma = suu + 2.0 * sud + sdd;
    // t^2 = sigma w, w = 1 / (4 phi^2 k_s^2 n^2), k_s^2 = 4 k_F / pi
    const Dual<2> w = (kPiX / (16.0 * kFermiX)) * n_m13 / square(phi * n);
    const Dual<3> e3 = variable<3>(eps.v, 0), p3 = variable<3>(phi.v, 1), t3 = variable<3>(sigma * w.v, 2);
    const Dual<3> gp3 = kPbeGamma * cube(p3);
    const Dual<3> a = (beta / kPbeGamma) / (dexp(-e3 / gp3) - 1.0);
    const Dual<3> at2 = a * t3;
    const Dual<3> h = gp3 * dlog1p((beta / kPbeGamma) * t3 * (1.0 + at2) / (1.0 + at2 + at2 * at2));
    Gga r;
    r.e = n.v * (eps.v + h.v);
#pragma unroll
    for (int k = 0; k < 2; ++k)
        r.dn[k] = (eps.v + h.v) * n.d[k] +
                  n.v * ((1.0 + h.d[0]) * eps.d[k] + h.d[1] * phi.d[k] + h.d[2] * (sigma * w.d[k]));
    const double ds = n.v * h.d[2] * w.v;
    r.ds[0] = ds;
    r.ds[1] = 2.0 * ds;
    r.ds[2] = ds;
    return r;
}

// ---- LYP (gga.py:125-159): first(n) - a b omega bracket, the bracket linear in the sigmas
__device__ __forceinline__ Gga lyp_c(const Dual<2>& up, const Dual<2>& dn, double suu, double sud, double sdd) {
    const double a = 0.04918, b = 0.132, c = 0.2533, d = 0.349;
    constexpr double c_f = 0.3 * kFermiX * kFermiX;  // 0.3 (3 pi^2)^(2/3)
    const Dual<2> n = up + dn;
    const Dual<2> n_m13 = inverse_cbrt(n);
    const Dual<2> inv_n = 1.0 / n;
    const Dual<2> inv_denom = 1.0 / (1.0 + d * n_m13);
    const Dual<2> omega = (-a * b) * dexp(-c * n_m13) * inv_denom * (square(n_m13) * cube(inv_n));
    const Dual<2> delta = c * n_m13 + d * n_m13 * inv_denom;
    const Dual<2> nab = up * dn;
    const Dual<2> first = (-4.0 * a) * inv_denom * nab * inv_n;
    // x^(8/3) with its derivative 8/3 x^(5/3)
    const double cu = cbrt(up.v), cd = cbrt(dn.v);
    const Dual<2> n83 = chain(up.v * up.v * (cu * cu), (8.0 / 3.0) * up.v * (cu * cu), up) +
                        chain(dn.v * dn.v * (cd * cd), (8.0 / 3.0) * dn.v * (cd * cd), dn);
    constexpr double p113 = 8.0 * kCbrt2X * kCbrt2X;  // 2^(11/3)
    // bracket = nab c0 n83 + sum_s g_s sigma_s
    const Dual<2> g_total = nab * (47.0 / 18.0 - (7.0 / 18.0) * delta) - (2.0 / 3.0) * n * n;  // times sigma
    const Dual<2> g_same = nab * (delta * (1.0 / 18.0) - 2.5);
    const Dual<2> g_part = nab * ((11.0 - delta) * (1.0 / 9.0)) * inv_n;
    const Dual<2> n2_23 = (2.0 / 3.0) * n * n;
    const Dual<2> g_uu = g_total + g_same + g_part * up + (n2_23 - dn * dn);
    const Dual<2> g_dd = g_total + g_same + g_part * dn + (n2_23 - up * up);
    const Dual<2> g_ud = 2.0 * g_total;
    const Dual<2> zero = (p113 * c_f) * nab * n83;
    const Dual<2> bracket = zero + g_uu * suu + g_ud * sud + g_dd * sdd;
    const Dual<2> energy = first + omega * bracket;
    return {energy.v, {energy.d[0], energy.d[1]}, {omega.v * g_uu.v, omega.v * g_ud.v, omega.v * g_dd.v}};
}

// cdftb_xc_id (include/cdftb.h)
enum : int {
    LDA_VWN = CDFTB_XC_LDA_VWN, LDA_PW92 = CDFTB_XC_LDA_PW92, LDA_PW92_MOD = CDFTB_XC_LDA_PW92_MOD,
    LDA_PZ81 = CDFTB_XC_LDA_PZ81, PBE = CDFTB_XC_PBE, BLYP = CDFTB_XC_BLYP, LDA_X = CDFTB_XC_LDA_X,
    LDA_C_VWN = CDFTB_XC_LDA_C_VWN, LDA_C_PW = CDFTB_XC_LDA_C_PW, LDA_C_PW_MOD = CDFTB_XC_LDA_C_PW_MOD,
    LDA_C_PZ = CDFTB_XC_LDA_C_PZ, GGA_X_PBE = CDFTB_XC_GGA_X_PBE, GGA_C_PBE = CDFTB_XC_GGA_C_PBE,
    GGA_X_B88 = CDFTB_XC_GGA_X_B88, GGA_C_LYP = CDFTB_XC_GGA_C_LYP, XC_COUNT = CDFTB_XC_GGA_C_LYP + 1
};

__host__ __device__ constexpr bool is_gga(int id) {
    return id == PBE || id == BLYP || id == GGA_X_PBE || id == GGA_C_PBE || id == GGA_X_B88 || id == GGA_C_LYP;
}

template <int ID, bool POL>
__device__ __forceinline__ Dual<2> lda_energy(const Dual<2>& u, const Dual<2>& dn) {
    if constexpr (ID == LDA_X) return slater(u, dn);
    else if constexpr (ID == LDA_C_VWN) return vwn5<POL>(u, dn);
    else if constexpr (ID == LDA_C_PW) return pw92<POL>(u, dn, false);
    else if constexpr (ID == LDA_C_PW_MOD) return pw92<POL>(u, dn, true);
    else if constexpr (ID == LDA_C_PZ) return pz81<POL>(u, dn);
    else if constexpr (ID == LDA_VWN) return slater(u, dn) + vwn5<POL>(u, dn);
    else if constexpr (ID == LDA_PW92) return slater(u, dn) + pw92<POL>(u, dn, false);
    else if constexpr (ID == LDA_PW92_MOD) return slater(u, dn) + pw92<POL>(u, dn, true);
    else return slater(u, dn) + pz81<POL>(u, dn);  // LDA_PZ81
}

// A clamped input passes no derivative: live[0..1] the densities, live[2..3] sigma_uu and sigma_dd.
template <int ID, bool POL>
__device__ __forceinline__ Gga gga_energy(double nu, double nd, double suu, double sud, double sdd,
                                          const bool (&live)[4]) {
    auto channel = [](double n, double s, bool n_live, bool s_live) {
        Dual<2> r[2] = {constant<2>(n), constant<2>(s)};
        if (n_live) r[0].d[0] = 1.0;
        if (s_live) r[1].d[1] = 1.0;
        if constexpr (ID == PBE || ID == GGA_X_PBE) return pbe_x_channel(r[0], r[1]);
        else return b88_x_channel(r[0], r[1]);
    };
    auto exchange = [&]() {
        const Dual<2> a = channel(nu, suu, live[0], live[2]);
        if constexpr (!POL) return both_channels(a, a);
        return both_channels(a, channel(nd, sdd, live[1], live[3]));
    };
    auto correlation = [&]() {
        Dual<2> u = constant<2>(nu), d = constant<2>(nd);
        if (live[0]) u.d[0] = 1.0;
        if (live[1]) d.d[1] = 1.0;
        Gga r;
        if constexpr (ID == PBE || ID == GGA_C_PBE) r = pbe_c<POL>(u, d, suu, sud, sdd);
        else r = lyp_c(u, d, suu, sud, sdd);
        if (!live[2]) r.ds[0] = 0.0;
        if (!live[3]) r.ds[2] = 0.0;
        return r;
    };
    if constexpr (ID == GGA_X_PBE || ID == GGA_X_B88) return exchange();
    else if constexpr (ID == GGA_C_PBE || ID == GGA_C_LYP) return correlation();
    else return exchange() + correlation();  // PBE, BLYP
}

// One thread per point; rows of `p` points: density (n_spin, p), sigma (1 or 3, p), v (n_spin, p),
// vs (1 or 3, p).
template <int ID, int NS>
__global__ void __launch_bounds__(128) xc_eval_kernel(const double* __restrict__ density,
                                                      const double* __restrict__ sigma, int64_t p,
                                                      double* __restrict__ e, double* __restrict__ v,
                                                      double* __restrict__ vs) {
    constexpr bool GGA = is_gga(ID);
    constexpr bool POL = NS == 2;
    for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < p; i += int64_t(gridDim.x) * blockDim.x) {
        double nu, nd, suu = 0.0, sud = 0.0, sdd = 0.0;
        if (NS == 1) {
            nu = nd = 0.5 * density[i];
            if (GGA) suu = sud = sdd = 0.25 * sigma[i];
        } else {
            nu = density[i];
            nd = density[p + i];
            if (GGA) {
                suu = sigma[i];
                sud = sigma[p + i];
                sdd = sigma[2 * p + i];
            }
        }
        if (!(nu + nd >= 1.0e-14)) {  // an empty point (base.py:176-189)
            e[i] = 0.0;
            v[i] = 0.0;
            if (NS == 2) v[p + i] = 0.0;
            if (GGA) {
                vs[i] = 0.0;
                if (NS == 2) {
                    vs[p + i] = 0.0;
                    vs[2 * p + i] = 0.0;
                }
            }
            continue;
        }
        const double floor = 0.5e-14;
        if constexpr (GGA) {
            const bool live[4] = {nu >= floor, nd >= floor, suu >= 1.0e-40, sdd >= 1.0e-40};
            Gga out = gga_energy<ID, POL>(live[0] ? nu : floor, live[1] ? nd : floor, live[2] ? suu : 1.0e-40, sud,
                                          live[3] ? sdd : 1.0e-40, live);
            if (out.e != out.e) {  // a NaN input: no derivative is a number either, whichever it depends on
#pragma unroll
                for (int k = 0; k < 3; ++k) out.ds[k] = out.e;
            }
            e[i] = out.e;
            if (NS == 1) {
                v[i] = 0.5 * (out.dn[0] + out.dn[1]);
                vs[i] = 0.25 * (out.ds[0] + out.ds[1] + out.ds[2]);
            } else {
                v[i] = out.dn[0];
                v[p + i] = out.dn[1];
                vs[i] = out.ds[0];
                vs[p + i] = out.ds[1];
                vs[2 * p + i] = out.ds[2];
            }
        } else {
            const Dual<2> u = clamp_min(variable<2>(nu, 0), floor);
            const Dual<2> dn = clamp_min(variable<2>(nd, 1), floor);
            const Dual<2> out = lda_energy<ID, POL>(u, dn);
            e[i] = out.v;
            if (NS == 1) {
                v[i] = 0.5 * (out.d[0] + out.d[1]);
            } else {
                v[i] = out.d[0];
                v[p + i] = out.d[1];
            }
        }
    }
}

template <int ID>
int launch_xc(int n_spin, const double* density, const double* sigma, int64_t p, double* e, double* v, double* vs,
              cudaStream_t st) {
    // a grid-stride loop: at most 64 CTAs of 128 threads per SM's worth (148 SMs), fewer for small p
    const unsigned blocks = static_cast<unsigned>(ceil_div(p, 128) < 148 * 16 ? ceil_div(p, 128) : 148 * 16);
    if (n_spin == 1)
        xc_eval_kernel<ID, 1><<<blocks, 128, 0, st>>>(density, sigma, p, e, v, vs);
    else
        xc_eval_kernel<ID, 2><<<blocks, 128, 0, st>>>(density, sigma, p, e, v, vs);
    return check_launch();
}

}  // namespace
}  // namespace cdftb

extern "C" int cdftb_xc_is_gga(int functional) {
    if (functional < 0 || functional >= cdftb::XC_COUNT) return -1;
    return cdftb::is_gga(functional) ? 1 : 0;
}

extern "C" int cdftb_xc_eval_f64(int functional, int n_spin, const double* density, const double* sigma, int64_t p,
                                 double* e, double* v, double* v_sigma, cdftb_stream_t stream) {
    using namespace cdftb;
    if (functional < 0 || functional >= XC_COUNT || (n_spin != 1 && n_spin != 2) || p < 0) return CDFTB_ERR_ARGUMENT;
    if (p == 0) return CDFTB_OK;
    if (!density || !e || !v || (is_gga(functional) && (!sigma || !v_sigma))) return CDFTB_ERR_ARGUMENT;
    cudaStream_t st = as_stream(stream);
    switch (functional) {
        case LDA_VWN: return launch_xc<LDA_VWN>(n_spin, density, sigma, p, e, v, v_sigma, st);
        case LDA_PW92: return launch_xc<LDA_PW92>(n_spin, density, sigma, p, e, v, v_sigma, st);
        case LDA_PW92_MOD: return launch_xc<LDA_PW92_MOD>(n_spin, density, sigma, p, e, v, v_sigma, st);
        case LDA_PZ81: return launch_xc<LDA_PZ81>(n_spin, density, sigma, p, e, v, v_sigma, st);
        case PBE: return launch_xc<PBE>(n_spin, density, sigma, p, e, v, v_sigma, st);
        case BLYP: return launch_xc<BLYP>(n_spin, density, sigma, p, e, v, v_sigma, st);
        case LDA_X: return launch_xc<LDA_X>(n_spin, density, sigma, p, e, v, v_sigma, st);
        case LDA_C_VWN: return launch_xc<LDA_C_VWN>(n_spin, density, sigma, p, e, v, v_sigma, st);
        case LDA_C_PW: return launch_xc<LDA_C_PW>(n_spin, density, sigma, p, e, v, v_sigma, st);
        case LDA_C_PW_MOD: return launch_xc<LDA_C_PW_MOD>(n_spin, density, sigma, p, e, v, v_sigma, st);
        case LDA_C_PZ: return launch_xc<LDA_C_PZ>(n_spin, density, sigma, p, e, v, v_sigma, st);
        case GGA_X_PBE: return launch_xc<GGA_X_PBE>(n_spin, density, sigma, p, e, v, v_sigma, st);
        case GGA_C_PBE: return launch_xc<GGA_C_PBE>(n_spin, density, sigma, p, e, v, v_sigma, st);
        case GGA_X_B88: return launch_xc<GGA_X_B88>(n_spin, density, sigma, p, e, v, v_sigma, st);
        default: return launch_xc<GGA_C_LYP>(n_spin, density, sigma, p, e, v, v_sigma, st);
    }
}
