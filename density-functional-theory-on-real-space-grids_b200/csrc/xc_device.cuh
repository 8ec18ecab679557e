// (d) Spin-restricted LDA (Slater + VWN5) and PBE energy densities with closed-form first
// derivatives, per point. The reference evaluates the same energy densities and differentiates
// them with autograd (src/cdft/xc/base.py:115-189, lda.py:113-159, 201-217, gga.py:28-90); here the
// derivatives are written out by hand. Conventions kept: the density is split n_up = n_dn = n/2
// and each channel clamped at 0.5e-14, a point with n < 1e-14 is empty (e = v = v_sigma = 0),
// sigma_uu = sigma_dd = max(sigma/4, 1e-40) with sigma_ud = sigma/4 unclamped (base.py:45-80,
// 171-189). At zeta = 0 every spin-interpolation term and its derivative vanish.
#pragma once

#include <math.h>

namespace cdftb {
namespace xc {

constexpr double kDensityThreshold = 1.0e-14;
constexpr double kSigmaThreshold = 1.0e-40;
constexpr double kPi = 3.141592653589793;

// What bounds these functions is FP64 issue: the cube root, logarithms, arc tangent and exponential, and
// the divisions, each a sequence of about ten dependent operations. So a point takes one cube root (the
// density's; r_s and k_F are constants over or times it), and quotients that share a denominator share
// its reciprocal. On B200: PBE at 531 k points 28.5 -> 16.4 us, the LDA fused into the grid potentials
// (8.8 M points) 261 -> 193 us.
constexpr double kSlater = 0.73855876638202240588;   // (3/4) (3/pi)^(1/3)
constexpr double kFermi = 3.09366772628013593097;    // (3 pi^2)^(1/3)
constexpr double kRs = 0.62035049089940001667;       // (3 / (4 pi))^(1/3): r_s = kRs n^(-1/3)
constexpr double kRsHalf = 0.49237251092134827059;   // kRs / 2^(1/3): r_s from half the density
constexpr double kSlaterSpin = 0.93052573634910002500;  // 2^(1/3) kSlater

struct VWNParams {
    double a, x0, b, c;
};

// a / b with a reciprocal of b good to a few units in the last place: the remainder's correction makes it
// as exact as the division.
__device__ __forceinline__ double quotient(double a, double b, double inv) {
    const double q = a * inv;
    return fma(fma(-q, b, a), inv, q);
}

// VWN eq. (4.4) fit eps(x) and x d eps/dx (lda.py:122-134). At low density its terms cancel to 1/x^2 of
// their size, so the arguments of the logarithms and of the arc tangent are exact quotients.
__device__ __forceinline__ void vwn_aux(double x, VWNParams p, double& value, double& x_deriv) {
    const double x2 = x * x;
    const double big_x = x2 + p.b * x + p.c;
    const double big_x0 = p.x0 * p.x0 + p.b * p.x0 + p.c;
    const double q = sqrt(4.0 * p.c - p.b * p.b);
    const double dx = 2.0 * x + p.b, xm = x - p.x0;
    // 1/X, 1/(x - x0) and 1/(2x + b) from one division
    const double all = 1.0 / (big_x * xm * dx);
    const double i_dx = all * (big_x * xm), i_xm = all * (big_x * dx), i_x = all * (xm * dx);
    const double at = atan(quotient(q, dx, i_dx));
    const double r = p.b * p.x0 / big_x0;
    value = p.a * (log(quotient(x2, big_x, i_x)) + (2.0 * p.b / q) * at -
                   r * (log(quotient(xm * xm, big_x, i_x)) + (2.0 * (p.b + 2.0 * p.x0) / q) * at));
    x_deriv = p.a * (2.0 - x * (dx + p.b) * i_x - r * (2.0 * x * i_xm - x * (dx + p.b + 2.0 * p.x0) * i_x));
}

// Slater exchange + VWN5 correlation: e (per volume) and v = de/dn.
__device__ __forceinline__ void lda_vwn(double n, double& e, double& v) {
    if (!(n >= kDensityThreshold)) {
        e = 0.0;
        v = 0.0;
        return;
    }
    const double floor = 0.5 * kDensityThreshold;
    const double nu = fmax(0.5 * n, floor);
    constexpr double factor = kSlaterSpin;
    const double nu13 = cbrt(nu);
    const double ex = -factor * (2.0 * (nu * nu13));
    const double vx = -factor * fma(nu13, 1.0 / 3.0, nu13);
    const double nt = nu + nu;
    const double rs = kRsHalf / nu13;
    double eps, x_deps;
    vwn_aux(sqrt(rs), VWNParams{0.0310907, -0.10498, 3.72744, 12.9352}, eps, x_deps);
    e = ex + nt * eps;
    v = vx + eps - (1.0 / 6.0) * x_deps;
}

struct PW92Params {
    double a, a1, b1, b2, b3, b4;
};

// PW92 G(rs) (lda.py:55-61) and rs dG/drs.
__device__ __forceinline__ void pw92_g(double rs, PW92Params p, double& g, double& rs_dg) {
    const double s = sqrt(rs);
    const double den = 2.0 * p.a * (p.b1 * s + p.b2 * rs + p.b3 * rs * s + p.b4 * rs * rs);
    const double rs_dden = 2.0 * p.a * (0.5 * p.b1 * s + p.b2 * rs + 1.5 * p.b3 * rs * s + 2.0 * p.b4 * rs * rs);
    const double both = 1.0 / (den * (den + 1.0));
    const double l = log1p((den + 1.0) * both);
    const double rs_dl = -rs_dden * both;
    g = -2.0 * p.a * (1.0 + p.a1 * rs) * l;
    rs_dg = -2.0 * p.a * p.a1 * rs * l - 2.0 * p.a * (1.0 + p.a1 * rs) * rs_dl;
}

// PBE exchange + correlation (gga.py:28-90): e, v = de/dn, vs = de/dsigma.
__device__ __forceinline__ void pbe(double n, double sigma, double& e, double& v, double& vs) {
    if (!(n >= kDensityThreshold)) {
        e = 0.0;
        v = 0.0;
        vs = 0.0;
        return;
    }
    const double kappa = 0.804, mu = 0.2195149727645171;
    const double beta = 0.06672455060314922;
    constexpr double gamma = 0.03109069086965489503;  // (1 - log 2) / pi^2
    const double floor = 0.5 * kDensityThreshold;
    const double nu = fmax(0.5 * n, floor);
    const double s_quarter = 0.25 * sigma;
    const bool s_clamped = !(s_quarter >= kSigmaThreshold);
    const double s_c = s_clamped ? kSigmaThreshold : s_quarter;
    // exchange: two equal channels of (1/2) e_x^unif(2 n_s) F_x(s^2), and 2 n_s is the density
    const double nt = nu + nu;
    const double n13 = cbrt(nt);
    const double n43 = nt * n13;
    const double i_s = 1.0 / (4.0 * kFermi * kFermi * (n43 * n43));
    const double s2 = 4.0 * s_c * i_s;
    const double i_den = 1.0 / (1.0 + (mu / kappa) * s2);
    const double fx = 1.0 + kappa - kappa * i_den;
    const double dfx = mu * i_den * i_den;
    const double ex = -kSlater * n43 * fx;
    const double vx = kSlater * n13 * (-(4.0 / 3.0) * fx + (8.0 / 3.0) * dfx * s2);
    const double vsx = s_clamped ? 0.0 : -kSlater * n43 * dfx * i_s;
    // correlation: PW92 (modified) at zeta = 0, phi = 1
    const double rs = kRs / n13;
    double eps, rs_deps;
    pw92_g(rs, PW92Params{0.0310907, 0.21370, 7.5957, 3.5876, 1.6382, 0.49294}, eps, rs_deps);
    const double n_deps = rs_deps * (-1.0 / 3.0);  // n d eps / dn
    const double sig_tot = s_c + 2.0 * s_quarter + s_c;
    const double dsig_tot = (s_clamped ? 0.0 : 0.5) + 0.5;
    const double i_t = 1.0 / ((16.0 * kFermi / kPi) * n13 * nt * nt);  // 1 / (4 k_s^2 n^2)
    const double t2 = sig_tot * i_t;
    const double bg = beta / gamma;
    const double ex_eps = exp(eps * (-1.0 / gamma));
    const double i_ex = 1.0 / (ex_eps - 1.0);
    const double a = bg * i_ex;
    const double da_deps = (bg / gamma) * ex_eps * i_ex * i_ex;
    const double at2 = a * t2;
    const double num = t2 * (1.0 + at2);
    const double dd = 1.0 + at2 + at2 * at2;
    const double i_dd = 1.0 / dd;
    const double ratio = num * i_dd;
    const double h = gamma * log1p(bg * ratio);
    const double common = gamma * bg / (1.0 + bg * ratio) * (i_dd * i_dd);
    const double dh_dy = common * ((1.0 + 2.0 * at2) * dd - num * (a + 2.0 * a * at2));
    const double dh_da = common * (t2 * t2 * dd - num * (t2 + 2.0 * at2 * t2));
    const double ec = nt * (eps + h);
    const double vc = eps + h + n_deps * (1.0 + dh_da * da_deps) - (7.0 / 3.0) * dh_dy * t2;
    const double vsc = nt * dh_dy * dsig_tot * i_t;
    e = ex + ec;
    v = vx + vc;
    vs = vsx + vsc;
}

}  // namespace xc
}  // namespace cdftb
