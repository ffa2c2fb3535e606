// knc_physics64.cuh — the FP64 zone and face arithmetic with few FP64
// instructions.
//
// The same expressions, in the same order and with the same roundings, as the
// templates of knc_physics.cuh give for double (which stay as the plain forms
// that an operand outside fp64's fast range falls back to). What differs is
// which pipe the work runs on (knc_fp64.cuh):
//   - divisions and square roots run on the integer and FP32 pipes; divisions
//     by one number share its start;
//   - so do comparisons, minima and halvings, and an exact product by a power
//     of two joins the addition that follows it;
//   - the flow through a face that is supersonic on both sides (an expanding
//     envelope, a wind, a beam along its axis) is its upwind side's flux: a
//     FP32 estimate with a margin far above its error decides that first, and
//     then neither the other side nor a wave speed is formed in FP64. A face
//     the estimate does not decide takes the full solve.
// FP64 instructions of a relativistic HLLE face: 20 supersonic, 111 otherwise
// (the plain form: about 240).
#pragma once

#include "knc_bits.cuh"
#include "knc_fp64.cuh"
#include "knc_physics.cuh"

namespace knc {

// ---- plain forms, out of line ---------------------------------------------------
static __device__ __noinline__ void riemann_plain(PhysT<double> ph, const double* pl, const double* pr, int axis,
                                                  double* out) {
    double l[5], r[5], o[5];
    for (int q = 0; q < 5; ++q) {
        l[q] = pl[q];
        r[q] = pr[q];
    }
    riemann(ph, l, r, l[4], r[4], axis, o);
    for (int q = 0; q < 5; ++q) out[q] = o[q];
}

static __device__ __noinline__ int srhd_c2p_plain(double gm, const double* U, double guess, double* P, int* iterations,
                                                  double* bad) {
    return srhd_c2p_newton_plain(gm, U, guess, P, *iterations, *bad);
}

// ---- supersonic faces -----------------------------------------------------------
// x in FP32, truncated, saturated at FP32's largest number (infinities and
// NaNs too), zero below its normal range.
__device__ __forceinline__ float estimate_f32(double x) {
    const uint32_t hi = hi_word(x), h = hi & 0x7fffffffu;
    const uint32_t c = max(min(h, 0x47efffffu), 0x38000000u) - 0x38000000u;
    return __uint_as_float(__funnelshift_l(lo_word(x), c, 3) | (hi & 0x80000000u));
}

// +1 (-1): the fastest left-going (right-going) wave of this state certainly
// moves right (left), 0: undecided. The FP32 estimate of a^2 and b^2, whose
// difference decides the sign of the wave speed (a -+ b) / (1 - v^2 cs^2), is
// good to 1e-4 for k = 1 - cs^2 > 0.01; the FP64 expression it stands for
// itself to 1e-8 for W^2 < 1e8; the margin is 2%. That holds for numbers the
// estimate neither saturates nor flushes: rho and p (unless it is zero) inside
// FP32's normal range with room for p / rho, and u_n^2 far above the smallest
// FP32 number, so that what underflows on the way to b^2 is too small to
// matter against a^2. Everything else is undecided, NaNs among it (they
// saturate, above every upper bound here).
template <bool SRHD>
__device__ __forceinline__ int sure_direction(float gm, float gh, const double* P, int axis) {
    const float rho = estimate_f32(P[0]), pre = estimate_f32(P[3]);
    const float un = estimate_f32(axis == 0 ? P[1] : P[2]);
    const float t = pre / rho, u2 = un * un;
    bool sure;
    if (SRHD) {
        const float ut = estimate_f32(axis == 0 ? P[2] : P[1]);
        const float w2 = 1.0f + u2 + ut * ut;
        const float o = 1.0f / w2;                     // 1 - v^2
        const float c2 = gm * t / (1.0f + gh * t);
        const float k = 1.0f - c2;
        const float a2 = u2 * o * k * k;
        const float b2 = c2 * o * (o + ut * ut * o * k);
        sure = w2 < 1e8f && k > 0.01f && a2 > 1.02f * b2;
    } else {
        sure = u2 > 1.02f * gm * t;
    }
    const bool cold = ((hi_word(P[3]) << 1) | lo_word(P[3])) == 0u;
    sure = sure && rho > 1e-30f && rho < 1e30f && (cold || (pre > 1e-36f && pre < 1e36f)) && t < 1e30f &&
           u2 > 1e-30f && u2 < 1e30f;
    return sure ? (un > 0.0f ? 1 : -1) : 0;
}

// ---- one side of a face ---------------------------------------------------------
// Component order here: D, normal, tangential momentum, tau, scalar.
struct Side64 {
    double U[5], F[5];
    double lm, lp, vn, pre;
};

// Flux of a side that carries a supersonic face. odd: an operand left the
// fast range (the caller repeats the face in the plain form).
template <bool SRHD>
__device__ __forceinline__ void upwind_flux64(const PhysT<double>& ph, double rho, double un, double ut, double pre,
                                              double s, bool axis1, double F[5], bool& odd) {
    if (SRHD) {
        odd = odd || fp64_odd_divisor(rho) || fp64_odd_numerator(pre) || fp64_odd_numerator(un);
        // u_r^2 + u_theta^2, whichever of the two is normal
        const double uu = un * un + ut * ut;
        const double w2 = 1.0 + uu;
        odd = odd || fp64_odd_positive(w2);
        const Start64 yw = rsqrt_start(w2);
        const double w = fp64_sqrt(w2, yw);
        const double h = 1.0 + fp64_div(pre, rho, rcp_start(rho)) * ph.gh;
        const double d = rho * w;
        const double m = d * h;
        const double vn = fp64_div(un, w, yw);
        F[0] = d * vn;
        F[1] = m * un * vn + pre;
        F[2] = m * ut * vn;
        F[3] = (m * w - pre - d + pre) * vn;
        F[4] = s * un;
    } else {
        odd = odd || fp64_odd_divisor(rho) || fp64_odd_numerator(pre);
        F[0] = rho * un;
        F[1] = rho * un * un + pre;
        F[2] = rho * ut * un;
        const double vr = axis1 ? ut : un, vq = axis1 ? un : ut;
        const double E = fp64_div(pre, ph.gm1, rcp_start(ph.gm1)) + fp64_half(rho) * (vr * vr + vq * vq);
        F[3] = (E + pre) * un;
        F[4] = s * un;
    }
}

template <bool SRHD>
__device__ __forceinline__ void side64(const PhysT<double>& ph, double rho, double un, double ut, double pre, double s,
                                       bool axis1, Side64& S, bool& odd) {
    odd = odd || fp64_odd_divisor(rho) || fp64_odd_numerator(pre) || (SRHD && fp64_odd_numerator(un));
    if (SRHD) {
        const double uu = un * un + ut * ut;
        const double w2 = 1.0 + uu;
        const Start64 yw = rsqrt_start(w2);
        const double w = fp64_sqrt(w2, yw);
        const double h = 1.0 + fp64_div(pre, rho, rcp_start(rho)) * ph.gh;
        const double d = rho * w;
        const double m = d * h;
        const double vn = fp64_div(un, w, yw);
        const double rh = rho * h;
        const double cs2 = fp64_div(ph.gm * pre, rh, rcp_start(rh));
        const double v2 = fp64_div(uu, w2, rcp_start(w2));
        const double k = 1.0 - cs2;
        const double a = vn * k;
        const double den = 1.0 - v2 * cs2;
        const double arg = cs2 * (1.0 - v2) * (den - vn * vn * k);
        odd = odd || fp64_odd_positive(w2) || fp64_odd_numerator(uu) || fp64_odd_divisor(rh) ||
              fp64_odd_positive(arg) || fp64_odd_positive(den);
        const double b = fp64_sqrt(arg, rsqrt_start(arg));
        const double inv = fp64_rcp(den, rcp_start(den));
        S.lm = (a - b) * inv;
        S.lp = (a + b) * inv;
        S.U[0] = d;
        S.U[1] = m * un;
        S.U[2] = m * ut;
        S.U[3] = m * w - pre - d;
        S.U[4] = s * w;
        S.F[4] = s * un;
        S.vn = vn;
    } else {
        const double cs2 = fp64_div(ph.gm * pre, rho, rcp_start(rho));
        odd = odd || fp64_odd_positive(cs2);
        const double cs = fp64_sqrt(cs2, rsqrt_start(cs2));
        const double vr = axis1 ? ut : un, vq = axis1 ? un : ut;
        S.lm = un - cs;
        S.lp = un + cs;
        S.U[0] = rho;
        S.U[1] = rho * un;
        S.U[2] = rho * ut;
        S.U[3] = fp64_div(pre, ph.gm1, rcp_start(ph.gm1)) + fp64_half(rho) * (vr * vr + vq * vq);
        S.U[4] = s;
        S.F[4] = s * un;
        S.vn = un;
    }
    S.F[0] = S.U[0] * S.vn;
    S.F[1] = S.U[1] * S.vn + pre;
    S.F[2] = S.U[2] * S.vn;
    S.F[3] = (S.U[3] + pre) * S.vn;
    S.pre = pre;
}

// ---- face fluxes from both sides (components as in Side64) ------------------------
__device__ __forceinline__ void hlle64(const Side64& L, const Side64& R, double out[5], bool& odd) {
    const double am = fp64_min(L.lm, R.lm), ap = fp64_max(L.lp, R.lp);
    if (fp64_ge0(am)) {
#pragma unroll
        for (int q = 0; q < 5; ++q) out[q] = L.F[q];
    } else if (fp64_le0(ap)) {
#pragma unroll
        for (int q = 0; q < 5; ++q) out[q] = R.F[q];
    } else {
        const double w = ap - am;
        odd = odd || fp64_odd_divisor(w);
        const double inv = fp64_rcp(w, rcp_start(w));
        const double apam = ap * am;
#pragma unroll
        for (int q = 0; q < 5; ++q) out[q] = (ap * L.F[q] - am * R.F[q] + apam * (R.U[q] - L.U[q])) * inv;
    }
}

__device__ __forceinline__ void srhd_hllc64(const Side64& L, const Side64& R, double out[5], bool& odd) {
    const double am = fp64_min(L.lm, R.lm), ap = fp64_max(L.lp, R.lp);
    if (fp64_ge0(am)) {
#pragma unroll
        for (int q = 0; q < 5; ++q) out[q] = L.F[q];
        return;
    }
    if (fp64_le0(ap)) {
#pragma unroll
        for (int q = 0; q < 5; ++q) out[q] = R.F[q];
        return;
    }
    const double wd = ap - am;
    odd = odd || fp64_odd_divisor(wd);
    const double inv = fp64_rcp(wd, rcp_start(wd));
    const double apam = ap * am;
    double Uh[4], Fh[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        if (q == 2) continue;   // the contact speed takes D, normal momentum and tau
        Uh[q] = (ap * R.U[q] - am * L.U[q] - (R.F[q] - L.F[q])) * inv;
        Fh[q] = (ap * L.F[q] - am * R.F[q] + apam * (R.U[q] - L.U[q])) * inv;
    }
    const double e_hll = Uh[3] + Uh[0];
    const double fe_hll = Fh[3] + Fh[0];
    const double m_hll = Uh[1];
    const double fm_hll = Fh[1];
    const double bq = e_hll + fm_hll;
    // bq^2 - 4 fe m (a negative or vanishing one is odd); 2 m / den as m / (den / 2)
    const double disc = __fma_rn(-4.0, __dmul_rn(fe_hll, m_hll), __dmul_rn(bq, bq));
    odd = odd || fp64_odd_positive(disc);
    const double den = bq + fp64_sqrt(disc, rsqrt_start(disc));
    odd = odd || fp64_odd_divisor(den) || fp64_odd_numerator(m_hll);
    const double half = fp64_half(den);
    const double lstar = fp64_div(m_hll, half, rcp_start(half));
    const double pstar = fm_hll - fe_hll * lstar;
    const bool left = fp64_ge0(lstar);
    const double lam = left ? am : ap;
    const double ll = lam - lstar;
    odd = odd || fp64_odd_divisor(ll);
    const double fac = fp64_rcp(ll, rcp_start(ll));
    const double vk = left ? L.vn : R.vn, pk = left ? L.pre : R.pre;
    const double lv = lam - vk;
    double U[5], F[5];
#pragma unroll
    for (int q = 0; q < 5; ++q) {
        U[q] = left ? L.U[q] : R.U[q];
        F[q] = left ? L.F[q] : R.F[q];
    }
    const double e_k = U[3] + U[0];
    double Us[5];
    Us[0] = U[0] * lv * fac;
    Us[1] = (U[1] * lv + pstar - pk) * fac;
    Us[2] = U[2] * lv * fac;
    const double e_s = (e_k * lv + pstar * lstar - pk * vk) * fac;
    Us[3] = e_s - Us[0];
    Us[4] = U[4] * lv * fac;
#pragma unroll
    for (int q = 0; q < 5; ++q) out[q] = F[q] + lam * (Us[q] - U[q]);
}

__device__ __forceinline__ void newt_hllc64(const Side64& L, const Side64& R, double out[5], bool& odd) {
    const double am = fp64_min(L.lm, R.lm), ap = fp64_max(L.lp, R.lp);
    if (fp64_ge0(am)) {
#pragma unroll
        for (int q = 0; q < 5; ++q) out[q] = L.F[q];
        return;
    }
    if (fp64_le0(ap)) {
#pragma unroll
        for (int q = 0; q < 5; ++q) out[q] = R.F[q];
        return;
    }
    const double dl = am - L.vn, dr = ap - R.vn;
    const double ql = L.U[0] * dl;
    const double qr = R.U[0] * dr;
    const double num = R.pre - L.pre + L.U[1] * dl - R.U[1] * dr;
    const double den = ql - qr;
    odd = odd || fp64_odd_numerator(num) || fp64_odd_divisor(den);
    const double sstar = fp64_div(num, den, rcp_start(den));
    const bool left = fp64_ge0(sstar);
    const double lam = left ? am : ap;
    const double vk = left ? L.vn : R.vn, pk = left ? L.pre : R.pre;
    double U[5], F[5];
#pragma unroll
    for (int q = 0; q < 5; ++q) {
        U[q] = left ? L.U[q] : R.U[q];
        F[q] = left ? L.F[q] : R.F[q];
    }
    const double rho = U[0];
    const double lv = left ? dl : dr;   // lam - v of the side
    const double rl = rho * lv, ls = lam - sstar;
    odd = odd || fp64_odd_divisor(rl) || fp64_odd_divisor(ls) || fp64_odd_numerator(U[2]) || fp64_odd_numerator(U[3]);
    const Start64 yr = rcp_start(rho), yl = rcp_start(ls);
    const double fac = fp64_div(rl, ls, yl);
    double Us[5];
    Us[0] = fac;
    Us[1] = fac * sstar;
    Us[2] = fac * fp64_div(U[2], rho, yr);
    Us[3] = fac * (fp64_div(U[3], rho, yr) + (sstar - vk) * (sstar + fp64_div(pk, rl, rcp_start(rl))));
    const double us = U[4] * lv;
    odd = odd || fp64_odd_numerator(us);
    Us[4] = fp64_div(us, ls, yl);
#pragma unroll
    for (int q = 0; q < 5; ++q) out[q] = F[q] + lam * (Us[q] - U[q]);
}

// The flux through a face (normal `axis`: 0 radial, 1 polar) between the
// states pl and pr (rho, u_r, u_theta, p, s), components (D, S_r, S_theta, tau, s).
template <bool SRHD, bool HLLC>
__device__ __forceinline__ void face64(const PhysT<double>& ph, float gmf, float ghf, const double* pl, const double* pr,
                                       int axis, double out[5]) {
    const bool ax = axis != 0;
    bool odd = false;
    double f[5];
    const int dl = sure_direction<SRHD>(gmf, ghf, pl, axis), dr = sure_direction<SRHD>(gmf, ghf, pr, axis);
    if (dl * dr > 0) {
        double v[5];
#pragma unroll
        for (int q = 0; q < 5; ++q) v[q] = dl > 0 ? pl[q] : pr[q];
        upwind_flux64<SRHD>(ph, v[0], ax ? v[2] : v[1], ax ? v[1] : v[2], v[3], v[4], ax, f, odd);
    } else {
        Side64 L, R;
        side64<SRHD>(ph, pl[0], ax ? pl[2] : pl[1], ax ? pl[1] : pl[2], pl[3], pl[4], ax, L, odd);
        side64<SRHD>(ph, pr[0], ax ? pr[2] : pr[1], ax ? pr[1] : pr[2], pr[3], pr[4], ax, R, odd);
        if (!HLLC) hlle64(L, R, f, odd);
        else if (SRHD) srhd_hllc64(L, R, f, odd);
        else newt_hllc64(L, R, f, odd);
    }
    out[0] = f[0];
    out[1] = ax ? f[2] : f[1];
    out[2] = ax ? f[1] : f[2];
    out[3] = f[3];
    out[4] = f[4];
    if (odd) {
        double a[5], b[5], o[5];
#pragma unroll
        for (int q = 0; q < 5; ++q) {
            a[q] = pl[q];
            b[q] = pr[q];
        }
        riemann_plain(ph, a, b, axis, o);
#pragma unroll
        for (int q = 0; q < 5; ++q) out[q] = o[q];
    }
}

// Geometric sources per unit volume of the momenta (sources; D's and tau's vanish).
template <bool SRHD>
__device__ __forceinline__ void sources64(const PhysT<double>& ph, const double* P, double r, double cot, double& s1,
                                          double& s2) {
    const double rho = P[0], ur = P[1], uq = P[2], pre = P[3];
    bool odd = fp64_odd_divisor(r) || (SRHD && (fp64_odd_divisor(rho) || fp64_odd_numerator(pre)));
    const double mass = SRHD ? rho * (1.0 + fp64_div(pre, rho, rcp_start(rho)) * ph.gh) : rho;
    const double n1 = __fma_rn(2.0, pre, mass * uq * uq);
    const double n2 = pre * cot - mass * ur * uq;
    odd = odd || fp64_odd_numerator(n1) || fp64_odd_numerator(n2);
    const Start64 y = rcp_start(r);
    s1 = fp64_div(n1, r, y);
    s2 = fp64_div(n2, r, y);
    if (odd) {
        const double m = SRHD ? rho * (1.0 + pre / rho * ph.gh) : rho;
        s1 = (2.0 * pre + m * uq * uq) / r;
        s2 = (pre * cot - m * ur * uq) / r;
    }
}

// ---- slopes ---------------------------------------------------------------------
// x / 2 as x * 0.5 rounds it, on the integer pipe: the exponent of normal
// numbers less one; from 2^-1021 down the bits are the number in units of
// 2^-1074, halved with ties to even; infinities and NaNs stay.
__device__ __forceinline__ double half64(double x) {
    const uint32_t h = hi_word(x) & 0x7fffffffu;
    if (h - (2u << 20) < (2045u << 20)) return fp64_half(x);
    if (h >= 0x7ff00000u) return x;
    const unsigned long long m = magnitude(x), half = (m >> 1) + (m & (m >> 1) & 1ull);
    return __longlong_as_double((long long)(half | ((unsigned long long)(hi_word(x) & 0x80000000u) << 32)));
}

// Half of plm_gradient from x = theta (b - a), z = theta (c - b) and s = c - a
// (whose half is the third candidate): x is the neighbour's z, so a slope
// costs three FP64 instructions, the differences and one product. The
// magnitudes are compared as integers; a NaN gives zero, as the comparisons of
// plm_gradient do.
__device__ __forceinline__ double half_slope64(double x, double s, double z) {
    const double y = half64(s);
    const unsigned long long mx = magnitude(x), my = magnitude(y), mz = magnitude(z);
    unsigned long long m = mx < mz ? mx : mz;
    m = m < my ? m : my;
    const uint32_t hx = hi_word(x), hy = hi_word(y), hz = hi_word(z);
    const bool agree = (int32_t)((hx ^ hy) | (hx ^ hz)) >= 0;
    const uint32_t top = max(max(hx & 0x7fffffffu, hy & 0x7fffffffu), hz & 0x7fffffffu);
    if (!agree || top >= 0x7ff80000u) return 0.0;
    const double g = half64(__longlong_as_double((long long)m));
    return words(hi_word(g) | (hx & 0x80000000u), lo_word(g));
}

// ---- primitive recovery -----------------------------------------------------------
// One Newton step of srhd_c2p_newton (p -> p - f / f'), the residual f. ZERO:
// p is 0, as in the first step from the plain guess (its products with p and
// sums with p drop out exactly). mt = m + tau.
template <bool ZERO>
__device__ __forceinline__ double newton_step64(double gm, double m, double tau, double mt, double ss, double& p,
                                                double& w, Start64& yw, bool& odd) {
    const double et = ZERO ? mt : tau + p + m;
    const double inv = fp64_rcp(et, rcp_start(et));
    const double bmax = 1.0 - 1e-10;
    double b2 = ss * inv * inv;
    if (magnitude(b2) >= (unsigned long long)__double_as_longlong(bmax)) b2 = bmax;
    const double omb = 1.0 - b2;
    const double w2 = fp64_rcp(omb, rcp_start(omb));
    yw = rsqrt_start(w2);
    w = fp64_sqrt(w2, yw);
    const double x = ZERO ? tau + m * (1.0 - w) : tau + m * (1.0 - w) + p * (1.0 - w2);
    const double de = x * omb;
    const double dh = ZERO ? m * omb * w + de : m * omb * w + de + p;
    const double f = ZERO ? de * (gm - 1.0) : de * (gm - 1.0) - p;
    const double num = f * dh;
    const double den = ZERO ? -dh : b2 * gm * p - dh;
    odd = odd || fp64_odd_divisor(et) || fp64_odd_numerator(num) || fp64_odd_divisor(den);
    const double step = fp64_div(num, den, rcp_start(den));
    p = ZERO ? -step : p - step;
    return f;
}

// srhd_c2p_newton_plain with the same results; a zone whose numbers leave the
// fast range repeats in the plain form.
__device__ __forceinline__ int srhd_c2p_newton(double gm, const double* U, double guess, double* P, int& iterations,
                                               double& bad) {
    const double m = U[0];
    const double tau = U[3];
    iterations = 0;
    if (fp64_negative(m)) { bad = m; return HYDRO_NEGATIVE_DENSITY; }
    if (fp64_negative(tau)) { bad = tau; return HYDRO_NEGATIVE_ENERGY_DENSITY; }
    bool odd = false;
    const double ss = U[1] * U[1] + U[2] * U[2];
    const double mt = m + tau;
    const double tol = NEWTON_TOLERANCE * mt;
    double p = guess, w0 = 1.0;
    Start64 yw = {0u, 0u, 0.0f};
    bool found = false;
    int n = 0;
    if (guess == 0.0) {
        const double f = newton_step64<true>(gm, m, tau, mt, ss, p, w0, yw, odd);
        n = 1;
        found = magnitude(f) < magnitude(tol);
    }
    while (!found && n < NEWTON_ITER_MAX && !odd) {
        const double f = newton_step64<false>(gm, m, tau, mt, ss, p, w0, yw, odd);
        ++n;
        found = magnitude(f) < magnitude(tol);
    }
    iterations = n;
    const double et = mt + p;
    odd = odd || !found || fp64_odd_divisor(et) || fp64_odd_numerator(m);
    const double n1 = w0 * U[1], n2 = w0 * U[2];
    odd = odd || fp64_odd_numerator(n1) || fp64_odd_numerator(n2);
    const Start64 ye = rcp_start(et);
    P[0] = fp64_div(m, w0, yw);
    P[1] = fp64_div(n1, et, ye);
    P[2] = fp64_div(n2, et, ye);
    P[3] = p;
    if (odd) {
        double u[4] = {m, U[1], U[2], tau}, v[4] = {0.0, 0.0, 0.0, 0.0}, b = 0.0;
        int it = 0;
        const int kind = srhd_c2p_plain(gm, u, guess, v, &it, &b);
        iterations = it;
        bad = b;
#pragma unroll
        for (int q = 0; q < 4; ++q) P[q] = v[q];
        return kind;
    }
    if (fp64_negative(p)) {
        P[3] = PRESSURE_FLOOR * P[0];
        return HYDRO_NEGATIVE_PRESSURE;
    }
    return HYDRO_NONE;
}

// U / dV of a zone's five volume integrals.
__device__ __forceinline__ void per_volume64(const double (&U)[5], double dV, double (&u)[5]) {
    bool odd = fp64_odd_divisor(dV);
    const Start64 y = rcp_start(dV);
#pragma unroll
    for (int q = 0; q < 5; ++q) {
        odd = odd || fp64_odd_numerator(U[q]);
        u[q] = fp64_div(U[q], dV, y);
    }
    if (odd) {
#pragma unroll 1
        for (int q = 0; q < 5; ++q) u[q] = U[q] / dV;
    }
}

// newt_c2p with the same results.
__device__ __forceinline__ int newt_c2p64(double gm1, const double* U, double* P, double& bad) {
    const double rho = U[0];
    if (fp64_odd_positive(rho) || fp64_odd_numerator(U[1]) || fp64_odd_numerator(U[2]))
        return newt_c2p(gm1, U, P, bad);
    const Start64 y = rcp_start(rho);
    const double vr = fp64_div(U[1], rho, y), vq = fp64_div(U[2], rho, y);
    P[0] = rho;
    P[1] = vr;
    P[2] = vq;
    P[3] = (U[3] - fp64_half(rho) * (vr * vr + vq * vq)) * gm1;
    return HYDRO_NONE;
}

// sqrt(1 + u^2) and x / W with it (x the scalar mass per volume), for a
// recovered four-velocity.
__device__ __forceinline__ double over_lorentz64(double x, double ur, double uq) {
    const double w2 = 1.0 + ur * ur + uq * uq;
    if (fp64_odd_positive(w2) || fp64_odd_numerator(x)) return x / sqrt(w2);
    const Start64 y = rsqrt_start(w2);
    return fp64_div(x, fp64_sqrt(w2, y), y);
}

// a / b
static __device__ __noinline__ double div_plain(double a, double b) { return a / b; }
__device__ __forceinline__ double div64(double a, double b) {
    if (fp64_odd_numerator(a) || fp64_odd_divisor(b)) return div_plain(a, b);
    return fp64_div(a, b, rcp_start(b));
}

// newton_fast in FP64 (the criterion on the residual alone) with its reciprocals, square root and
// comparisons off the FP64 pipe; false also for operands outside the fast range
// (the callers then take the plain recovery).
__device__ __forceinline__ bool newton_fast64(double m, double ss, double tau, double gm, double p, double tol,
                                              double& p_out, double& w_out, int& iters) {
    const double bmax = 1.0 - 1e-10;
    for (int n = 0; n < NEWTON_ITER_MAX; ++n) {
        const double et = tau + p + m;
        if (fp64_odd_divisor(et)) return false;
        const double inv = fp64_rcp(et, rcp_start(et));
        double b2 = ss * inv * inv;
        if (magnitude(b2) >= (unsigned long long)__double_as_longlong(bmax)) b2 = bmax;
        const double omb = 1.0 - b2;
        const Start64 y = rsqrt_start(omb);
        const double r = fp64_sqrt(omb, y);
        const double w = fp64_rcp(r, y);
        const double X = tau + m * (1.0 - w) + p * (1.0 - w * w);
        const double de = X * omb;
        const double f = (gm - 1.0) * de - p;
        const double dh = m * omb * w + de + p;
        const double den = b2 * gm * p - dh;
        const double num = f * dh;
        if (fp64_odd_divisor(den) || fp64_odd_numerator(num)) return false;
        p = p - fp64_div(num, den, rcp_start(den));
        iters = n + 1;
        if (magnitude(f) < magnitude(tol)) {
            p_out = p;
            w_out = w;
            return !is_nan_bits(p);
        }
    }
    return false;
}

// Max signal speed of a primitive state (max_signal_speed).
__device__ __forceinline__ double max_signal_speed64(const PhysT<double>& ph, const double* P) {
    bool odd = false;
    double a;
    if (ph.srhd) {
        Side64 S, T;
        side64<true>(ph, P[0], P[1], P[2], P[3], 0.0, false, S, odd);
        side64<true>(ph, P[0], P[2], P[1], P[3], 0.0, true, T, odd);
        unsigned long long m = magnitude(S.lm);
        m = max(m, magnitude(S.lp));
        m = max(m, magnitude(T.lm));
        m = max(m, magnitude(T.lp));
        a = __longlong_as_double((long long)m);
    } else {
        const double v2 = P[1] * P[1] + P[2] * P[2];
        const double c2 = fp64_div(ph.gm * P[3], P[0], rcp_start(P[0]));
        odd = fp64_odd_divisor(P[0]) || fp64_odd_numerator(P[3]) || fp64_odd_positive(c2) ||
              (v2 != 0.0 && fp64_odd_positive(v2));
        const double v = v2 != 0.0 ? fp64_sqrt(v2, rsqrt_start(v2)) : 0.0;
        a = v + fp64_sqrt(c2, rsqrt_start(c2));
    }
    return odd ? max_signal_speed(ph, P) : a;
}

}  // namespace knc
