// eu3d_device.cuh — device-side types and per-cell / per-face arithmetic of the
// EU3D reacting-Euler timestep for sm_100a.
//
// Included by the kernel translation units. EU_EXACT_THERMO selects the state
// recovery and EU_EXACT_RATES the rate and trapezoid expressions with the
// reference's operand order and divisions (compiled with --fmad=false they
// round exactly as the reference's CPU build); without them, algebraically
// equivalent fast forms are used. The flux reconstruction has its own switch (EU_EXACT_FLUX).
#pragma once

#include <cmath>
#include <cstdint>
#include <type_traits>

#include <cuda_runtime.h>

#include "eu3d_types.h"

namespace eu3d {

__device__ __forceinline__ long long cell_index(const DevGrid &g, int i, int j, int k)
{
    return ((long long)i * g.ny + j) * g.nz + k;
}

// floor(n / f.d) for n < 2^31 (see FastDiv)
__device__ __forceinline__ int fdiv(long long n, const FastDiv &f)
{
    return int((static_cast<unsigned long long>(n) * f.m) >> (32 + f.s));
}

// Interior node (i, j, k) of flat interior index t (k fastest), ghosts offset.
__device__ __forceinline__ void interior_node(const DevGrid &g, long long t, int &i, int &j, int &k)
{
    const int ij = fdiv(t, g.d_nk);
    i = fdiv(t, g.d_njnk);
    k = g.bc + int(t - (long long)ij * g.nk);
    j = g.bc + (ij - i * g.nj);
    i += g.bc;
}

// Reciprocal of a nonzero, non-denormal double: the hardware approximation
// (rcp.approx.ftz.f64, about 20 bits) refined by one third-order step, y + y (e +
// e^2) with e = 1 - a y (the remainder is e^3 < 2^-59); relative error near one
// unit in the last place. One operation less than two Newton steps.
__device__ __forceinline__ double rcp_nr(double a)
{
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(a));
    const double e = fma(-a, y, 1.0);
    return fma(y, fma(e, e, e), y);
}

// x / sqrt(x d) for positive normal x d, the same way: rsqrt.approx.ftz.f64 and
// one third-order step, y + y e (1/2 + 3/8 e) with e = 1 - x d y^2. Without the
// special cases of rsqrt(); a negative or NaN argument gives NaN as there.
__device__ __forceinline__ double sound_speed(double x, double d)
{
    const double a = x * d;
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(a));
    const double e = fma(-(a * y), y, 1.0);
    return x * fma(y * e, fma(0.375, e, 0.5), y);
}
__device__ __forceinline__ float sound_speed(float x, float d) { return x * rsqrt(x * d); }

// min(max(x, 0), 1) on the words of x (one unsigned comparison tells whether x
// lies in [0, 1)): integer selects instead of FP64 comparisons. A NaN, whose
// sign the hardware leaves clear, gives 1.
__device__ __forceinline__ double saturate(double x)
{
    const int hi = __double2hiint(x), lo = __double2loint(x);
    const bool in = unsigned(hi) < 0x3ff00000u;
    return __hiloint2double(min(max(hi, 0), 0x3ff00000), in ? lo : 0);
}

// q = n / d without an IEEE division; for d == 0 (where the Newton steps give
// NaN) the product with the signed infinity is the quotient.
__device__ __forceinline__ double div_fast(double n, double d)
{
    const double y = rcp_nr(d);
    return n * (d == 0.0 ? copysign(INFINITY, d) : y);
}
__device__ __forceinline__ float div_fast(float n, float d) { return __fdividef(n, d); }

// exp(x) for |x| <= kExpMost: x = k ln 2 + r, |r| <= ln(2)/2, e^r = 1 + r + r^2 q(r)
// with q the degree-9 polynomial through (e^r - 1 - r) / r^2 at the ten Chebyshev
// nodes of that interval (relative error of e^r below 4e-17), scaled by 2^k. Within
// one unit in the last place; a NaN stays a NaN. Straight code (no special-case
// branches), so that a cell's twenty-odd exponentials interleave: whoever calls it
// keeps to the range (DevMech::t_lo, t_hi).
constexpr double kExpMost = 708.0;

__device__ __forceinline__ double exp_fast(double x)
{
    constexpr double kShift = 6755399441055744.0; // 1.5 * 2^52: rounds to an integer in the low word
    const double t = fma(x, 1.4426950408889634, kShift), kd = t - kShift;
    const int k = __double2loint(t);
    double r = fma(kd, -0x1.62e42fefa39efp-1, x);
    r = fma(kd, -0x1.abc9e3b39803fp-56, r);
    double q = 0x1.af38b4925be09p-26;
    q = fma(q, r, 0x1.28918e390a71ep-22);
    q = fma(q, r, 0x1.71de0da9d06acp-19);
    q = fma(q, r, 0x1.a019b905bafb1p-16);
    q = fma(q, r, 0x1.a01a01a7c54aep-13);
    q = fma(q, r, 0x1.6c16c1788dc33p-10);
    q = fma(q, r, 0x1.11111111109b2p-7);
    q = fma(q, r, 0x1.5555555553d5ep-5);
    q = fma(q, r, 0x1.5555555555556p-3);
    q = fma(q, r, 0.5);
    const double scale = __hiloint2double((k + 1023) << 20, 0);
    return fma(scale, fma(r * r, q, r), scale);
}

// exp_fast with its polynomial's terms paired (a third of the dependent operations).
__device__ __forceinline__ double exp_paired(double x)
{
    constexpr double kShift = 6755399441055744.0;
    const double t = fma(x, 1.4426950408889634, kShift), kd = t - kShift;
    const int k = __double2loint(t);
    double r = fma(kd, -0x1.62e42fefa39efp-1, x);
    r = fma(kd, -0x1.abc9e3b39803fp-56, r);
    const double r2 = r * r, r4 = r2 * r2;
    const double a = fma(0x1.5555555555556p-3, r, 0.5), b = fma(0x1.11111111109b2p-7, r, 0x1.5555555553d5ep-5),
                 c = fma(0x1.a01a01a7c54aep-13, r, 0x1.6c16c1788dc33p-10),
                 d = fma(0x1.71de0da9d06acp-19, r, 0x1.a019b905bafb1p-16),
                 e = fma(0x1.af38b4925be09p-26, r, 0x1.28918e390a71ep-22);
    const double q = fma(fma(e, r4, fma(d, r2, c)), r4, fma(b, r2, a));
    const double scale = __hiloint2double((k + 1023) << 20, 0);
    return fma(scale, fma(r2, q, r), scale);
}

// ------------------------------------------------------------------ thermo
// NASA 9-coefficient polynomials (src/Reaction.cpp:1165-1220). T powers are
// formed once per temperature.
struct TPow {
    double T, inv, inv2, t2, t3, t4, t5, lnT;
    bool low;
};

__device__ __forceinline__ TPow make_tpow(double T, bool need_log)
{
    TPow p;
    p.T = T;
    p.low = T < kThermoSwitch;
    p.inv = 1.0 / T;
    p.inv2 = p.inv * p.inv;
    p.t2 = T * T;
    p.t3 = p.t2 * T;
    p.t4 = p.t3 * T;
    p.t5 = p.t4 * T;
    p.lnT = need_log ? log(T) : 0.0;
    return p;
}

// Coefficient k of species s in the range of p. kRange 1 / 2: the low / high
// range fixed at compile time, so the value is an operand of the kernel's
// constant bank; 0: chosen per thread, a load whose address differs between
// threads (those loads throttle the memory pipe). by_range() picks the form.
template <int NS, int kRange = 0>
__device__ __forceinline__ double coeff(const DevMech &m, const TPow &p, int k, int s)
{
    if (kRange == 1)
        return m.clo[k][s];
    if (kRange == 2)
        return m.chi[k][s];
    return p.low ? m.clo[k][s] : m.chi[k][s];
}

// Runs f(std::integral_constant<int, R>) with R = 1 when every active thread of
// the warp is on the low NASA range, 2 when all are on the high one, 0
// otherwise. The range changes only at the 1000 K isotherm, so nearly every
// warp takes a fixed-range form; the arithmetic is the same in all three.
template <class F>
__device__ __forceinline__ void by_range(bool low, F &&f)
{
    const unsigned active = __activemask();
    if (__all_sync(active, low))
        f(std::integral_constant<int, 1>{});
    else if (__all_sync(active, !low))
        f(std::integral_constant<int, 2>{});
    else
        f(std::integral_constant<int, 0>{});
}

// Reaction::GetCpi: R*(a1 T^-2 + a2 T^-1 + a3 + a4 T + a5 T^2 + a6 T^3 + a7 T^4)
template <int NS, int kRange = 0>
__device__ __forceinline__ double cp_species(const DevMech &m, const TPow &p, double R, int s)
{
    const double a0 = coeff<NS, kRange>(m, p, 0, s), a1 = coeff<NS, kRange>(m, p, 1, s), a2 = coeff<NS, kRange>(m, p, 2, s),
                 a3 = coeff<NS, kRange>(m, p, 3, s), a4 = coeff<NS, kRange>(m, p, 4, s), a5 = coeff<NS, kRange>(m, p, 5, s),
                 a6 = coeff<NS, kRange>(m, p, 6, s);
    return R * (a0 * p.inv2 + a1 * p.inv + a2 + a3 * p.T + a4 * p.t2 + a5 * p.t3 + a6 * p.t4);
}

// Reaction::GetHi: R*(-a1/T + a2 lnT + a3 T + a4 T^2/2 + a5 T^3/3 + a6 T^4/4 + a7 T^5/5 + b1)
template <int NS, int kRange = 0>
__device__ __forceinline__ double h_species(const DevMech &m, const TPow &p, double R, int s)
{
    const double a0 = coeff<NS, kRange>(m, p, 0, s), a1 = coeff<NS, kRange>(m, p, 1, s), a2 = coeff<NS, kRange>(m, p, 2, s),
                 a3 = coeff<NS, kRange>(m, p, 3, s), a4 = coeff<NS, kRange>(m, p, 4, s), a5 = coeff<NS, kRange>(m, p, 5, s),
                 a6 = coeff<NS, kRange>(m, p, 6, s), a7 = coeff<NS, kRange>(m, p, 7, s);
#ifdef EU_EXACT_RATES
    return R * (-a0 * p.inv + a1 * p.lnT + a2 * p.T + a3 * p.t2 / 2 + a4 * p.t3 / 3 + a5 * p.t4 / 4 +
                a6 * p.t5 / 5 + a7);
#else
    return R * (-a0 * p.inv + a1 * p.lnT + a2 * p.T + a3 * p.t2 * 0.5 + a4 * p.t3 * (1.0 / 3.0) +
                a5 * p.t4 * 0.25 + a6 * p.t5 * 0.2 + a7);
#endif
}

// Reaction::GetSi: R*(-a1 T^-2/2 - a2/T + a3 lnT + a4 T + a5 T^2/2 + a6 T^3/3 + a7 T^4/4 + b2)
template <int NS, int kRange = 0>
__device__ __forceinline__ double s_species(const DevMech &m, const TPow &p, double R, int s)
{
    const double a0 = coeff<NS, kRange>(m, p, 0, s), a1 = coeff<NS, kRange>(m, p, 1, s), a2 = coeff<NS, kRange>(m, p, 2, s),
                 a3 = coeff<NS, kRange>(m, p, 3, s), a4 = coeff<NS, kRange>(m, p, 4, s), a5 = coeff<NS, kRange>(m, p, 5, s),
                 a6 = coeff<NS, kRange>(m, p, 6, s), a8 = coeff<NS, kRange>(m, p, 8, s);
#ifdef EU_EXACT_RATES
    return R * (-a0 * p.inv2 / 2 - a1 * p.inv + a2 * p.lnT + a3 * p.T + a4 * p.t2 / 2 + a5 * p.t3 / 3 +
                a6 * p.t4 / 4 + a8);
#else
    return R * (-a0 * p.inv2 * 0.5 - a1 * p.inv + a2 * p.lnT + a3 * p.T + a4 * p.t2 * 0.5 +
                a5 * p.t3 * (1.0 / 3.0) + a6 * p.t4 * 0.25 + a8);
#endif
}

#ifdef EU_EXACT_RATES
// G_s = H_s - S_s T of every species (src/Reaction.cpp:597-600), the
// reference's per-species expression.
template <int NS>
__device__ __forceinline__ void gibbs_all(const DevMech &m, const TPow &p, double T, double (&G)[NS])
{
    by_range(p.low, [&](auto range) {
        constexpr int kR = decltype(range)::value;
#pragma unroll
        for (int s = 0; s < NS; ++s) G[s] = h_species<NS, kR>(m, p, kRUniv, s) - s_species<NS, kR>(m, p, kRUniv, s) * T;
    });
}
#else
// The nine functions of T whose sums with a species' coefficients give G_s/(R T):
// the enthalpy's term over R T minus the entropy's over R, coefficient by
// coefficient (src/Reaction.cpp:597-600, 1180-1220).
__device__ __forceinline__ void gibbs_terms(double T, double inv, double lnT, double (&f)[9])
{
    const double t2 = T * T;
    f[0] = -0.5 * (inv * inv);
    f[1] = (lnT + 1.0) * inv;
    f[2] = 1.0 - lnT;
    f[3] = -0.5 * T;
    f[4] = t2 * (-1.0 / 6.0);
    f[5] = (t2 * T) * (-1.0 / 12.0);
    f[6] = (t2 * t2) * (-1.0 / 20.0);
    f[7] = inv;
    f[8] = -1.0;
}

// g_s = G_s/(R T) of every species: nine multiply-adds each.
template <int NS>
__device__ __forceinline__ void gibbs_rt(const DevMech &m, double T, double inv, double lnT, double (&g)[NS])
{
    double f[9];
    gibbs_terms(T, inv, lnT, f);
    by_range(T < kThermoSwitch, [&](auto range) {
        constexpr int kR = decltype(range)::value;
        TPow p;
        p.low = T < kThermoSwitch;
#pragma unroll
        for (int s = 0; s < NS; ++s) {
            double v = f[0] * coeff<NS, kR>(m, p, 0, s);
#pragma unroll
            for (int k = 1; k < 9; ++k) v = fma(f[k], coeff<NS, kR>(m, p, k, s), v);
            g[s] = v;
        }
    });
}
#endif

// --------------------------------------------------------- state recovery

// Flowfield::Get_temp (src/Flowfield.cpp:2072-2131): Newton on
// sum_s Y_s h_s(T) - E*1e-3 - (sum_s Y_s R_s) T = 0, at most 10 iterations,
// stop when |dT| < 1e-6 K. E is the cell's previous internal energy.
#ifdef EU_EXACT_THERMO
template <int NS>
__device__ __forceinline__ double newton_temperature(const DevMech &m, double T, double E, const double (&Y)[NS])
{
    double rsum = 0;
#pragma unroll
    for (int s = 0; s < NS; ++s) rsum += Y[s] * m.ri[s];
    const double e_scaled = E * 1e-3;
    double T_temp = T;
    for (int count = 0; count < 10; ++count) {
        const double T0 = T_temp;
        const TPow p = make_tpow(T0, true);
        double hsum = 0, cpsum = 0;
        by_range(p.low, [&](auto range) {
            constexpr int kR = decltype(range)::value;
#pragma unroll
            for (int s = 0; s < NS; ++s) hsum += Y[s] * h_species<NS, kR>(m, p, m.ri[s], s);
#pragma unroll
            for (int s = 0; s < NS; ++s) cpsum += Y[s] * cp_species<NS, kR>(m, p, m.ri[s], s);
        });
        const double temp1 = (hsum - e_scaled) - rsum * T0;
        const double temp2 = cpsum - rsum;
        T_temp = T0 - temp1 / temp2;
        if (fabs(T_temp - T0) < 1e-6)
            break;
    }
    return T_temp;
}

// The exact forms keep no thermo sums between recovery and the primitives.
template <int NS>
struct ThermoCache {
};
#else
// Mixture polynomial of one NASA range: c_k = sum_s Y_s R_s a_k,s, with the
// enthalpy's divisors folded in (h/R uses a_k T^(k-1)/(k-1) for k >= 3).
template <int NS>
struct MixPoly {
    double a0, a1, a2, a3, a4, a5, a6, a7; // cp form: a0/T^2 + a1/T + a2 + a3 T + ... + a6 T^4
    double h3, h4, h5, h6;                 // a3/2, a4/3, a5/4, a6/5
};

// The coefficients of one range, read from the kernel's constant parameter:
// with the range fixed at compile time every coefficient is an operand of the
// constant bank; with a per-thread choice each is a load whose address differs
// between threads. The range is the same across a warp almost everywhere (it
// changes only at the 1000 K isotherm), so the warp takes a fixed-range form
// whenever all its active threads agree; the sums are the same either way.
template <int NS, int kRange>
__device__ __forceinline__ void mix_sums(const DevMech &m, const double (&Y)[NS], bool low, double (&a)[8])
{
#pragma unroll
    for (int s = 0; s < NS; ++s) {
        const double w = Y[s] * m.ri[s];
#pragma unroll
        for (int q = 0; q < 8; ++q)
            a[q] = fma(w, kRange == 1 ? m.clo[q][s] : (kRange == 2 ? m.chi[q][s] : (low ? m.clo[q][s] : m.chi[q][s])),
                       a[q]);
    }
}

template <int NS>
__device__ __forceinline__ void mix_poly(const DevMech &m, const double (&Y)[NS], bool low, MixPoly<NS> &c)
{
    double a[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    const unsigned active = __activemask();
    if (__all_sync(active, low))
        mix_sums<NS, 1>(m, Y, low, a);
    else if (__all_sync(active, !low))
        mix_sums<NS, 2>(m, Y, low, a);
    else
        mix_sums<NS, 0>(m, Y, low, a);
    c.a0 = a[0];
    c.a1 = a[1];
    c.a2 = a[2];
    c.a3 = a[3];
    c.a4 = a[4];
    c.a5 = a[5];
    c.a6 = a[6];
    c.a7 = a[7];
    c.h3 = a[3] * 0.5;
    c.h4 = a[4] * (1.0 / 3.0);
    c.h5 = a[5] * 0.25;
    c.h6 = a[6] * 0.2;
}

// The mixture polynomial of the Newton's last iterate and its range: the
// primitives that follow the recovery (cp for Gamma) reuse it when the final
// temperature lies in the same range (the same sums, so the same values).
template <int NS>
struct ThermoCache {
    MixPoly<NS> c;
    int low = -1; // 1: low range, 0: high, -1: no sums
};

template <int NS>
__device__ __forceinline__ double newton_temperature(const DevMech &m, double T, double E, const double (&Y)[NS],
                                                     ThermoCache<NS> &tc)
{
    double rsum = 0;
#pragma unroll
    for (int s = 0; s < NS; ++s) rsum += Y[s] * m.ri[s];
    const double e_scaled = E * 1e-3;
    bool low = T < kThermoSwitch;
    MixPoly<NS> &c = tc.c;
    mix_poly<NS>(m, Y, low, c);
    double T_temp = T;
    for (int count = 0; count < 10; ++count) {
        const double T0 = T_temp;
        const bool l = T0 < kThermoSwitch;
        if (l != low) {
            low = l;
            mix_poly<NS>(m, Y, low, c);
        }
        const double inv = rcp_nr(T0);
        const double h = fma(T0, fma(T0, fma(T0, fma(T0, fma(T0, c.h6, c.h5), c.h4), c.h3), c.a2), c.a7) -
                         c.a0 * inv + c.a1 * log(T0);
        const double cp = fma(T0, fma(T0, fma(T0, fma(T0, c.a6, c.a5), c.a4), c.a3), c.a2) +
                          inv * fma(c.a0, inv, c.a1);
        const double temp1 = (h - e_scaled) - rsum * T0;
        const double temp2 = cp - rsum;
        T_temp = T0 - div_fast(temp1, temp2);
        if (fabs(T_temp - T0) < 1e-6)
            break;
    }
    tc.low = low;
    return T_temp;
}

template <int NS>
__device__ __forceinline__ double newton_temperature(const DevMech &m, double T, double E, const double (&Y)[NS])
{
    ThermoCache<NS> tc;
    return newton_temperature<NS>(m, T, E, Y, tc);
}

// log(1 + x) for |x| <= 2^-6 by its series to x^9 (truncation below 2^-57 |x|):
// the change of log T between Newton iterates without a logarithm.
__device__ __forceinline__ double log1p_small(double x)
{
    double s = 1.0 / 9.0;
    s = fma(s, x, -1.0 / 8.0);
    s = fma(s, x, 1.0 / 7.0);
    s = fma(s, x, -1.0 / 6.0);
    s = fma(s, x, 1.0 / 5.0);
    s = fma(s, x, -1.0 / 4.0);
    s = fma(s, x, 1.0 / 3.0);
    s = fma(s, x, -1.0 / 2.0);
    s = fma(s, x, 1.0);
    return s * x;
}

// log T1 from log T0 and x = (T1 - T0) / T0.
__device__ __forceinline__ double advance_log(double ln0, double x, double T1)
{
    return fabs(x) <= 0x1p-6 ? ln0 + log1p_small(x) : log(T1);
}

// The Newton above for the kinetics, whose substeps' rates and rebuilds each
// start from the last rebuild's temperature: inv and lnT are 1/T and log T of
// the starting temperature on entry and of the result on return, and each
// iterate's log comes from the previous one's (advance_log), so that a cell's
// substeps take one logarithm.
template <int NS>
__device__ __forceinline__ double newton_temperature_carry(const DevMech &m, double T, double E, const double (&Y)[NS],
                                                           ThermoCache<NS> &tc, double &inv, double &lnT)
{
    double rsum = 0;
#pragma unroll
    for (int s = 0; s < NS; ++s) rsum += Y[s] * m.ri[s];
    const double e_scaled = E * 1e-3;
    bool low = T < kThermoSwitch;
    MixPoly<NS> &c = tc.c;
    mix_poly<NS>(m, Y, low, c);
    double T0 = T, inv0 = inv, ln0 = lnT, T_temp = T;
    for (int count = 0; count < 10; ++count) {
        if (count > 0) {
            const double x = (T_temp - T0) * inv0;
            ln0 = advance_log(ln0, x, T_temp);
            T0 = T_temp;
            inv0 = rcp_nr(T0);
        }
        const bool l = T0 < kThermoSwitch;
        if (l != low) {
            low = l;
            mix_poly<NS>(m, Y, low, c);
        }
        const double h = fma(T0, fma(T0, fma(T0, fma(T0, fma(T0, c.h6, c.h5), c.h4), c.h3), c.a2), c.a7) -
                         c.a0 * inv0 + c.a1 * ln0;
        const double cp = fma(T0, fma(T0, fma(T0, fma(T0, c.a6, c.a5), c.a4), c.a3), c.a2) +
                          inv0 * fma(c.a0, inv0, c.a1);
        const double temp1 = (h - e_scaled) - rsum * T0;
        const double temp2 = cp - rsum;
        T_temp = T0 - div_fast(temp1, temp2);
        if (fabs(T_temp - T0) < 1e-6)
            break;
    }
    tc.low = low;
    lnT = advance_log(ln0, (T_temp - T0) * inv0, T_temp);
    inv = rcp_nr(T_temp);
    return T_temp;
}
#endif

// Per-cell flow state kept in registers by the recovery / kinetics kernel.
template <int NS>
struct CellState {
    double cs[NS + 4];
    double Y[NS];
    double D, T, E, U, V, W;
    double inv, lnT; // 1/T and log T (fast forms; carried by the temperature Newton)
};

// 1/T and log T of a temperature just loaded.
template <int NS>
__device__ __forceinline__ void load_temperature(CellState<NS> &c, double T)
{
    c.T = T;
#ifndef EU_EXACT_RATES
    c.inv = rcp_nr(T);
    c.lnT = log(T);
#endif
}

// Flowfield::Update_after_CS (src/Flowfield.cpp:1579-1617 / :1639-1673) for one
// cell, up to the point where P, H, Gamma are needed (those are formed by
// finish_primitives when the cell's primitives are written). kCarry: within the
// kinetics, whose rates read c.inv and c.lnT (newton_temperature_carry).
template <int NS, bool kCarry = false>
__device__ __forceinline__ void recover_state(const DevMech &m, CellState<NS> &c, ThermoCache<NS> &tcache)
{
    double D = 0;
#pragma unroll
    for (int s = 0; s < NS; ++s) D += c.cs[s];
#ifdef EU_EXACT_THERMO
#pragma unroll
    for (int s = 0; s < NS; ++s) c.Y[s] = c.cs[s] / D;
    c.D = D;
    c.T = newton_temperature<NS>(m, c.T, c.E, c.Y);
    if (kCarry)
        load_temperature<NS>(c, c.T);
    c.U = c.cs[NS + 0] / D;
    c.V = c.cs[NS + 1] / D;
    c.W = c.cs[NS + 2] / D;
    c.E = (c.cs[NS + 3] - 0.5 * D * (c.U * c.U + c.V * c.V + c.W * c.W)) / D;
#else
    // one refined reciprocal of the density instead of NS + 4 divisions
    const double invD = rcp_nr(D);
#pragma unroll
    for (int s = 0; s < NS; ++s) c.Y[s] = c.cs[s] * invD;
    c.D = D;
    if (kCarry)
        c.T = newton_temperature_carry<NS>(m, c.T, c.E, c.Y, tcache, c.inv, c.lnT);
    else
        c.T = newton_temperature<NS>(m, c.T, c.E, c.Y, tcache);
    c.U = c.cs[NS + 0] * invD;
    c.V = c.cs[NS + 1] * invD;
    c.W = c.cs[NS + 2] * invD;
    c.E = (c.cs[NS + 3] - 0.5 * D * (c.U * c.U + c.V * c.V + c.W * c.W)) * invD;
#endif
}

// P, H, Gamma of Update_after_CS (src/Flowfield.cpp:1606-1614). tcache: the
// recovery's thermo sums for this state, or null.
template <int NS>
__device__ __forceinline__ void finish_primitives(const DevMech &m, const CellState<NS> &c,
                                                  const ThermoCache<NS> *tcache, double &P, double &H, double &G)
{
#ifdef EU_EXACT_THERMO
    double inv_w = 0;
#pragma unroll
    for (int s = 0; s < NS; ++s) inv_w += c.Y[s] / m.mw[s];
    const double Wav = 1.0 / inv_w;
    const double Rgas = kRUniv * 1000 / Wav;
    P = c.T * c.D * Rgas;
    H = P / c.D + c.E;
    const TPow p = make_tpow(c.T, false);
    double cp = 0;
    by_range(p.low, [&](auto range) {
        constexpr int kR = decltype(range)::value;
#pragma unroll
        for (int s = 0; s < NS; ++s) cp += cp_species<NS, kR>(m, p, m.ri[s], s) * c.Y[s];
    });
    const double Cp = cp * 1000;
    G = Cp / (Cp - kRUniv * inv_w * 1000);
#else
    // R_mix = 1000 sum_s Y_s R_s (R_s = R/W_s), so p/rho = T R_mix: no divisions
    double rg = 0;
#pragma unroll
    for (int s = 0; s < NS; ++s) rg = fma(c.Y[s], m.ri[s], rg);
    const double Rgas = rg * 1000;
    P = c.T * c.D * Rgas;
    H = c.T * Rgas + c.E;
    MixPoly<NS> mp;
    const bool low = c.T < kThermoSwitch;
    if (tcache && tcache->low == int(low))
        mp = tcache->c;
    else
        mix_poly<NS>(m, c.Y, low, mp);
    const double T0 = c.T, inv = rcp_nr(T0);
    const double cp = fma(T0, fma(T0, fma(T0, fma(T0, mp.a6, mp.a5), mp.a4), mp.a3), mp.a2) +
                      inv * fma(mp.a0, inv, mp.a1);
    const double Cp = cp * 1000;
    G = div_fast(Cp, Cp - Rgas);
#endif
}

template <int NS>
__device__ __forceinline__ void finish_primitives(const DevMech &m, const CellState<NS> &c, double &P, double &H,
                                                  double &G)
{
    finish_primitives<NS>(m, c, static_cast<const ThermoCache<NS> *>(nullptr), P, H, G);
}

// ------------------------------------------------------------- kinetics

// pow(x, nu) for the reference's stoichiometric exponents (0, 1, 2 are exact).
__device__ __forceinline__ double pow_nu(double x, double nu, bool nu_int)
{
    if (nu_int)
        return nu == 0.0 ? 1.0 : (nu == 1.0 ? x : x * x);
    return pow(x, nu);
}

__device__ __forceinline__ double pow_int_or_real(double x, double e)
{
    if (e == 0.0)
        return 1.0;
    if (e == 1.0)
        return x;
    if (e == -1.0)
        return 1.0 / x;
    return pow(x, e);
}

// Per-species production/loss sums of one cell, accumulated reaction by
// reaction (src/Reaction.cpp:597-623 rates, :720-727 mass rates Wi, :786-797
// trapezoid P and Q). Summation order over reactions is the reference's for
// every species; terms whose stoichiometric coefficients vanish are exact zeros
// in the reference and are skipped here. P and Q do not depend on the substep
// length, so the prediction's evaluation serves the first substep too.
// Per reaction W's term is Q's minus P's, and the fast forms take W from the
// sums: W_s = mw_s (Q_s - P_s), a third of the sums less to keep.
template <int NS>
struct SpeciesRates {
    double P[NS], Q[NS];
#ifdef EU_EXACT_RATES
    double W[NS]; // Wi (mass rate, g/cm^3/s)
    __device__ __forceinline__ double w(const DevMech &, int s) const { return W[s]; }
#else
    __device__ __forceinline__ double w(const DevMech &m, int s) const { return m.mw[s] * (Q[s] - P[s]); }
#endif
};

#ifdef EU_EXACT_RATES
// Strict form: the reference's expressions (pow, exp of each Kp, divisions).
template <int NS, int NR>
__device__ __forceinline__ void eval_rates(const DevMech &m, double T, double, double, const double (&mc)[NS],
                                           SpeciesRates<NS> &k)
{
    double Gi[NS];
    {
        const TPow p = make_tpow(T, true);
        gibbs_all<NS>(m, p, T, Gi);
    }
    const bool nu_int = m.nu_int != 0;
    const double RT = kRUniv * T;
    const double RuT = kRuCal * T;
    const double p0 = kP0 * 1e-6;
#pragma unroll
    for (int s = 0; s < NS; ++s) {
        k.P[s] = 0.0;
        k.Q[s] = 0.0;
        k.W[s] = 0.0;
    }
#pragma unroll
    for (int r = 0; r < NR; ++r) {
        double delta_g = 0.0, rrf = 1.0, rrb = 1.0, rtb = 0.0;
        const double kf =
            m.af[r] * pow_int_or_real(T, m.bf[r]) * (m.eaf[r] == 0.0 ? 1.0 : exp(-m.eaf[r] / RuT));
#pragma unroll
        for (int s = 0; s < NS; ++s) {
            const double f = m.sf[r][s], b = m.sb[r][s];
            delta_g += (b - f) * Gi[s];
            rrf *= pow_nu(mc[s], f, nu_int);
            rrb *= pow_nu(mc[s], b, nu_int);
            rtb += mc[s] * m.tb[r][s];
        }
        const double Xr = m.xr[r];
        const double Kp = exp(-delta_g / RT) * pow_int_or_real(p0, Xr);
        const double Kc = Kp * pow_int_or_real(RT, -Xr);
        const double kb = kf / Kc;
        if (rtb == 0.0)
            rtb = 1.0;
        const double fwd = kf * rrf, bwd = kb * rrb;
        const double rr = fwd - bwd;
#pragma unroll
        for (int s = 0; s < NS; ++s) {
            const double b = m.sb[r][s], f = m.sf[r][s];
            if (b != 0.0 || f != 0.0) {
                k.W[s] += (b - f) * rtb * rr;
                k.Q[s] += (b * fwd + f * bwd) * rtb;
                k.P[s] += (b * bwd + f * fwd) * rtb;
            }
        }
    }
#pragma unroll
    for (int s = 0; s < NS; ++s) k.W[s] = m.mw[s] * k.W[s];
}
#else
// x^n for a whole n; ix = 1/x.
__device__ __forceinline__ double pow_whole(double x, double ix, double n)
{
    double r = 1.0;
#pragma unroll 1
    for (int q = int(fabs(n)); q > 0; --q) r *= n > 0.0 ? x : ix;
    return r;
}

// The rates outside [t_lo, t_hi] (very cold gas: of H2_JA919's factors the square
// of atomic hydrogen's exp(G/RT) is the first to leave the range, at 85 K), where
// the products of the form below would meet an underflowed factor with an
// overflowed one: one exponential of each reaction's
// whole exponent, forward and backward, by exp. Rare, so out of line and rolled.
template <int NS, int NR>
__device__ __noinline__ void eval_rates_far(const DevMech &m, double T, double inv, double lnT, const double *mc,
                                            double *Q, double *P)
{
    double g[NS], f[9];
    gibbs_terms(T, inv, lnT, f);
    const bool low = T < kThermoSwitch;
#pragma unroll 1
    for (int s = 0; s < NS; ++s) {
        double v = 0.0;
#pragma unroll
        for (int k = 0; k < 9; ++k) v = fma(f[k], low ? m.clo[k][s] : m.chi[k][s], v);
        g[s] = v;
        P[s] = Q[s] = 0.0;
    }
    const double rt_p0 = T * (kRUniv / (kP0 * 1e-6)), p0_rt = inv * (kP0 * 1e-6 / kRUniv);
#pragma unroll 1
    for (int r = 0; r < NR; ++r) {
        double rrf = 1.0, rrb = 1.0, rtb = 0.0, dg = 0.0;
#pragma unroll 1
        for (int s = 0; s < NS; ++s) {
            const double nf = m.sf[r][s], nb = m.sb[r][s], c = mc[s];
            rrf *= nf == 0.0 ? 1.0 : nf == 1.0 ? c : c * c;
            rrb *= nb == 0.0 ? 1.0 : nb == 1.0 ? c : c * c;
            dg = fma(nb - nf, g[s], dg);
            rtb += c * m.tb[r][s];
        }
        if (rtb == 0.0)
            rtb = 1.0;
        const double e = m.bf[r] * lnT - m.eaf[r] * (inv * (1.0 / kRuCal));
        const double fr = m.af[r] * exp(e) * rrf * rtb;
        const double br = m.af[r] * exp(e + dg) * pow_whole(rt_p0, p0_rt, m.xr[r]) * rrb * rtb;
#pragma unroll 1
        for (int s = 0; s < NS; ++s) {
            const double nf = m.sf[r][s], nb = m.sb[r][s];
            if (nf != 0.0 || nb != 0.0) {
                Q[s] += nb * fr + nf * br;
                P[s] += nb * br + nf * fr;
            }
        }
    }
}

// Whether the rates at T were formed by eval_rates_far.
template <int NS, int NR>
__device__ __forceinline__ bool rates_far(const DevMech &m, double T, double inv, double lnT, const double (&mc)[NS],
                                          SpeciesRates<NS> &k)
{
    if (T >= m.t_lo && T <= m.t_hi)
        return false;
    double c[NS], Q[NS], P[NS]; // the call's own copies: the caller's arrays stay in registers
#pragma unroll
    for (int s = 0; s < NS; ++s) c[s] = mc[s];
    eval_rates_far<NS, NR>(m, T, inv, lnT, c, Q, P);
#pragma unroll
    for (int s = 0; s < NS; ++s) {
        k.Q[s] = Q[s];
        k.P[s] = P[s];
    }
    return true;
}

// Fast form, algebraically the reference's:
//   Kc_r = exp(-sum_s nu_rs g_s) (p0/RT)^Xr with g_s = G_s/(R T) per species, so
//   kb_r = kf_r * prod_s exp(g_s)^nu_rs * (RT/p0)^Xr  (one exp per species);
//   kf_r = A_r exp(b_r ln T - E_r/(Ru T))            (one exp per reaction).
template <int NS, int NR>
__device__ __forceinline__ void eval_rates(const DevMech &m, double T, double inv, double lnT, const double (&mc)[NS],
                                           SpeciesRates<NS> &k)
{
    if (rates_far<NS, NR>(m, T, inv, lnT, mc, k))
        return;
    double eg[NS], ieg[NS];
    gibbs_rt<NS>(m, T, inv, lnT, eg);
#pragma unroll
    for (int s = 0; s < NS; ++s) {
        eg[s] = exp_fast(eg[s]);
        ieg[s] = rcp_nr(eg[s]);
    }
    const double inv2 = inv * inv;
    const double invRuT = inv * (1.0 / kRuCal);
    const double rt_p0 = T * (kRUniv / (kP0 * 1e-6));
    const double p0_rt = inv * (kP0 * 1e-6 / kRUniv);
#pragma unroll
    for (int s = 0; s < NS; ++s) {
        k.P[s] = 0.0;
        k.Q[s] = 0.0;
    }
#pragma unroll
    for (int r = 0; r < NR; ++r) {
        double rrf = 1.0, rrb = 1.0, rtb = 0.0, kc_inv = 1.0;
        const double b = m.bf[r];
        double kf;
        if (m.eaf[r] == 0.0 && (b == 0.0 || b == 1.0 || b == -1.0 || b == -2.0))
            kf = m.af[r] * (b == 0.0 ? 1.0 : b == 1.0 ? T : b == -1.0 ? inv : inv2);
        else
            kf = m.af[r] * exp_fast(b * lnT - m.eaf[r] * invRuT);
#pragma unroll
        for (int s = 0; s < NS; ++s) {
            const double f = m.sf[r][s], bb = m.sb[r][s];
            rrf *= (f == 0.0 ? 1.0 : (f == 1.0 ? mc[s] : mc[s] * mc[s]));
            rrb *= (bb == 0.0 ? 1.0 : (bb == 1.0 ? mc[s] : mc[s] * mc[s]));
            const double d = bb - f;
            kc_inv *= (d == 0.0 ? 1.0 : d == 1.0 ? eg[s] : d == -1.0 ? ieg[s] : d == 2.0 ? eg[s] * eg[s]
                                                                                  : ieg[s] * ieg[s]);
            rtb += mc[s] * m.tb[r][s];
        }
        const double Xr = m.xr[r];
        kc_inv *= (Xr == 0.0 ? 1.0 : Xr == 1.0 ? rt_p0 : Xr == -1.0 ? p0_rt : pow_whole(rt_p0, p0_rt, Xr));
        const double kb = kf * kc_inv;
        if (rtb == 0.0)
            rtb = 1.0;
        const double fwd = kf * rrf, bwd = kb * rrb;
#pragma unroll
        for (int s = 0; s < NS; ++s) {
            const double bb = m.sb[r][s], f = m.sf[r][s];
            if (bb != 0.0 || f != 0.0) {
                k.Q[s] += (bb * fwd + f * bwd) * rtb;
                k.P[s] += (bb * bwd + f * fwd) * rtb;
            }
        }
    }
}

// P_s / mc_s, the trapezoid's loss frequency (0 where the species is absent,
// src/Reaction.cpp:786-797), with a refined reciprocal. Traces below 1e-200,
// whose reciprocal would leave the normal range, are scaled first.
__device__ __forceinline__ double loss_frequency(double P, double mc)
{
    const double s = fabs(mc) < 1e-200 ? 0x1p+300 : 1.0;
    const double q = (P * s) * rcp_nr(mc * s);
    return mc == 0.0 ? 0.0 : q;
}
#endif

// One linearised trapezoid substep (src/Reaction.cpp:786-805) followed by
// Flowfield::Explicit(step,i,j,k) (src/Flowfield.cpp:1521-1536) and the state
// recovery. mc holds the scaled concentrations the rates used; the scaled
// densities are cs * 1e-3.
template <int NS>
__device__ __forceinline__ void trapezoid_substep(const DevMech &m, const SpeciesRates<NS> &k, double dts,
                                                  const double (&mc)[NS], CellState<NS> &c, ThermoCache<NS> &tcache)
{
#ifdef EU_EXACT_RATES
    const double half = dts / 2.0;
#else
    const double half = dts * 0.5;
#endif
    double D = 0.0;
#pragma unroll
    for (int s = 0; s < NS; ++s) {
        const double di = c.cs[s] * 1e-3;
        const double q = m.mw[s] * k.Q[s];
#ifdef EU_EXACT_RATES
        // the quotient formed before the choice: a select, not a branch on
        // which the threads (cells with and without the species) diverge
        const double pq = k.P[s] / mc[s];
        const double p = (mc[s] == 0) ? 0.0 : pq;
        const double nd = ((1.0 - half * p) * di + dts * q) / (1.0 + half * p) * 1e3;
#else
        const double hp = half * loss_frequency(k.P[s], mc[s]);
        const double nd = fma(dts, q, fma(-hp, di, di)) * rcp_nr(1.0 + hp) * 1e3;
#endif
        c.cs[s] = nd;
        D += nd;
    }
    c.cs[NS + 0] = c.U * D;
    c.cs[NS + 1] = c.V * D;
    c.cs[NS + 2] = c.W * D;
    c.cs[NS + 3] = D * c.E + 0.5 * (c.U * c.U + c.V * c.V + c.W * c.W) * D;
    recover_state<NS, true>(m, c, tcache);
}

// Concentrations scaled to mol/cm^3 as the kinetics reads them: Mc = Di/Mw*1000
// (src/Flowfield.cpp:1589) times 1e-6 (src/Reaction.cpp:580).
template <int NS>
__device__ __forceinline__ void scaled_concentrations(const DevMech &m, const CellState<NS> &c, double (&mc)[NS])
{
#pragma unroll
    for (int s = 0; s < NS; ++s) mc[s] = (c.cs[s] / m.mw[s] * 1000) * 1e-6;
}

// ----------------------------------------------------------------- fluxes

// Minmod (include/Differ.hpp:33-43) as selects.
template <typename R>
__device__ __forceinline__ R minmod(R r)
{
    return r > R(0) ? ((R(1) < r) ? R(1) : r) : R(0);
}

// MUSCL_2, kappa = 1/3, minmod (include/Differ.hpp:149-238) for the face
// between m and m+1: fm1, f0, f1, f2 are values at m-1, m, m+1, m+2.
//
// Strict form: the reference's expression, with its divisions
//   L = A1/(A0+1e-12), R = A1/(A2+1e-12), limiter values minmod(L), minmod(1/L).
// Fast form: the same limiter written without the reciprocal ratios. For
// L > 0 the reference's slope term 0.25((1-k) min(L,1) + (1+k) min(1/L,1) L) A0
// equals 0.5 min(L,1) A0 (k = 1/3); for L <= 0 it is 0: 0.5 A0 times L
// saturated to [0, 1], L formed with a refined reciprocal. Results agree to a
// few units in the last place (A0 = -1e-12 exactly, where L has no value, takes
// the slope 0.5 A0).
// The 1e-12 guard is kept in every form: it flattens the slopes of fields
// whose differences are below it (trace species), so the first-order value
// the reference takes there is kept.

// Slope term t of one side: the left state is f0 + t(A0, A1), the right state
// f1 - t(A2, A1).
template <typename R, bool kStrict>
__device__ __forceinline__ R muscl_slope(R a, R A1)
{
    if (kStrict) {
        const R kk = R(1.0) / R(3.0);
        const R L = A1 / (a + R(1e-12));
        const R L1 = minmod(L), L2 = minmod(R(1.0) / L);
        return R(0.25) * ((R(1.0) - kk) * L1 + (R(1) + kk) * L2 * L) * a;
    } else if constexpr (std::is_same<R, float>::value) {
        // min(max(L, 0), 1) is the saturation of the product that forms L
        // (NaN saturates to 0, as L > 0 fails for it)
        const R L = __saturatef(div_fast(A1, a + R(1e-12)));
        return R(0.5) * a * L;
    } else {
        return R(0.5) * a * saturate(A1 * rcp_nr(a + R(1e-12)));
    }
}

template <typename R, bool kStrict>
__device__ __forceinline__ void muscl(R fm1, R f0, R f1, R f2, R &left, R &right)
{
    const R A0 = f0 - fm1;
    const R A1 = f1 - f0;
    const R A2 = f2 - f1;
    left = f0 + muscl_slope<R, kStrict>(A0, A1);
    right = f1 - muscl_slope<R, kStrict>(A2, A1);
}

// Only the upwind side of a face, from the three points it reads: u and w on
// the upwind side (u next to the face), v across it, e = +1e-12 when the left
// side is upwind, else -1e-12. The right side's value f1 - t(f2 - f1, f1 - f0)
// is u + t with every operand of the slope negated, and round-to-nearest is
// symmetric, so in the strict form the value is bitwise the reference's (a zero
// denominator takes the sign it has there).
template <typename R, bool kStrict>
__device__ __forceinline__ R muscl_upwind(R u, R w, R v, R e)
{
    const R a = u - w, A1 = v - u;
    if constexpr (kStrict) {
        R d = a + e;
        d = d == R(0) ? copysign(R(0), e) : d;
        const R kk = R(1.0) / R(3.0);
        const R L = A1 / d;
        const R L1 = minmod(L), L2 = minmod(R(1.0) / L);
        return u + R(0.25) * ((R(1.0) - kk) * L1 + (R(1) + kk) * L2 * L) * a;
    } else if constexpr (std::is_same<R, float>::value) {
        return fmaf(R(0.5) * a, __saturatef(div_fast(A1, a + e)), u);
    } else {
        return fma(R(0.5) * a, saturate(A1 * rcp_nr(a + e)), u);
    }
}

// The part of a face's AUSM+ flux that needs both reconstructed sides
// (src/Flowfield.cpp:1794-1870): sound speeds, split Mach numbers and pressures
// from p, rho, gamma and the normal velocity.
template <typename R>
struct FaceState {
    R PL, PR, DL, DR, UnL, UnR, G1, G2, VI;
};

template <typename R, bool kStrict>
__device__ __forceinline__ void face_split(FaceState<R> &w, R GaL, R GaR)
{
    R CI, MaL, MaR;
    if (kStrict) {
        const R CL = sqrt(GaL * w.PL / w.DL);
        const R CR = sqrt(GaR * w.PR / w.DR);
        CI = R(0.5) * (CL + CR);
        MaL = w.UnL / CI;
        MaR = w.UnR / CI;
    } else {
        // c = sqrt(g p / rho) = (g p) / sqrt(g p rho)
        const R gpL = GaL * w.PL, gpR = GaR * w.PR;
        const R CL = sound_speed(gpL, w.DL);
        const R CR = sound_speed(gpR, w.DR);
        CI = R(0.5) * (CL + CR);
        const R inv = div_fast(R(1), CI);
        MaL = w.UnL * inv;
        MaR = w.UnR * inv;
    }
    // Split Mach and pressure functions: both regimes formed, then selected
    // (a branch per regime would split a warp whose faces straddle Mach 1)
    R B1, B2;
    {
        const R a = MaL + R(1.0), t = MaL * MaL - R(1.0);
        const R Bs = R(0.25) * (a * a) + R(0.125) * (t * t);
        const R Gs = R(0.25) * (a * a) * (R(2.0) - MaL) + R(3.0) / R(16.0) * MaL * (t * t);
        const R Bp = R(0.5) * (MaL + fabs(MaL));
        // Bp / MaL is exactly 1 (MaL >= 1) or 0 (MaL <= -1)
        const R Gp = kStrict ? Bp / MaL : (MaL > R(0) ? R(1) : R(0));
        const bool sub = fabs(MaL) < R(1.0);
        B1 = sub ? Bs : Bp;
        w.G1 = sub ? Gs : Gp;
    }
    {
        const R a = MaR - R(1.0), t = MaR * MaR - R(1.0);
        const R Bs = -R(0.25) * (a * a) - R(0.125) * (t * t);
        const R Gs = R(0.25) * (a * a) * (R(2.0) + MaR) - R(3.0) / R(16.0) * MaR * (t * t);
        const R Bp = R(0.5) * (MaR - fabs(MaR));
        const R Gp = kStrict ? Bp / MaR : (MaR < R(0) ? R(1) : R(0));
        const bool sub = fabs(MaR) < R(1.0);
        B2 = sub ? Bs : Bp;
        w.G2 = sub ? Gs : Gp;
    }
    w.VI = (B1 + B2) * CI;
}

// MUSCL reconstruction and AUSM+ flux of one face (src/Flowfield.cpp:1794-1930)
// for direction DIR (0: x, 1: y, 2: z). get(f, p) returns stencil point p
// (0..3: cells m-1, m, m+1, m+2 across the face m+1/2) of primitive f; upwind(f,
// up, u, w, v) the three points of muscl_upwind.
//
// AUSM+ reads both reconstructed sides only of p, rho, gamma and the normal
// velocity (sound speeds, Mach numbers, pressure split). Every other flux
// term takes the upwind side (VI >= 0: left, src/Flowfield.cpp:1870): the two
// tangential velocities, H and the species. Those twelve quantities are
// reconstructed on the upwind side alone, with the same expression, so the
// flux is the same as with both sides formed.
template <int NS, int DIR, typename R, class Get, class Upwind>
__device__ __forceinline__ void face_ausm(Get get, Upwind upwind, R (&F)[NS + 4])
{
    constexpr int kN = kU + DIR;
    FaceState<R> w;
    R GaL, GaR;
    muscl<R, false>(get(kP, 0), get(kP, 1), get(kP, 2), get(kP, 3), w.PL, w.PR);
    muscl<R, false>(get(kD, 0), get(kD, 1), get(kD, 2), get(kD, 3), w.DL, w.DR);
    muscl<R, false>(get(kN, 0), get(kN, 1), get(kN, 2), get(kN, 3), w.UnL, w.UnR);
    muscl<R, false>(get(kG, 0), get(kG, 1), get(kG, 2), get(kG, 3), GaL, GaR);
    face_split<R, false>(w, GaL, GaR);
    const R VI = w.VI;
    const bool up = VI >= R(0.0);
    const R e = up ? R(1e-12) : R(-1e-12);
    auto side = [&](int f) {
        R u, o, v;
        upwind(f, up, u, o, v);
        return muscl_upwind<R, false>(u, o, v, e);
    };
    const R Du = up ? w.DL : w.DR;
    const R m = VI * Du;
#pragma unroll
    for (int s = 0; s < NS; ++s) F[s] = m * side(kY0 + s);
    R vel[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) vel[d] = (d == DIR) ? (up ? w.UnL : w.UnR) : side(kU + d);
    const R Hu = side(kH);
    R mom[3] = {m * vel[0], m * vel[1], m * vel[2]};
    mom[DIR] = mom[DIR] + w.G1 * w.PL + w.G2 * w.PR;
    F[NS + 0] = mom[0];
    F[NS + 1] = mom[1];
    F[NS + 2] = mom[2];
    F[NS + 3] = VI * (Du * Hu + R(0.5) * Du * (vel[0] * vel[0] + vel[1] * vel[1] + vel[2] * vel[2]));
}

// face_ausm with the direction at run time, so that one instance of the code
// serves the x, y and z faces of a kernel (a third of the instructions in the
// instruction cache). p: stencil point 0 (cell m-1) of plane 0, points `stride`
// apart, planes n3 apart. The twelve quantities that only the upwind side
// enters are read once that side is known: three points instead of four, and
// no selects between the sides. put(q, v) takes flux component q as soon as
// it is formed.
template <int NS, typename R, bool kStrict, class Put>
__device__ __forceinline__ void face_ausm_dir(int dir, const R *__restrict__ p, unsigned n3, int stride, Put put)
{
    const int kN = kU + dir, kA = dir == 0 ? kV : kU, kB = dir == 2 ? kV : kW; // normal, tangential planes
    FaceState<R> w;
    R GaL, GaR;
    auto both = [&](int q, R &l, R &r) {
        const R *b = p + (unsigned long long)n3 * unsigned(q);
        muscl<R, kStrict>(__ldg(b), __ldg(b + stride), __ldg(b + 2 * stride), __ldg(b + 3 * stride), l, r);
    };
    both(kP, w.PL, w.PR);
    both(kD, w.DL, w.DR);
    both(kN, w.UnL, w.UnR);
    both(kG, GaL, GaR);
    face_split<R, kStrict>(w, GaL, GaR);
    const R VI = w.VI;
    const bool up = VI >= R(0.0);
    const R e = up ? R(1e-12) : R(-1e-12);
    const R *pu = p + (up ? stride : 2 * stride), *pw = p + (up ? 0 : 3 * stride), *pv = p + (up ? 2 * stride : stride);
    auto side = [&](int q) {
        const unsigned long long o = (unsigned long long)n3 * unsigned(q);
        return muscl_upwind<R, kStrict>(__ldg(pu + o), __ldg(pw + o), __ldg(pv + o), e);
    };
    const R Du = up ? w.DL : w.DR;
    const R m = VI * Du;
#pragma unroll
    for (int s = 0; s < NS; ++s) put(s, m * side(kY0 + s));
    const R un = up ? w.UnL : w.UnR, va = side(kA), vb = side(kB), Hu = side(kH);
    const R momn = m * un;
    put(NS + dir, momn + w.G1 * w.PL + w.G2 * w.PR);
    put(NS + kA - kU, m * va);
    put(NS + kB - kU, m * vb);
    const R v0 = dir == 0 ? un : va, v1 = dir == 0 ? va : (dir == 1 ? un : vb), v2 = dir == 2 ? un : vb;
    put(NS + 3, VI * (Du * Hu + R(0.5) * Du * (v0 * v0 + v1 * v1 + v2 * v2)));
}

} // namespace eu3d
