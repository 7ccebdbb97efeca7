// eu3d_heavy.cuh — the stiff kinetics of one cell advanced by a whole warp: the
// same prediction, trapezoid substeps and state rebuilds as a thread per cell, for
// cells whose long serial substep chains would set the step's time on one
// thread. Included by eu3d_kernels.cuh inside the flavour's namespace.
//
// What bounds it is the latency of one substep, a chain of dependent FP64
// operations, so each stage is spread over the lanes until its chain is short
// and results change hands through a few broadcast words in shared memory:
//   rates      lane r forms reaction r (both exponentials side by side); the
//              species' Gibbs terms come from lanes s;
//   sums       the production and loss sums of species s;
//   update     lane s advances species s;
//   rebuild    the sums over species that the temperature Newton needs.
// Fast forms: the sums run on three lanes a species, each a third of its
// reactions; the rebuild works with densities (sum rho_s (h_s - R_s T) = rho e,
// no division by rho) whose ten sums (eight polynomial coefficients, R and rho)
// run on three lanes each; U, V, W and e, which the kinetics holds, are kept
// as they are. Strict forms (EU_EXACT_RATES): the expressions, operand order and
// summation order of the thread-per-cell form, so the result is bitwise that
// form's; the sums of W, Q and P run on a lane each.
#pragma once

// Tables of a block, built once from the mechanism; arrays [entry][lane], so a
// warp reads 32 consecutive words. Lanes past NR have no reaction, lanes past
// the last sum's no entries: their factors are exactly 1, their terms exactly 0.
template <int NS, int NR>
struct HeavyTables {
    static_assert(NS <= 10 && NR < 31, "three lanes a species, slot 31 holds zero rates");
    double af[32], bf[32], eaf[32], xr[32], tb[NS][32];
    double dg[6][32];                      // nu'' - nu' of the species of dgi
    unsigned char dgi[6][32];              // species whose coefficient changes, ascending
    unsigned char fi[3][32], bi[3][32];    // species of the concentration products (slot 31: a factor of 1)
#ifdef EU_EXACT_RATES
    unsigned char fsq[3][32], bsq[3][32];  // 1: the species enters squared
    double lo[9][NS], hi[9][NS], mw[NS];
    double sb[NR][32], sf[NR][32];         // lanes s, s + NS, s + 2 NS: species s's reactions, ascending
    unsigned char si[NR][32];
#else
    static constexpr int Third = (NR + 2) / 3;
    double sb[Third][32], sf[Third][32];   // lane s + NS p: species s's reactions p, p + 3, ...
    unsigned char si[Third][32];
    double wlo[(NS + 2) / 3][32], whi[(NS + 2) / 3][32]; // lane q + 10 p: weights of sum q over species 3 p ..
    double glo[9][32], ghi[9][32];         // lane s: NASA coefficients of species s
    double imw[32], mw[32];
#endif
    int most;                              // longest reaction list of a species
};

// A warp's exchange words.
struct __align__(16) HeavyScratch {
    double g[32], mc[32], nd[32], fwd[32], bwd[32], sum[32];
#ifdef EU_EXACT_RATES
    double rtb[32], y[32];
#endif
};

template <int NS, int NR>
struct HeavyShared {
    HeavyTables<NS, NR> t;
    HeavyScratch x[4]; // 128-thread blocks: four warps
};

template <int NS, int NR>
__device__ __forceinline__ void heavy_setup(const DevMech &m, HeavyShared<NS, NR> &sh)
{
    HeavyTables<NS, NR> &t = sh.t;
    for (int e = threadIdx.x; e < NS * 32; e += blockDim.x) {
        const int s = e / 32, r = e % 32;
        t.tb[s][r] = r < NR ? m.tb[r][s] : 0.0;
    }
    if (threadIdx.x < 32) {
        const int l = threadIdx.x;
        const bool real = l < NR;
        const int r = real ? l : 0;
        t.af[l] = real ? m.af[r] : 0.0;
        t.bf[l] = real ? m.bf[r] : 0.0;
        t.eaf[l] = real ? m.eaf[r] : 0.0;
        t.xr[l] = real ? m.xr[r] : 0.0;
        for (int q = 0; q < 6; ++q) {
            t.dg[q][l] = 0.0;
            t.dgi[q][l] = 0;
        }
        for (int q = 0; q < 3; ++q) {
            t.fi[q][l] = t.bi[q][l] = 31;
#ifdef EU_EXACT_RATES
            t.fsq[q][l] = t.bsq[q][l] = 0;
#endif
        }
        int nd = 0, nf = 0, nb = 0;
        for (int s = 0; real && s < NS; ++s) {
            const double f = m.sf[r][s], b = m.sb[r][s];
            if (b != f && nd < 6) {
                t.dg[nd][l] = b - f;
                t.dgi[nd++][l] = (unsigned char)s;
            }
#ifdef EU_EXACT_RATES
            if (f != 0.0 && nf < 3) {
                t.fsq[nf][l] = f == 2.0;
                t.fi[nf++][l] = (unsigned char)s;
            }
            if (b != 0.0 && nb < 3) {
                t.bsq[nb][l] = b == 2.0;
                t.bi[nb++][l] = (unsigned char)s;
            }
#else
            for (int q = 0; q < int(f) && nf < 3; ++q) t.fi[nf++][l] = (unsigned char)s;
            for (int q = 0; q < int(b) && nb < 3; ++q) t.bi[nb++][l] = (unsigned char)s;
#endif
        }
        // the reaction lists of the species sums
        const int part = l / NS, sp = l % NS;
        int n = 0, all = 0;
#ifdef EU_EXACT_RATES
        constexpr int kLen = NR, kParts = 1;
#else
        constexpr int kLen = HeavyTables<NS, NR>::Third, kParts = 3;
#endif
        for (int q = 0; part < 3 && q < NR; ++q) {
            const double b = m.sb[q][sp], f = m.sf[q][sp];
            if (b == 0.0 && f == 0.0)
                continue;
            if (kParts == 1 || all % kParts == part) {
                t.si[n][l] = (unsigned char)q;
                t.sb[n][l] = b;
                t.sf[n][l] = f;
                ++n;
            }
            ++all;
        }
        int most = n;
        for (int o = 16; o > 0; o >>= 1) most = max(most, __shfl_xor_sync(0xffffffffu, most, o));
        if (l == 0)
            t.most = most;
        for (; n < kLen; ++n) {
            t.si[n][l] = 31;
            t.sb[n][l] = t.sf[n][l] = 0.0;
        }
#ifdef EU_EXACT_RATES
        for (int k = 0; k < 9 && l < NS; ++k) {
            t.lo[k][l] = m.clo[k][l];
            t.hi[k][l] = m.chi[k][l];
        }
        if (l < NS)
            t.mw[l] = m.mw[l];
#else
        for (int k = 0; k < 9; ++k) {
            t.glo[k][l] = l < NS ? m.clo[k][l] : 0.0;
            t.ghi[k][l] = l < NS ? m.chi[k][l] : 0.0;
        }
        t.imw[l] = l < NS ? 1e-3 / m.mw[l] : 0.0;
        t.mw[l] = l < NS ? m.mw[l] : 0.0;
        // sums q = l % 10: R a_q of the enthalpy form (a3 .. a6 over 2 .. 5), R, rho
        const int q = l % 10, p = l / 10;
        const double div[8] = {1.0, 1.0, 1.0, 0.5, 1.0 / 3.0, 0.25, 0.2, 1.0};
        for (int e = 0; e < (NS + 2) / 3; ++e) {
            const int s = (NS + 2) / 3 * p + e;
            const bool in = p < 3 && s < NS;
            t.wlo[e][l] = !in ? 0.0 : q < 8 ? m.ri[s] * m.clo[q][s] * div[q] : q == 8 ? m.ri[s] : 1.0;
            t.whi[e][l] = !in ? 0.0 : q < 8 ? m.ri[s] * m.chi[q][s] * div[q] : q == 8 ? m.ri[s] : 1.0;
        }
#endif
    }
    for (int w = threadIdx.x; w < 4 * 32; w += blockDim.x) {
        HeavyScratch &x = sh.x[w / 32];
        x.mc[w % 32] = 1.0; // slot 31: the products' padding
        x.nd[w % 32] = 0.0;
        x.fwd[w % 32] = x.bwd[w % 32] = 0.0; // slot 31: the sums' padding
#ifdef EU_EXACT_RATES
        x.rtb[w % 32] = 0.0;
        x.y[w % 32] = 0.0;
#endif
    }
}

#ifdef EU_EXACT_RATES
// One rate evaluation of the strict form: lanes s, s + NS, s + 2 NS return W, Q
// and P of species s (gen_mech's emit_strict and eval_rates, term by term).
template <int NS, int NR>
__device__ __forceinline__ double heavy_rates(const HeavyTables<NS, NR> &t, HeavyScratch &x, double T,
                                              const double (&mc)[NS], int lane)
{
    const TPow p = make_tpow(T, true);
    if (lane < NS) {
        const double(*c)[NS] = p.low ? t.lo : t.hi;
        const double a0 = c[0][lane], a1 = c[1][lane], a2 = c[2][lane], a3 = c[3][lane], a4 = c[4][lane],
                     a5 = c[5][lane], a6 = c[6][lane], a7 = c[7][lane], a8 = c[8][lane];
        const double h = kRUniv * (-a0 * p.inv + a1 * p.lnT + a2 * p.T + a3 * p.t2 / 2 + a4 * p.t3 / 3 +
                                   a5 * p.t4 / 4 + a6 * p.t5 / 5 + a7);
        const double s = kRUniv * (-a0 * p.inv2 / 2 - a1 * p.inv + a2 * p.lnT + a3 * p.T + a4 * p.t2 / 2 +
                                   a5 * p.t3 / 3 + a6 * p.t4 / 4 + a8);
        x.g[lane] = h - s * T;
    }
    const double RT = kRUniv * T, RuT = kRuCal * T, p0 = kP0 * 1e-6;
    const double b = t.bf[lane], E = t.eaf[lane], Xr = t.xr[lane];
    // powers by integer exponents as selects (the thread form's values); the
    // general power on the lanes that need one
    double tp = b == 1.0 ? T : b == -1.0 ? p.inv : 1.0;
    if (b != 0.0 && b != 1.0 && b != -1.0)
        tp = pow(T, b);
    const double invRT = 1.0 / RT;
    const double ex = exp(-E / RuT);
    const double kf = t.af[lane] * tp * (E == 0.0 ? 1.0 : ex);
    double rtb = 0.0, rrf = 1.0, rrb = 1.0;
#pragma unroll
    for (int s = 0; s < NS; ++s) rtb += mc[s] * t.tb[s][lane];
    if (rtb == 0.0)
        rtb = 1.0;
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        const double f = x.mc[t.fi[q][lane]], bb = x.mc[t.bi[q][lane]];
        rrf *= t.fsq[q][lane] ? f * f : f;
        rrb *= t.bsq[q][lane] ? bb * bb : bb;
    }
    __syncwarp();
    double delta_g = 0.0;
#pragma unroll
    for (int q = 0; q < 6; ++q) delta_g += t.dg[q][lane] * x.g[t.dgi[q][lane]];
    // (|Xr| <= 1 in the mechanisms that come here)
    const double Kp = exp(-delta_g / RT) * (Xr == 0.0 ? 1.0 : Xr == 1.0 ? p0 : 1.0 / p0);
    const double Kc = Kp * (Xr == 0.0 ? 1.0 : Xr == 1.0 ? invRT : RT);
    const double kb = kf / Kc;
    const bool real = lane < NR;
    x.fwd[lane] = real ? kf * rrf : 0.0;
    x.bwd[lane] = real ? kb * rrb : 0.0;
    x.rtb[lane] = real ? rtb : 0.0;
    __syncwarp();
    double sum = 0.0;
    const int kind = lane / NS, most = t.most; // 0: W, 1: Q, 2: P
#pragma unroll 4
    for (int i = 0; i < most; ++i) {
        const int q = t.si[i][lane];
        const double bb = t.sb[i][lane], f = t.sf[i][lane], fr = x.fwd[q], br = x.bwd[q], tr = x.rtb[q];
        const double w = (bb - f) * tr * (fr - br);
        const double qp = kind == 1 ? (bb * fr + f * br) * tr : (bb * br + f * fr) * tr;
        sum += kind == 0 ? w : qp;
    }
    __syncwarp();
    return sum;
}

// Advances the recovered cell by dtm in the strict form. Returns Nchem.
template <int NS, int NR>
__device__ __forceinline__ int heavy_advance(const DevMech &m, const HeavyTables<NS, NR> &t, HeavyScratch &x,
                                             CellState<NS> &cell, double dtm, int max_substeps,
                                             unsigned long long *counters, double *cms, long long cms_stride, int lane)
{
    const int sp = lane < NS ? lane : 0;
    const double mw = t.mw[sp];
    double csl = 0.0; // lane s: species s's density
#pragma unroll
    for (int s = 0; s < NS; ++s) csl = sp == s ? cell.cs[s] : csl;
    double mc[NS];
    auto rates = [&](double &W, double &Q, double &P) {
        const double mcl = (csl / mw * 1000) * 1e-6; // scaled_concentrations, a species a lane
        if (lane < NS)
            x.mc[lane] = mcl;
        __syncwarp();
#pragma unroll
        for (int s = 0; s < NS; ++s) mc[s] = x.mc[s];
        const double v = heavy_rates<NS, NR>(t, x, cell.T, mc, lane);
        W = mw * v;
        Q = __shfl_sync(0xffffffffu, v, sp + NS);
        P = __shfl_sync(0xffffffffu, v, sp + 2 * NS);
        return mcl;
    };
    double W, Q, P;
    double mcl = rates(W, Q, P);
    double dt = dtm;
    {
        double yl = 0.0;
#pragma unroll
        for (int s = 0; s < NS; ++s) yl = sp == s ? cell.Y[s] : yl;
        const double d = fabs(-(csl * 1e-3) / W);
        if (lane < NS && yl >= 1e-6 && W != 0 && d < dt)
            dt = d;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) dt = fmin(dt, __shfl_xor_sync(0xffffffffu, dt, o));
    int nchem = 0;
    if (lane == 0) {
        bool bad;
        nchem = nchem_from_dt(dtm, dt, max_substeps, bad);
        count_nchem(counters, nchem, bad);
    }
    nchem = __shfl_sync(0xffffffffu, nchem, 0);
    const double dts = dtm / nchem, half = dts / 2.0;
    for (int step = 0; step < nchem; ++step) {
        if (step > 0)
            mcl = rates(W, Q, P);
        if (cms && lane < NS)
            cms[lane * cms_stride] = W * 1e3;
        const double di = csl * 1e-3, q = mw * Q;
        const double pq = P / mcl;
        const double p = (mcl == 0) ? 0.0 : pq;
        csl = ((1.0 - half * p) * di + dts * q) / (1.0 + half * p) * 1e3;
        if (lane < NS)
            x.nd[lane] = csl;
        __syncwarp();
        double D = 0.0;
#pragma unroll
        for (int s = 0; s < NS; ++s) {
            cell.cs[s] = x.nd[s];
            D += cell.cs[s];
        }
        cell.cs[NS + 0] = cell.U * D;
        cell.cs[NS + 1] = cell.V * D;
        cell.cs[NS + 2] = cell.W * D;
        cell.cs[NS + 3] = D * cell.E + 0.5 * (cell.U * cell.U + cell.V * cell.V + cell.W * cell.W) * D;
        // recover_state, the divisions by the density and the species' terms of
        // the Newton's sums on their lanes, the sums in species order on all
        double Dr = 0.0;
#pragma unroll
        for (int s = 0; s < NS; ++s) Dr += cell.cs[s];
        const double yl = csl / Dr;
        if (lane < NS)
            x.y[lane] = yl;
        const double mom = lane == 0 ? cell.cs[NS + 0] : lane == 1 ? cell.cs[NS + 1] : cell.cs[NS + 2];
        const double vel = mom / Dr;
        __syncwarp();
        double rsum = 0;
#pragma unroll
        for (int s = 0; s < NS; ++s) {
            cell.Y[s] = x.y[s];
            rsum += cell.Y[s] * m.ri[s];
        }
        cell.D = Dr;
        const double e_scaled = cell.E * 1e-3;
        double T_temp = cell.T;
        const double ri = kRUniv / mw;
        for (int count = 0; count < 10; ++count) {
            const double T0 = T_temp;
            const TPow pw = make_tpow(T0, true);
            const double(*c)[NS] = pw.low ? t.lo : t.hi;
            const int s = lane < NS ? lane : lane < 2 * NS ? lane - NS : 0;
            const double a0 = c[0][s], a1 = c[1][s], a2 = c[2][s], a3 = c[3][s], a4 = c[4][s], a5 = c[5][s],
                         a6 = c[6][s], a7 = c[7][s];
            const double Rs = __shfl_sync(0xffffffffu, ri, s);
            const double hv = Rs * (-a0 * pw.inv + a1 * pw.lnT + a2 * pw.T + a3 * pw.t2 / 2 + a4 * pw.t3 / 3 +
                                    a5 * pw.t4 / 4 + a6 * pw.t5 / 5 + a7);
            const double cv = Rs * (a0 * pw.inv2 + a1 * pw.inv + a2 + a3 * pw.T + a4 * pw.t2 + a5 * pw.t3 + a6 * pw.t4);
            x.sum[lane] = x.y[s] * (lane < NS ? hv : cv);
            __syncwarp();
            double hsum = 0, cpsum = 0;
#pragma unroll
            for (int q2 = 0; q2 < NS; ++q2) {
                hsum += x.sum[q2];
                cpsum += x.sum[NS + q2];
            }
            __syncwarp();
            const double temp1 = (hsum - e_scaled) - rsum * T0;
            const double temp2 = cpsum - rsum;
            T_temp = T0 - temp1 / temp2;
            if (fabs(T_temp - T0) < 1e-6)
                break;
        }
        cell.T = T_temp;
        cell.U = __shfl_sync(0xffffffffu, vel, 0);
        cell.V = __shfl_sync(0xffffffffu, vel, 1);
        cell.W = __shfl_sync(0xffffffffu, vel, 2);
        cell.E = (cell.cs[NS + 3] - 0.5 * Dr * (cell.U * cell.U + cell.V * cell.V + cell.W * cell.W)) / Dr;
    }
    return nchem;
}
#else
// log(1 + x), |x| <= 2^-6, as log1p_small with the terms paired (a third of the
// dependent operations).
__device__ __forceinline__ double log1p_paired(double x)
{
    const double x2 = x * x, x4 = x2 * x2;
    const double a = fma(-1.0 / 2.0, x, 1.0), b = fma(-1.0 / 4.0, x, 1.0 / 3.0), c = fma(-1.0 / 6.0, x, 1.0 / 5.0),
                 d = fma(-1.0 / 8.0, x, 1.0 / 7.0);
    const double ab = fma(b, x2, a), cd = fma(d, x2, c);
    return x * fma(fma(1.0 / 9.0, x4, cd), x4, ab);
}

// One rate evaluation of the fast form: lane s returns Q and P of species s.
// mc: every species' concentration is in x.mc, this lane's in mcl.
template <int NS, int NR>
__device__ __forceinline__ void heavy_rates(const HeavyTables<NS, NR> &t, HeavyScratch &x, double T, double inv,
                                            double lnT, int lane, double &Q, double &P)
{
    {
        // g_s = G_s/(R T) on lanes s
        const double(*c)[32] = T < kThermoSwitch ? t.glo : t.ghi;
        double f[9];
        gibbs_terms(T, inv, lnT, f);
        const double u = fma(f[1], c[1][lane], f[0] * c[0][lane]), v = fma(f[3], c[3][lane], f[2] * c[2][lane]),
                     w = fma(f[5], c[5][lane], f[4] * c[4][lane]), y = fma(f[7], c[7][lane], f[6] * c[6][lane]);
        x.g[lane] = ((u + v) + (w + y)) - c[8][lane];
    }
    const double b = t.bf[lane], E = t.eaf[lane], Xr = t.xr[lane];
    // Every candidate is formed before it is chosen, so the choices are
    // selects: the lanes hold different reactions.
    const double e = fma(b, lnT, -E * (inv * (1.0 / kRuCal))), ex = exp_paired(e);
    double tpow = ex;
    const bool plain = E == 0.0;
    tpow = plain && b == 1.0 ? T : tpow;
    tpow = plain && b == -1.0 ? inv : tpow;
    tpow = plain && b == -2.0 ? inv * inv : tpow;
    const double kf = t.af[lane] * tpow;
    double r0 = 0.0, r1 = 0.0;
#pragma unroll
    for (int s = 0; s < NS; ++s) {
        if (s % 2)
            r1 = fma(x.mc[s], t.tb[s][lane], r1);
        else
            r0 = fma(x.mc[s], t.tb[s][lane], r0);
    }
    double rtb = r0 + r1;
    if (rtb == 0.0)
        rtb = 1.0;
    const double rrf = (x.mc[t.fi[0][lane]] * x.mc[t.fi[1][lane]]) * x.mc[t.fi[2][lane]];
    const double rrb = (x.mc[t.bi[0][lane]] * x.mc[t.bi[1][lane]]) * x.mc[t.bi[2][lane]];
    double kt = kf * rtb;
    double back = rrb;
    back *= Xr == 0.0 ? 1.0 : Xr == 1.0 ? T * (kRUniv / (kP0 * 1e-6)) : inv * (kP0 * 1e-6 / kRUniv);
    __syncwarp();
    double d0 = 0.0, d1 = 0.0;
#pragma unroll
    for (int q = 0; q < 6; q += 2) {
        d0 = fma(t.dg[q][lane], x.g[t.dgi[q][lane]], d0);
        d1 = fma(t.dg[q + 1][lane], x.g[t.dgi[q + 1][lane]], d1);
    }
    const bool real = lane < NR; // slot 31 (and every slot past NR) holds zero rates
    const double dg = d0 + d1;
    double fr = kt * rrf, br = (kt * back) * exp_paired(dg);
    if (max(__double2hiint(e) & 0x7fffffff, __double2hiint(dg) & 0x7fffffff) >= __double2hiint(kExpMost)) { // as eval_rates_far
        const double art = t.af[lane] * rtb;
        fr = art * exp(e) * rrf;
        br = art * exp(e + dg) * back;
    }
    x.fwd[lane] = real ? fr : 0.0;
    x.bwd[lane] = real ? br : 0.0;
    __syncwarp();
    // species sums, a third of the reactions a lane
    double q0 = 0.0, p0 = 0.0;
    auto sums = [&](auto len) {
        constexpr int L = decltype(len)::value;
#pragma unroll
        for (int i = 0; i < L; ++i) {
            const int r = t.si[i][lane];
            const double bb = t.sb[i][lane], f = t.sf[i][lane], fr = x.fwd[r], br = x.bwd[r];
            q0 = fma(bb, fr, fma(f, br, q0));
            p0 = fma(bb, br, fma(f, fr, p0));
        }
    };
    if (t.most <= 4)
        sums(std::integral_constant<int, 4>{});
    else
        sums(std::integral_constant<int, HeavyTables<NS, NR>::Third>{});
    const int l1 = lane + NS < 32 ? lane + NS : lane, l2 = lane + 2 * NS < 32 ? lane + 2 * NS : lane;
    const double qa = __shfl_sync(0xffffffffu, q0, l1), qb = __shfl_sync(0xffffffffu, q0, l2);
    const double pa = __shfl_sync(0xffffffffu, p0, l1), pb = __shfl_sync(0xffffffffu, p0, l2);
    Q = q0 + (qa + qb);
    P = p0 + (pa + pb);
}

// Advances the recovered cell by dtm in the fast form. Returns Nchem.
template <int NS, int NR>
__device__ __forceinline__ int heavy_advance(const DevMech &m, const HeavyTables<NS, NR> &t, HeavyScratch &x,
                                             CellState<NS> &cell, double dtm, int max_substeps,
                                             unsigned long long *counters, double *cms, long long cms_stride, int lane)
{
    constexpr int kPer = (NS + 2) / 3;
    const double mw = t.mw[lane], imw = t.imw[lane];
    double csl = 0.0; // lane s: species s's density
#pragma unroll
    for (int s = 0; s < NS; ++s) csl = lane == s ? cell.cs[s] : csl;
    double T = cell.T, inv = cell.inv, lnT = cell.lnT, Q, P;
    auto rates = [&] {
        const double mcl = csl * imw;
        if (lane < NS) {
            x.mc[lane] = mcl;
            x.nd[lane] = csl;
        }
        __syncwarp();
        heavy_rates<NS, NR>(t, x, T, inv, lnT, lane, Q, P);
        return mcl;
    };
    double mcl = rates();
    // prediction: min over the species lanes, then every lane has Nchem
    double dt = dtm;
    {
        const double W = mw * (Q - P);
        double yl = 0.0;
#pragma unroll
        for (int s = 0; s < NS; ++s) yl = lane == s ? cell.Y[s] : yl;
        const double d = fabs(csl * 1e-3 * rcp_nr(W));
        if (lane < NS && yl >= 1e-6 && W != 0 && d < dt)
            dt = d;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) dt = fmin(dt, __shfl_xor_sync(0xffffffffu, dt, o));
    int nchem = 0;
    if (lane == 0) {
        bool bad;
        nchem = nchem_from_dt(dtm, dt, max_substeps, bad);
        count_nchem(counters, nchem, bad);
    }
    nchem = __shfl_sync(0xffffffffu, nchem, 0);
    const double dts = dtm / nchem, half = dts * 0.5, e_scaled = cell.E * 1e-3;
    const int sum_at = lane / 10 < 3 ? kPer * (lane / 10) : 0; // first species of this lane's share of its sum
    for (int step = 0; step < nchem; ++step) {
        if (step > 0)
            mcl = rates();
        if (cms && lane < NS)
            cms[lane * cms_stride] = mw * (Q - P) * 1e3;
        {
            const double di = csl * 1e-3;
            const double hp = half * loss_frequency(P, mcl);
            csl = fma(dts, mw * Q, fma(-hp, di, di)) * rcp_nr(1.0 + hp) * 1e3;
        }
        __syncwarp();
        if (lane < NS)
            x.nd[lane] = csl;
        __syncwarp();
        // the rebuild's sums over species for the NASA range of T0
        double A[10];
        bool low = T < kThermoSwitch;
        auto sums = [&] {
            const double(*w)[32] = low ? t.wlo : t.whi;
            double v = 0.0;
#pragma unroll
            for (int e = 0; e < kPer; ++e) v = fma(x.nd[sum_at + e], w[e][lane], v);
            const double a = __shfl_down_sync(0xffffffffu, v, 10), b = __shfl_down_sync(0xffffffffu, v, 20);
            x.sum[lane] = v + (a + b);
            __syncwarp();
#pragma unroll
            for (int q = 0; q < 10; ++q) A[q] = x.sum[q];
            __syncwarp();
        };
        sums();
        double T0 = T, inv0 = inv, ln0 = lnT;
        for (int count = 0; count < 10; ++count) {
            const bool l = T0 < kThermoSwitch;
            if (l != low) {
                low = l;
                sums();
            }
            const double t2 = T0 * T0;
            // rho (h - e) - rho R T and its derivative
            const double h = fma(fma(fma(A[6], T0, A[5]), t2, fma(A[4], T0, A[3])), t2, fma(A[2], T0, A[7])) +
                             fma(A[1], ln0, -A[0] * inv0);
            const double c = fma(fma(5.0 * A[6], t2, fma(4.0 * A[5], T0, 3.0 * A[4])), t2, fma(2.0 * A[3], T0, A[2])) +
                             inv0 * fma(A[0], inv0, A[1]);
            const double resid = h - fma(A[8], T0, A[9] * e_scaled);
            const double step_T = resid * rcp_nr(c - A[8]);
            const double T1 = T0 - step_T;
            const double xr = (T1 - T0) * inv0;
            ln0 = fabs(xr) <= 0x1p-6 ? ln0 + log1p_paired(xr) : log(T1);
            inv0 = rcp_nr(T1);
            const bool done = fabs(T1 - T0) < 1e-6;
            T0 = T1;
            if (done)
                break;
        }
        T = T0;
        inv = inv0;
        lnT = ln0;
    }
    // the cell's state from the last densities
    cell.T = T;
    cell.inv = inv;
    cell.lnT = lnT;
    double D = 0.0;
#pragma unroll
    for (int s = 0; s < NS; ++s) {
        cell.cs[s] = x.nd[s];
        D += cell.cs[s];
    }
    const double invD = rcp_nr(D);
#pragma unroll
    for (int s = 0; s < NS; ++s) cell.Y[s] = cell.cs[s] * invD;
    cell.D = D;
    cell.cs[NS + 0] = cell.U * D;
    cell.cs[NS + 1] = cell.V * D;
    cell.cs[NS + 2] = cell.W * D;
    cell.cs[NS + 3] = D * cell.E + 0.5 * (cell.U * cell.U + cell.V * cell.V + cell.W * cell.W) * D;
    __syncwarp();
    return nchem;
}
#endif

// One deferred cell whose recovered state is stored.
template <int NS, int NR>
__device__ __forceinline__ void react_heavy_cell(const DevMech &m, const HeavyTables<NS, NR> &t, HeavyScratch &x,
                                                 const DevState &st, long long n3, long long c, double dtm,
                                                 int max_substeps, int lane)
{
    CellState<NS> cell;
    load_recovered<NS>(st, n3, c, cell);
    const int nchem = heavy_advance<NS, NR>(m, t, x, cell, dtm, max_substeps, st.counters,
                                            st.cms ? st.cms + c : nullptr, n3, lane);
    if (lane == 0) {
        st.nchem[c] = nchem;
        store_cell<NS>(m, st, n3, c, cell);
    }
    __syncwarp();
}

// The order in which the warps of a persistent grid take deferred cells:
// position p of n is entry p * s mod n, s near 0.618 n and coprime with n (a
// bijection of [0, n)). The queue holds the cells in about the order the
// recovery met them, so neighbouring cells, whose stiffness is alike, sit
// next to each other; the warps that start together belong to few blocks,
// and without the scatter the stiffest cells would share a few SMs.
__device__ __forceinline__ long long scatter_stride(long long n)
{
    long long s = static_cast<long long>(0.6180339887498949 * double(n)) | 1;
    for (;;) {
        long long a = s, b = n;
        while (b != 0) {
            const long long t = a % b;
            a = b;
            b = t;
        }
        if (a == 1)
            return s;
        s += 2;
    }
}

// Every position of [0, count) given to one warp of the grid, in scattered
// order, from the counter *next (zero at launch): one(entry, scratch, lane).
template <int NS, int NR, class One>
__device__ __forceinline__ void heavy_drain(const DevMech &m, int count, int *next, One one)
{
    __shared__ HeavyShared<NS, NR> sh;
    if (count == 0) // no deferred cell: skip the tables
        return;
    heavy_setup<NS, NR>(m, sh);
    __syncthreads();
    const int lane = threadIdx.x & 31;
    HeavyScratch &x = sh.x[threadIdx.x / 32];
    const long long stride = scatter_stride(count);
    for (;;) {
        int q = 0;
        if (lane == 0)
            q = atomicAdd(next, 1);
        q = __shfl_sync(0xffffffffu, q, 0);
        if (q >= count)
            break;
        one(int((q * stride) % count), sh.t, x, lane);
    }
}

constexpr int kHeavyBlocksPerSm = 3; // resident 128-thread blocks the register allocation aims at

template <int NS, int NR>
__global__ void __launch_bounds__(128, kHeavyBlocksPerSm)
    k_react_heavy(const __grid_constant__ DevMech m, const DevGrid g, const DevState st,
                  const double *__restrict__ dt_dev, int max_substeps)
{
    heavy_drain<NS, NR>(m, st.heavy[0], &st.heavy[1], [&](int e, const auto &t, HeavyScratch &x, int lane) {
        react_heavy_cell<NS, NR>(m, t, x, st, g.n3, st.heavy[2 + e], *dt_dev, max_substeps, lane);
    });
}

// The deferred cells of every instance of a batch, their heavy queues taken
// end to end, drained by one persistent grid (one warp per cell, one counter).
template <int NS, int NR>
__global__ void __launch_bounds__(128, kHeavyBlocksPerSm)
    k_react_heavy_batch(const __grid_constant__ DevMech m, const BatchCell *__restrict__ tab, int n, int *next,
                        int max_substeps)
{
    auto len = [&](int q) { return tab[q].st.heavy ? *(volatile const int *)tab[q].st.heavy : 0; };
    int total = 0;
    for (int q = 0; q < n; ++q) total += len(q);
    heavy_drain<NS, NR>(m, total, next, [&](int e, const auto &t, HeavyScratch &x, int lane) {
        int local = 0;
        const int q = batch_locate(n, e, len, local);
        if (q < n) {
            const BatchCell &b = tab[q];
            react_heavy_cell<NS, NR>(m, t, x, b.st, b.n3, b.st.heavy[2 + local], *b.dt, max_substeps, lane);
        }
    });
}

// The deferred samples of k_chem_samples (eu_chem_advance).
template <int NS, int NR>
__global__ void __launch_bounds__(128, kHeavyBlocksPerSm)
    k_chem_heavy(const __grid_constant__ DevMech m, long long n, double *cs, double *T, double *E,
                 const double *__restrict__ dt, int *nchem, int max_substeps, unsigned long long *counters, int *heavy)
{
    heavy_drain<NS, NR>(m, heavy[0], &heavy[1], [&](int e, const auto &t, HeavyScratch &x, int lane) {
        const long long i = heavy[2 + e];
        CellState<NS> cell;
        load_sample<NS>(n, i, cs, T, E, cell);
        const int nc = heavy_advance<NS, NR>(m, t, x, cell, dt[i], max_substeps, counters, nullptr, 0, lane);
        if (lane == 0) {
            if (nchem)
                nchem[i] = nc;
            store_sample<NS>(n, i, cs, T, E, cell);
        }
        __syncwarp();
    });
}
