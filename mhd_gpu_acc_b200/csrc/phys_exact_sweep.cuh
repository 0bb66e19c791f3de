// phys_exact_sweep.cuh -- the FP64 physics of the sweeps: phys_exact.cuh's
// results, bit for bit, arranged for the device.
//
//   * Quotients and roots come in branch-free groups (exact_div.cuh) that share a
//     denominator's reciprocal where they can: a state's 1 / rho serves its
//     velocities and the three quotients of its fast speed, S - S_M the star
//     density and energy, HLLD's d four quotients.
//   * A face-side state carries its primitives (Side): the reconstruction makes
//     them for its positivity test, and phys_exact.cuh's solvers would form
//     the same values again from the conserved state.
//   * The solvers evaluate the flux and star state of the side that owns the
//     face only (the other side's would be computed and not used).
// Every value that is used is formed by phys_exact.cuh's operations in
// phys_exact.cuh's order (a + b = b + a and a b = b a are the only exchanges),
// so results are identical; tests/exact_sweep_check.cu compares the two.
// Measured on B200 at 2048^2 (HLLD, van Leer): see ExactPolicy (step_f64.cu).
#pragma once

#include "exact_div.cuh"
#include "phys_exact.cuh"

namespace mhd {
namespace exact {

// [0, 9) U, then u, v, w, p and 1 / rho of it.
struct Side {
    double v[14];
    MHD_HD_INLINE double ir() const { return v[13]; }
    MHD_HD_INLINE double p() const { return v[12]; }
    MHD_HD_INLINE double vel(int k) const { return v[9 + k]; }
};

// Low 32 bits do not matter: a double is finite when its exponent is not all ones.
MHD_HD_INLINE bool finite_d(double a) {
    const unsigned h = hi_word(a);
    return h + h < 0xffe00000u;
}

// u, v, w, p (and 1 / rho at ir) of a conserved state, as c2p and flux form them.
MHD_HD_INLINE void prim_of(const double* U, double ir, double g, double& u, double& v, double& w, double& p) {
    u = U[MX] * ir;
    v = U[MY] * ir;
    w = U[MZ] * ir;
    const double Bmag2 = U[BX] * U[BX] + U[BY] * U[BY] + U[BZ] * U[BZ];
    const double ke = 0.5 * U[RHO] * (u * u + v * v + w * w);
    p = (g - 1.0) * (U[EN] - ke - 0.5 * Bmag2);
}

MHD_HD_INLINE void side_of(const double* U, double g, Side& S) {
    double ir;
    reciprocals<1>(U, &ir);  // of U[RHO]
#pragma unroll
    for (int k = 0; k < NV; ++k) S.v[k] = U[k];
    S.v[13] = ir;
    prim_of(U, ir, g, S.v[9], S.v[10], S.v[11], S.v[12]);
}

MHD_HD_INLINE void c2p_grouped(const double* U, double g, double* W) {
    double ir;
    reciprocals<1>(U, &ir);
    W[RHO] = U[RHO];
    prim_of(U, ir, g, W[PU], W[PV], W[PW], W[PP]);
    W[BX] = U[BX]; W[BY] = U[BY]; W[BZ] = U[BZ]; W[PSI] = U[PSI];
}

// flux<DIR> of a state with its primitives
template <int DIR>
MHD_HD_INLINE void flux_of(const double* U, double ux, double uy, double uz, double p, double ch, double* F) {
    const double Bmag2 = U[BX] * U[BX] + U[BY] * U[BY] + U[BZ] * U[BZ];
    const double p_tot = p + 0.5 * Bmag2;
    const double BdotU = U[BX] * ux + U[BY] * uy + U[BZ] * uz;
    if (DIR == 0) {
        F[0] = U[MX];
        F[1] = U[MX] * ux + p_tot - U[BX] * U[BX];
        F[2] = U[MX] * uy - U[BX] * U[BY];
        F[3] = U[MX] * uz - U[BX] * U[BZ];
        F[4] = U[PSI];
        F[5] = U[BY] * ux - U[BX] * uy;
        F[6] = U[BZ] * ux - U[BX] * uz;
        F[7] = (U[EN] + p_tot) * ux - U[BX] * BdotU;
        F[8] = ch * ch * U[BX];
    } else {
        F[0] = U[MY];
        F[1] = U[MY] * ux - U[BY] * U[BX];
        F[2] = U[MY] * uy + p_tot - U[BY] * U[BY];
        F[3] = U[MY] * uz - U[BY] * U[BZ];
        F[4] = U[BX] * uy - U[BY] * ux;
        F[5] = U[PSI];
        F[6] = U[BZ] * uy - U[BY] * uz;
        F[7] = (U[EN] + p_tot) * uy - U[BY] * BdotU;
        F[8] = ch * ch * U[BY];
    }
}
template <int DIR>
MHD_HD_INLINE void flux_of(const Side& S, double ch, double* F) {
    flux_of<DIR>(S.v, S.v[9], S.v[10], S.v[11], S.v[12], ch, F);
}

// fast_speed<DIR> of both sides of a face.
MHD_HD_INLINE double fast_native(double gp, double B2, double Bn, double rho) {
    const double a2 = gp / rho, b2 = B2 / rho, bn2 = Bn * Bn / rho;
    const double disc = (a2 + b2) * (a2 + b2) - 4.0 * a2 * bn2;
    return sqrt(0.5 * (a2 + b2 + sqrt(disc > 0.0 ? disc : 0.0)));
}
MHD_HD_INLINE double fast_group(double gp, double B2, double Bn, double rho, double ir, bool& bad) {
    const Recip r = recip_of(rho, ir);
    const double Bn2 = Bn * Bn;
    // p > 0 and rho > 0 here (riemann_physical), so no quotient is a negative zero
    const double a2 = quot_pos(gp, r), b2 = quot_pos(B2, r), bn2 = quot_pos(Bn2, r);
    const double disc = (a2 + b2) * (a2 + b2) - 4.0 * a2 * bn2;
    const double d0 = disc > 0.0 ? disc : 0.0;
    const double h = 0.5 * (a2 + b2 + root(d0));
    bad = bad | out_den(rho) | out_num(gp) | out_num(B2) | out_num(Bn2) | out_rad(d0) | out_rad(h);
    return root(h);
}
template <int DIR>
MHD_HD_INLINE void fast_speeds(const Side& L, const Side& R, double g, double& cfL, double& cfR) {
    const double gpL = g * L.p(), gpR = g * R.p();
    const double B2L = L.v[BX] * L.v[BX] + L.v[BY] * L.v[BY] + L.v[BZ] * L.v[BZ];
    const double B2R = R.v[BX] * R.v[BX] + R.v[BY] * R.v[BY] + R.v[BZ] * R.v[BZ];
    const double BnL = (DIR == 0) ? L.v[BX] : L.v[BY], BnR = (DIR == 0) ? R.v[BX] : R.v[BY];
    bool bad = false;
    cfL = fast_group(gpL, B2L, BnL, L.v[RHO], L.ir(), bad);
    cfR = fast_group(gpR, B2R, BnR, R.v[RHO], R.ir(), bad);
    if (bad) {
        cfL = fast_native(gpL, B2L, BnL, L.v[RHO]);
        cfR = fast_native(gpR, B2R, BnR, R.v[RHO]);
    }
}

MHD_HD_INLINE bool usable(const Side& S) {
    return finite_d(S.v[RHO]) && finite_d(S.p()) && S.v[RHO] > 0.0 && S.p() > 0.0;
}

template <int DIR>
MHD_HD_INLINE void rotate_side(const Side& S, double& un, double& ut, double& uw, double& Bn, double& Bt, double& Bw) {
    uw = S.vel(2);
    Bw = S.v[BZ];
    if (DIR == 0) { un = S.vel(0); ut = S.vel(1); Bn = S.v[BX]; Bt = S.v[BY]; }
    else          { un = S.vel(1); ut = S.vel(0); Bn = S.v[BY]; Bt = S.v[BX]; }
}

template <int DIR>
MHD_HD_INLINE void hll_of(const Side& L, const Side& R, double ch, double g, double* F) {
    double FL[NV], FR[NV];
    flux_of<DIR>(L, ch, FL);
    flux_of<DIR>(R, ch, FR);
    if (!usable(L) || !usable(R)) {
#pragma unroll
        for (int k = 0; k < NV; ++k) F[k] = 0.5 * (FL[k] + FR[k]);
        return;
    }
    double cfL, cfR;
    fast_speeds<DIR>(L, R, g, cfL, cfR);
    const double unL = L.vel(DIR), unR = R.vel(DIR);
    const double SL = fmin(fmin(unL - cfL, unR - cfR), -ch);
    const double SR = fmax(fmax(unL + cfL, unR + cfR), ch);
    if (SL >= 0.0) {
#pragma unroll
        for (int k = 0; k < NV; ++k) F[k] = FL[k];
        return;
    }
    if (SR <= 0.0) {
#pragma unroll
        for (int k = 0; k < NV; ++k) F[k] = FR[k];
        return;
    }
    const double denom = SR - SL;
    if (fabs(denom) < 1.0e-14) {
#pragma unroll
        for (int k = 0; k < NV; ++k) F[k] = 0.5 * (FL[k] + FR[k]);
        return;
    }
    double inv;
    reciprocals<1>(&denom, &inv);
    const double SLSR = SL * SR;
#pragma unroll
    for (int k = 0; k < NV; ++k) F[k] = inv * (SR * FL[k] - SL * FR[k] + SLSR * (R.v[k] - L.v[k]));
}

// The contact speed and both star densities (the solvers' common part), with
// r = 1 / (S - S_M) of the side that owns the face.  False where the solver gives up.
MHD_HD_INLINE bool contact(double rhoL, double unL, double ptL, double SL, double rhoR, double unR, double ptR, double SR,
                           double& SM, double& rhoLs, double& rhoRs, Recip& rs) {
    const double numerSM = (SR - unR) * rhoR * unR - (SL - unL) * rhoL * unL + ptL - ptR;
    const double denomSM = (SR - unR) * rhoR - (SL - unL) * rhoL;
    if (fabs(denomSM) < 1.0e-14) return false;
    SM = quot(numerSM, recip(denomSM));
    const double nL = rhoL * (SL - unL), nR = rhoR * (SR - unR);
    Recip rL = recip(SL - SM), rR = recip(SR - SM);
    rhoLs = quot(nL, rL);
    rhoRs = quot(nR, rR);
    if (out_num(numerSM) | out_den(denomSM) | out_num(nL) | out_num(nR) | out_den(rL.b) | out_den(rR.b)) {
        SM = numerSM / denomSM;
        rL = recip(SL - SM);
        rR = recip(SR - SM);
        rhoLs = nL / rL.b;
        rhoRs = nR / rR.b;
    }
    const bool left = SM >= 0.0;
    rs.b = left ? rL.b : rR.b;
    rs.y1 = left ? rL.y1 : rR.y1;
    rs.e1 = left ? rL.e1 : rR.e1;
    rs.y = left ? rL.y : rR.y;
    return !(rhoLs <= 0.0 || rhoRs <= 0.0 || !finite_d(rhoLs) || !finite_d(rhoRs));
}

template <int DIR>
MHD_HD_INLINE bool hllc_star_of(const Side& L, const Side& R, double ch, double g, double* F) {
    if (!usable(L) || !usable(R)) return false;
    double unL, unR, utL, utR, uwL, uwR, BnL, BnR, BtL, BtR, BwL, BwR;
    rotate_side<DIR>(L, unL, utL, uwL, BnL, BtL, BwL);
    rotate_side<DIR>(R, unR, utR, uwR, BnR, BtR, BwR);
    double cfL, cfR;
    fast_speeds<DIR>(L, R, g, cfL, cfR);
    const double SL = fmin(unL - cfL, unR - cfR);
    const double SR = fmax(unL + cfL, unR + cfR);
    if (SL >= 0.0) { flux_of<DIR>(L, ch, F); return true; }
    if (SR <= 0.0) { flux_of<DIR>(R, ch, F); return true; }
    const double ptL = L.p() + 0.5 * (BnL * BnL + BtL * BtL + BwL * BwL);
    const double ptR = R.p() + 0.5 * (BnR * BnR + BtR * BtR + BwR * BwR);
    double SM, rhoLs, rhoRs;
    Recip rs;
    if (!contact(L.v[RHO], unL, ptL, SL, R.v[RHO], unR, ptR, SR, SM, rhoLs, rhoRs, rs)) return false;
    const double psiM = 0.5 * (L.v[PSI] + R.v[PSI]) - 0.5 * ch * (BnR - BnL);
    const bool left = SM >= 0.0;
    const double S = left ? SL : SR, rho = left ? L.v[RHO] : R.v[RHO], un = left ? unL : unR;
    const double ut = left ? utL : utR, uw = left ? uwL : uwR, Bn = left ? BnL : BnR, Bt = left ? BtL : BtR;
    const double Bw = left ? BwL : BwR, pt = left ? ptL : ptR, rhos = left ? rhoLs : rhoRs;
    Side O;
#pragma unroll
    for (int k = 0; k < 13; ++k) O.v[k] = left ? L.v[k] : R.v[k];
    const double pts = pt + rho * (S - un) * (SM - un);
    const double BdotU = Bn * un + Bt * ut + Bw * uw, BdotUs = Bn * SM + Bt * ut + Bw * uw;
    const double nE = (S - un) * O.v[EN] - pt * un + pts * SM + Bn * (BdotUs - BdotU);
    double Es = quot(nE, rs);
    if (out_num(nE) | out_den(rs.b)) Es = nE / rs.b;
    double Us[NV], Fs[NV];
    build_star<DIR>(rhos, SM, ut, uw, Bn, Bt, Bw, Es, psiM, Us);
    flux_of<DIR>(O, ch, Fs);
#pragma unroll
    for (int k = 0; k < NV; ++k) F[k] = Fs[k] + S * (Us[k] - O.v[k]);
    return true;
}

// HLLD's single-star tangential state of a side; adds to `bad` where the group's
// quotients do not hold (star_native then forms them).
struct Star {
    double ut, uw, Bt, Bw;
};
MHD_HD_INLINE Star star_native(double rho, double un, double ut, double uw, double Bn, double Bt, double Bw, double S,
                               double SM) {
    const double d = rho * (S - un) * (S - SM) - Bn * Bn;
    if (fabs(d) < 1.0e-14) return Star{ut, uw, Bt, Bw};
    return Star{ut - Bn * Bt * (SM - un) / d, uw - Bn * Bw * (SM - un) / d,
                Bt * (rho * (S - un) * (S - un) - Bn * Bn) / d, Bw * (rho * (S - un) * (S - un) - Bn * Bn) / d};
}
MHD_HD_INLINE Star star_group(double rho, double un, double ut, double uw, double Bn, double Bt, double Bw, double S,
                              double SM, bool& bad) {
    const double d = rho * (S - un) * (S - SM) - Bn * Bn;
    const bool degenerate = fabs(d) < 1.0e-14;
    const Recip r = recip(d);
    const double n1 = Bn * Bt * (SM - un), n2 = Bn * Bw * (SM - un);
    const double f = rho * (S - un) * (S - un) - Bn * Bn, n3 = Bt * f, n4 = Bw * f;
    const double q1 = quot(n1, r), q2 = quot(n2, r), q3 = quot(n3, r), q4 = quot(n4, r);
    bad = bad | (!degenerate & (out_den(d) | out_num(n1) | out_num(n2) | out_num(n3) | out_num(n4)));
    return Star{degenerate ? ut : ut - q1, degenerate ? uw : uw - q2, degenerate ? Bt : q3, degenerate ? Bw : q4};
}

template <int DIR>
MHD_HD_INLINE bool hlld_star_of(const Side& L, const Side& R, double ch, double g, double* F) {
    if (!usable(L) || !usable(R)) return false;
    double unL, unR, utL, utR, uwL, uwR, BnL, BnR, BtL, BtR, BwL, BwR;
    rotate_side<DIR>(L, unL, utL, uwL, BnL, BtL, BwL);
    rotate_side<DIR>(R, unR, utR, uwR, BnR, BtR, BwR);
    const double rhoL = L.v[RHO], rhoR = R.v[RHO];
    double cfL, cfR;
    fast_speeds<DIR>(L, R, g, cfL, cfR);
    const double SL = fmin(unL - cfL, unR - cfR);
    const double SR = fmax(unL + cfL, unR + cfR);
    const double denom_RL = SR - SL;
    if (fabs(denom_RL) < 1.0e-14) return false;
    const double ptL = L.p() + 0.5 * (BnL * BnL + BtL * BtL + BwL * BwL);
    const double ptR = R.p() + 0.5 * (BnR * BnR + BtR * BtR + BwR * BwR);
    double SM, rhoLs, rhoRs;
    Recip rs;
    if (!contact(rhoL, unL, ptL, SL, rhoR, unR, ptR, SR, SM, rhoLs, rhoRs, rs)) return false;
    if (SL >= 0.0) { flux_of<DIR>(L, ch, F); return true; }
    if (SR <= 0.0) { flux_of<DIR>(R, ch, F); return true; }
    const double ptstar = ptL + rhoL * (SL - unL) * (SM - unL);
    const double psiM = 0.5 * (L.v[PSI] + R.v[PSI]) - 0.5 * ch * (BnR - BnL);
    // the owning side (S_M >= 0: left)
    const bool left = SM >= 0.0;
    const double S = left ? SL : SR, rho = left ? rhoL : rhoR, un = left ? unL : unR, ut = left ? utL : utR;
    const double uw = left ? uwL : uwR, Bn = left ? BnL : BnR, Bt = left ? BtL : BtR, Bw = left ? BwL : BwR;
    const double pt = left ? ptL : ptR, rhos = left ? rhoLs : rhoRs;
    Side O;
#pragma unroll
    for (int k = 0; k < 13; ++k) O.v[k] = left ? L.v[k] : R.v[k];
    bool bad = out_rad(rhos);
    Star s = star_group(rho, un, ut, uw, Bn, Bt, Bw, S, SM, bad);
    double sq = root(rhos);
    const double aBn = fabs(Bn);
    double vA = quot_pos(aBn, recip(sq));
    const double BdotU = Bn * un + Bt * ut + Bw * uw;
    double BdotUs = Bn * SM + s.Bt * s.ut + s.Bw * s.uw;
    double nE = O.v[EN] * (S - un) - pt * un + ptstar * SM + Bn * (BdotUs - BdotU);
    double Es = quot(nE, rs);
    bad = bad | out_num(aBn) | out_den(sq) | out_num(nE) | out_den(rs.b);
    if (bad) {
        s = star_native(rho, un, ut, uw, Bn, Bt, Bw, S, SM);
        sq = sqrt(rhos);
        vA = aBn / sq;
        BdotUs = Bn * SM + s.Bt * s.ut + s.Bw * s.uw;
        nE = O.v[EN] * (S - un) - pt * un + ptstar * SM + Bn * (BdotUs - BdotU);
        Es = nE / rs.b;
    }
    double Us[NV], Fs[NV];
    build_star<DIR>(rhos, SM, s.ut, s.uw, Bn, s.Bt, s.Bw, Es, psiM, Us);
    flux_of<DIR>(O, ch, Fs);
    const double Ss = left ? SM - vA : SM + vA;
#pragma unroll
    for (int k = 0; k < NV; ++k) F[k] = Fs[k] + S * (Us[k] - O.v[k]);
    if (left ? Ss >= 0.0 : Ss <= 0.0) return true;
    // the double-star state needs the other side's star state as well
    const double rhoso = left ? rhoRs : rhoLs;
    const double oS = left ? SR : SL, orho = left ? rhoR : rhoL, oun = left ? unR : unL, out = left ? utR : utL;
    const double ouw = left ? uwR : uwL, oBn = left ? BnR : BnL, oBt = left ? BtR : BtL, oBw = left ? BwR : BwL;
    bool bado = out_rad(rhoso);
    Star o = star_group(orho, oun, out, ouw, oBn, oBt, oBw, oS, SM, bado);
    double sqo = root(rhoso);
    double denom2 = left ? sq + sqo : sqo + sq;
    double inv_d2 = recip(denom2).y;
    bado = bado | out_den(denom2);
    if (bado) {
        o = star_native(orho, oun, out, ouw, oBn, oBt, oBw, oS, SM);
        sqo = sqrt(rhoso);
        denom2 = left ? sq + sqo : sqo + sq;
        inv_d2 = 1.0 / denom2;
    }
    const double signBn = (BnL >= 0.0) ? 1.0 : -1.0;
    const double sqL = left ? sq : sqo, sqR = left ? sqo : sq;
    const double utLs = left ? s.ut : o.ut, uwLs = left ? s.uw : o.uw, BtLs = left ? s.Bt : o.Bt, BwLs = left ? s.Bw : o.Bw;
    const double utRs = left ? o.ut : s.ut, uwRs = left ? o.uw : s.uw, BtRs = left ? o.Bt : s.Bt, BwRs = left ? o.Bw : s.Bw;
    double utss = s.ut, uwss = s.uw, Btss = s.Bt, Bwss = s.Bw, Ess = Es;
    if (!(fabs(denom2) < 1.0e-14)) {
        utss = (sqL * utLs + sqR * utRs + signBn * (BtRs - BtLs)) * inv_d2;
        uwss = (sqL * uwLs + sqR * uwRs + signBn * (BwRs - BwLs)) * inv_d2;
        Btss = (sqL * BtRs + sqR * BtLs + signBn * sqL * sqR * (utRs - utLs)) * inv_d2;
        Bwss = (sqL * BwRs + sqR * BwLs + signBn * sqL * sqR * (uwRs - uwLs)) * inv_d2;
        const double BdotUss = Bn * SM + Btss * utss + Bwss * uwss;
        Ess = left ? Es - sq * signBn * (BdotUss - BdotUs) : Es + sq * signBn * (BdotUss - BdotUs);
    }
    double Uss[NV];
    build_star<DIR>(rhos, SM, utss, uwss, Bn, Btss, Bwss, Ess, psiM, Uss);
#pragma unroll
    for (int k = 0; k < NV; ++k) F[k] = F[k] + Ss * (Uss[k] - Us[k]);
    return true;
}

template <int DIR>
MHD_HD_INLINE void force_of(const Side& L, const Side& R, double ch, double g, double* F) {
    double FL[NV], FR[NV];
    flux_of<DIR>(L, ch, FL);
    flux_of<DIR>(R, ch, FR);
    if (!usable(L) || !usable(R)) {
#pragma unroll
        for (int k = 0; k < NV; ++k) F[k] = 0.5 * (FL[k] + FR[k]);
        return;
    }
    double cfL, cfR;
    fast_speeds<DIR>(L, R, g, cfL, cfR);
    const double unL = L.vel(DIR), unR = R.vel(DIR);
    const double alpha = fmax(fmax(fabs(unL) + cfL, fabs(unR) + cfR), ch);
    if (alpha < 1.0e-14) {
#pragma unroll
        for (int k = 0; k < NV; ++k) F[k] = 0.5 * (FL[k] + FR[k]);
        return;
    }
    double ia;
    reciprocals<1>(&alpha, &ia);
    double Flf[NV];
    Side S;
    const double ha = 0.5 * alpha, hia = 0.5 * ia;
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        Flf[k] = 0.5 * (FL[k] + FR[k]) - ha * (R.v[k] - L.v[k]);
        S.v[k] = 0.5 * (L.v[k] + R.v[k]) - hia * (FR[k] - FL[k]);
    }
    reciprocals<1>(S.v, &S.v[13]);
    prim_of(S.v, S.v[13], g, S.v[9], S.v[10], S.v[11], S.v[12]);
    if (!usable(S)) {
#pragma unroll
        for (int k = 0; k < NV; ++k) F[k] = Flf[k];
        return;
    }
    flux_of<DIR>(S, ch, FR);
#pragma unroll
    for (int k = 0; k < NV; ++k) F[k] = 0.5 * (Flf[k] + FR[k]);
}

template <int DIR, int SOLVER>
MHD_HD_INLINE void riemann_of(const Side& L, const Side& R, double ch, double g, double* F) {
    if (SOLVER == HLL) { hll_of<DIR>(L, R, ch, g, F); return; }
    bool ok = true;
    if (SOLVER == HLLC) ok = hllc_star_of<DIR>(L, R, ch, g, F);
    else if (SOLVER == HLLD) ok = hlld_star_of<DIR>(L, R, ch, g, F);
    else force_of<DIR>(L, R, ch, g, F);
    bool overwrite = true;
    if (ok && (!finite_d(F[RHO]) || !finite_d(F[EN]) || !finite_d(F[BX]) || !finite_d(F[PSI]))) overwrite = false;
    if (!ok || !overwrite) hll_of<DIR>(L, R, ch, g, F);
    if (!ok && (!finite_d(F[RHO]) || !finite_d(F[EN]) || !finite_d(F[BX]) || !finite_d(F[PSI]))) overwrite = false;
    if (overwrite) glm_overwrite<DIR>(F, L.v, R.v, ch);
}

// rho and p above their floors, every value finite
MHD_HD_INLINE bool physical(const double* V, double u, double v, double w, double p) {
    return finite_d(V[RHO]) && V[RHO] > kRhoFloor && finite_d(p) && p > kPFloor && finite_d(u) && finite_d(v) &&
           finite_d(w) && finite_d(V[BX]) && finite_d(V[BY]) && finite_d(V[BZ]) && finite_d(V[PSI]);
}

// The same for a state whose pressure p follows from its conserved values: p is
// finite only if rho, u, v, w, B (and E) are, so four tests stand for nine.
MHD_HD_INLINE bool physical_p(const double* V, double p, double floor_p) {
    return (V[RHO] > kRhoFloor) & finite_d(p) & (p > floor_p) & finite_d(V[PSI]);
}

// The limited slopes of all fields.
template <int LIMITER>
MHD_HD_INLINE void slopes(const double* Wm, const double* Wc, const double* Wp, double* s) {
    if (LIMITER != VANLEER) {
#pragma unroll
        for (int k = 0; k < NV; ++k) s[k] = minmod(Wc[k] - Wm[k], Wp[k] - Wc[k]);
        return;
    }
    bool bad = false;
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        const double a = Wc[k] - Wm[k], b = Wp[k] - Wc[k];
        const bool flat = a * b <= 0.0;
        const double n = 2.0 * a * b, d = a + b;  // a b > 0: n > 0 and d has the slopes' sign
        const Recip r = recip(d);
        s[k] = flat ? 0.0 : quot_pos(n, r);
        bad = bad | (!flat & (out_den(d) | xd_out<-960, 540>(n)));
    }
    if (bad) {
#pragma unroll
        for (int k = 0; k < NV; ++k) s[k] = vanleer(Wc[k] - Wm[k], Wp[k] - Wc[k]);
    }
}

template <int DIR, int LIMITER>
MHD_HD_INLINE void reconstruct_of(const double* Wm, const double* Wc, const double* Wp, double dtd, double ch, double g,
                                  Side& L, Side& R) {
    double Wl[NV], Wr[NV];
    {
        double s[NV];
        slopes<LIMITER>(Wm, Wc, Wp, s);
#pragma unroll
        for (int k = 0; k < NV; ++k) {
            Wl[k] = Wc[k] - 0.5 * s[k];
            Wr[k] = Wc[k] + 0.5 * s[k];
        }
    }
    // p / (g - 1) and 1 / rho of both
    const double gm1 = g - 1.0;
    const Recip rg = recip(gm1);
    double el = quot(Wl[PP], rg), er = quot(Wr[PP], rg), irl = recip(Wl[RHO]).y, irr = recip(Wr[RHO]).y;
    if (out_den(gm1) | out_num(Wl[PP]) | out_num(Wr[PP]) | out_den(Wl[RHO]) | out_den(Wr[RHO])) {
        el = Wl[PP] / gm1;
        er = Wr[PP] / gm1;
        irl = 1.0 / Wl[RHO];
        irr = 1.0 / Wr[RHO];
    }
    double Ul[NV], Ur[NV], Fl[NV], Fr[NV];
    double ul, vl, wl, pl, ur, vr, wr, pr;
    auto cons = [](const double* W, double ep, double* U) {  // p2c, with p / (g - 1) given
        const double Bmag2 = W[BX] * W[BX] + W[BY] * W[BY] + W[BZ] * W[BZ];
        const double ke = 0.5 * W[RHO] * (W[PU] * W[PU] + W[PV] * W[PV] + W[PW] * W[PW]);
        U[RHO] = W[RHO]; U[MX] = W[RHO] * W[PU]; U[MY] = W[RHO] * W[PV]; U[MZ] = W[RHO] * W[PW];
        U[BX] = W[BX]; U[BY] = W[BY]; U[BZ] = W[BZ]; U[EN] = ep + ke + 0.5 * Bmag2; U[PSI] = W[PSI];
    };
    cons(Wl, el, Ul);
    cons(Wr, er, Ur);
    prim_of(Ul, irl, g, ul, vl, wl, pl);
    prim_of(Ur, irr, g, ur, vr, wr, pr);
    // A face state with a finite recomputed pressure has every value but psi
    // finite (an infinity or NaN in any would reach it): physical at once.  The
    // others take the full test, which fails the face state over to the centre's.
    if (!((Wl[PP] > kPFloor) & physical_p(Wl, pl, -HUGE_VAL) & (Wr[PP] > kPFloor) & physical_p(Wr, pr, -HUGE_VAL))) {
        const bool okl = physical(Wl, Wl[PU], Wl[PV], Wl[PW], Wl[PP]), okr = physical(Wr, Wr[PU], Wr[PV], Wr[PW], Wr[PP]);
#pragma unroll
        for (int k = 0; k < NV; ++k) {
            if (!okl) Wl[k] = Wc[k];
            if (!okr) Wr[k] = Wc[k];
        }
        irl = 1.0 / Wl[RHO];
        irr = 1.0 / Wr[RHO];
        cons(Wl, Wl[PP] / gm1, Ul);
        cons(Wr, Wr[PP] / gm1, Ur);
        prim_of(Ul, irl, g, ul, vl, wl, pl);
        prim_of(Ur, irr, g, ur, vr, wr, pr);
    }
    flux_of<DIR>(Ul, ul, vl, wl, pl, ch, Fl);
    flux_of<DIR>(Ur, ur, vr, wr, pr, ch, Fr);
    const double s = 0.5 * dtd;
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        const double d = s * (Fr[k] - Fl[k]);
        L.v[k] = Ul[k] - d;
        R.v[k] = Ur[k] - d;
    }
    const double rho2[2] = {L.v[RHO], R.v[RHO]};
    double ir2[2];
    reciprocals<2>(rho2, ir2);
    L.v[13] = ir2[0];
    R.v[13] = ir2[1];
    prim_of(L.v, L.v[13], g, L.v[9], L.v[10], L.v[11], L.v[12]);
    prim_of(R.v, R.v[13], g, R.v[9], R.v[10], R.v[11], R.v[12]);
    if (!physical_p(L.v, L.v[12], kPFloor)) {
#pragma unroll
        for (int k = 0; k < NV; ++k) L.v[k] = Ul[k];
        L.v[9] = ul; L.v[10] = vl; L.v[11] = wl; L.v[12] = pl; L.v[13] = irl;
    }
    if (!physical_p(R.v, R.v[12], kPFloor)) {
#pragma unroll
        for (int k = 0; k < NV; ++k) R.v[k] = Ur[k];
        R.v[9] = ur; R.v[10] = vr; R.v[11] = wr; R.v[12] = pr; R.v[13] = irr;
    }
}

// cell_speed of a cell
MHD_HD_INLINE double cell_speed_of(const double* U, double g, double ch) {
    double W[NV];
    double ir;
    reciprocals<1>(U, &ir);
    prim_of(U, ir, g, W[PU], W[PV], W[PW], W[PP]);
    const double rho = U[RHO], p = W[PP];
    if (!finite_d(rho) || !finite_d(p) || rho <= 0.0 || p <= 0.0) return -1.0;
    const double gp = g * p, B2 = U[BX] * U[BX] + U[BY] * U[BY] + U[BZ] * U[BZ];
    bool bad = false;
    double cx = fast_group(gp, B2, U[BX], rho, ir, bad), cy = fast_group(gp, B2, U[BY], rho, ir, bad);
    if (bad) {
        cx = fast_native(gp, B2, U[BX], rho);
        cy = fast_native(gp, B2, U[BY], rho);
    }
    const double sx = fmax(fabs(W[PU]) + cx, ch), sy = fmax(fabs(W[PV]) + cy, ch);
    if (finite_d(sx) && finite_d(sy)) return (sx < sy) ? sy : sx;
    return -1.0;
}

// cell_speed folded into a running maximum acc, skipping the fast speeds of a
// cell whose speed provably stays under the floor ch: cell_speed returns
// exactly ch for such a cell (both directional speeds are floored by it), so
// the maximum is the same bit for bit.  The test needs no division: with
// r = rho, r e = r E - (|m|^2 + r |B|^2) / 2 (rho times the internal energy)
// and X = g (g - 1) r e + r |B|^2 = r^2 (a^2 + b^2), the speed is under
// max(|u|, |v|) + sqrt(a^2 + b^2) = (max(|m_x|, |m_y|) + sqrt(X)) / r, as
// c_f^2 = (s + sqrt(s^2 - 4 a^2 b_n^2)) / 2 <= s = a^2 + b^2; and without its root:
// sqrt(X) < t for t = ch r (1 - 1e-12) - max(|m_x|, |m_y|) > 0 when X < t^2 (1 - 1e-12).
// Margins: the internal energy above 1e-6 of |E| (c2p's pressure then is surely
// positive) and the bound 1e-12 under ch (far above the rounding of either
// form).  Non-physical and non-finite cells take cell_speed.
MHD_HD_INLINE void fold_cell_speed(const double* U, double g, double ch, double& acc) {
    const double r = U[RHO];
    const double m2 = U[MX] * U[MX] + U[MY] * U[MY] + U[MZ] * U[MZ];
    const double B2r = (U[BX] * U[BX] + U[BY] * U[BY] + U[BZ] * U[BZ]) * r;
    const double re = U[EN] * r - 0.5 * (m2 + B2r);
    const double X = g * (g - 1.0) * re + B2r;
    const double t = ch * r * (1.0 - 1.0e-12) - fmax(fabs(U[MX]), fabs(U[MY]));
    if (r > 0.0 && re > 1.0e-6 * fabs(U[EN]) * r && t > 0.0 && X < t * t * (1.0 - 1.0e-12)) {
        acc = (acc < ch) ? ch : acc;
        return;
    }
    const double s = cell_speed_of(U, g, ch);
    acc = (acc < s) ? s : acc;
}

}  // namespace exact
}  // namespace mhd
