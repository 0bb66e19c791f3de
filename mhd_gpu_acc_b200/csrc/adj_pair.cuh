// adj_pair.cuh -- the adjoint's local functions on pairs of states.
//
// A cell's MUSCL-Hancock predictor treats its left-face and right-face states
// identically, and a face its left and right sides, forwards and backwards.  So
// both are carried as pairs (.x = left, .y = right) and advanced together: in
// FP32 one sm_100 paired instruction serves both (one issue slot instead of
// two), in FP64 the two chains interleave.  The formulas are those of
// adj_physics.cuh (its flux, c2p, p2c, fast, hll and recon with their *_adj),
// with the values that forward and reverse share computed once.
#pragma once

#include "adj_physics.cuh"

namespace mhd {
namespace adj {

template <typename R>
struct Pr {
    R x, y;
};

template <typename R>
ADJ_HD Pr<R> dup(R a) { return Pr<R>{a, a}; }

#ifdef __CUDA_ARCH__
__device__ __forceinline__ float2 f2(const Pr<float>& a) { return make_float2(a.x, a.y); }
__device__ __forceinline__ Pr<float> pr(float2 a) { return Pr<float>{a.x, a.y}; }
__device__ __forceinline__ Pr<float> operator+(const Pr<float>& a, const Pr<float>& b) { return pr(__fadd2_rn(f2(a), f2(b))); }
__device__ __forceinline__ Pr<float> operator-(const Pr<float>& a, const Pr<float>& b) {
    return pr(__fadd2_rn(f2(a), make_float2(-b.x, -b.y)));
}
__device__ __forceinline__ Pr<float> operator*(const Pr<float>& a, const Pr<float>& b) { return pr(__fmul2_rn(f2(a), f2(b))); }
// a b + c
__device__ __forceinline__ Pr<float> mad(const Pr<float>& a, const Pr<float>& b, const Pr<float>& c) {
    return pr(__ffma2_rn(f2(a), f2(b), f2(c)));
}
// c - a b
__device__ __forceinline__ Pr<float> nmad(const Pr<float>& a, const Pr<float>& b, const Pr<float>& c) {
    return pr(__ffma2_rn(make_float2(-a.x, -a.y), f2(b), f2(c)));
}
#else
ADJ_HD Pr<float> operator+(const Pr<float>& a, const Pr<float>& b) { return {a.x + b.x, a.y + b.y}; }
ADJ_HD Pr<float> operator-(const Pr<float>& a, const Pr<float>& b) { return {a.x - b.x, a.y - b.y}; }
ADJ_HD Pr<float> operator*(const Pr<float>& a, const Pr<float>& b) { return {a.x * b.x, a.y * b.y}; }
ADJ_HD Pr<float> mad(const Pr<float>& a, const Pr<float>& b, const Pr<float>& c) { return {a.x * b.x + c.x, a.y * b.y + c.y}; }
ADJ_HD Pr<float> nmad(const Pr<float>& a, const Pr<float>& b, const Pr<float>& c) { return {c.x - a.x * b.x, c.y - a.y * b.y}; }
#endif
ADJ_HD Pr<double> operator+(const Pr<double>& a, const Pr<double>& b) { return {a.x + b.x, a.y + b.y}; }
ADJ_HD Pr<double> operator-(const Pr<double>& a, const Pr<double>& b) { return {a.x - b.x, a.y - b.y}; }
ADJ_HD Pr<double> operator*(const Pr<double>& a, const Pr<double>& b) { return {a.x * b.x, a.y * b.y}; }
ADJ_HD Pr<double> mad(const Pr<double>& a, const Pr<double>& b, const Pr<double>& c) { return {a.x * b.x + c.x, a.y * b.y + c.y}; }
ADJ_HD Pr<double> nmad(const Pr<double>& a, const Pr<double>& b, const Pr<double>& c) { return {c.x - a.x * b.x, c.y - a.y * b.y}; }

template <typename R>
ADJ_HD Pr<R> operator*(R a, const Pr<R>& b) { return dup(a) * b; }

template <typename R>
ADJ_HD Pr<R> rcp(const Pr<R>& a) { return {rcp(a.x), rcp(a.y)}; }

// W -> U of both
template <typename R>
ADJ_HD void p2c2(const Pr<R>* W, R igm1, Pr<R>* U) {
    const Pr<R> B2 = mad(W[BZ], W[BZ], mad(W[BY], W[BY], W[BX] * W[BX]));
    const Pr<R> v2 = mad(W[PW], W[PW], mad(W[PV], W[PV], W[PU] * W[PU]));
    const Pr<R> h = dup(R(0.5));
    U[RHO] = W[RHO]; U[MX] = W[RHO] * W[PU]; U[MY] = W[RHO] * W[PV]; U[MZ] = W[RHO] * W[PW];
    U[BX] = W[BX]; U[BY] = W[BY]; U[BZ] = W[BZ];
    U[EN] = mad(W[PP], dup(igm1), h * mad(W[RHO], v2, B2));
    U[PSI] = W[PSI];
}

// U -> W of both; ir = 1 / rho
template <typename R>
ADJ_HD void c2p2(const Pr<R>* U, R gm1, Pr<R>* W, Pr<R>& ir) {
    ir = rcp(U[RHO]);
    const Pr<R> u = U[MX] * ir, v = U[MY] * ir, w = U[MZ] * ir;
    const Pr<R> B2 = mad(U[BZ], U[BZ], mad(U[BY], U[BY], U[BX] * U[BX]));
    const Pr<R> mu = mad(U[MZ], w, mad(U[MY], v, U[MX] * u));
    W[RHO] = U[RHO]; W[PU] = u; W[PV] = v; W[PW] = w;
    W[BX] = U[BX]; W[BY] = U[BY]; W[BZ] = U[BZ];
    W[PP] = dup(gm1) * nmad(dup(R(0.5)), mu + B2, U[EN]);
    W[PSI] = U[PSI];
}

// GLM-MHD x-flux of both from consistent (U, W)
template <typename R>
ADJ_HD void flux2(const Pr<R>* U, const Pr<R>* W, R ch, Pr<R>* F) {
    const Pr<R> B2 = mad(W[BZ], W[BZ], mad(W[BY], W[BY], W[BX] * W[BX]));
    const Pr<R> pt = mad(dup(R(0.5)), B2, W[PP]);
    const Pr<R> uB = mad(W[PW], W[BZ], mad(W[PV], W[BY], W[PU] * W[BX]));
    F[0] = U[MX];
    F[1] = mad(U[MX], W[PU], nmad(W[BX], W[BX], pt));
    F[2] = nmad(W[BX], W[BY], U[MX] * W[PV]);
    F[3] = nmad(W[BX], W[BZ], U[MX] * W[PW]);
    F[4] = W[PSI];
    F[5] = nmad(W[BX], W[PV], W[BY] * W[PU]);
    F[6] = nmad(W[BX], W[PW], W[BZ] * W[PU]);
    F[7] = nmad(W[BX], uB, (U[EN] + pt) * W[PU]);
    F[8] = dup(ch * ch) * W[BX];
}

// lW += (dF/dW)^T lF; lch2 += (dF/dch) . lF
template <typename R>
ADJ_HD void flux_adj2(const Pr<R>* W, R ch, R gr /* g / (g - 1) */, const Pr<R>* lF, Pr<R>* lW, Pr<R>& lch2) {
    const Pr<R> r = W[RHO], u = W[PU], v = W[PV], w = W[PW], bx = W[BX], by = W[BY], bz = W[BZ];
    const Pr<R> B2 = mad(bz, bz, mad(by, by, bx * bx)), uB = mad(w, bz, mad(v, by, u * bx));
    const Pr<R> hv2 = dup(R(0.5)) * mad(w, w, mad(v, v, u * u));
    const Pr<R> H = mad(r, hv2, mad(W[PP], dup(gr), B2));  // E + p_tot
    const Pr<R> l7u = lF[7] * u;
    // the momentum flux (r u)(u, v, w): its cotangent with (u, v, w)
    const Pr<R> m = mad(lF[3], w, mad(lF[2], v, mad(lF[1], u, lF[0])));
    lW[RHO] = lW[RHO] + mad(m, u, l7u * hv2);
    const Pr<R> ru = r * u, l1 = mad(l7u, r, lF[1] * r);  // r (lF1 + lF7 u)
    lW[PU] = lW[PU] + mad(l1, u, mad(lF[5], by, mad(lF[6], bz, mad(m, r, lF[7] * nmad(bx, bx, H)))));
    const Pr<R> l7bx = lF[7] * bx;
    lW[PV] = lW[PV] + mad(mad(lF[7], v, lF[2]), ru, nmad(bx, lF[5], dup(R(0)) - l7bx * by));
    lW[PW] = lW[PW] + mad(mad(lF[7], w, lF[3]), ru, nmad(bx, lF[6], dup(R(0)) - l7bx * bz));
    const Pr<R> k1 = lF[1] - l7u;
    lW[BX] = lW[BX] + mad(lF[8], dup(ch * ch), nmad(k1, bx, nmad(lF[2], by, nmad(lF[3], bz, nmad(lF[5], v,
                      nmad(lF[6], w, dup(R(0)) - lF[7] * uB))))));
    const Pr<R> k2 = mad(dup(R(2)), l7u, lF[1]);
    lW[BY] = lW[BY] + mad(k2, by, nmad(bx, mad(lF[7], v, lF[2]), lF[5] * u));
    lW[BZ] = lW[BZ] + mad(k2, bz, nmad(bx, mad(lF[7], w, lF[3]), lF[6] * u));
    lW[PP] = lW[PP] + mad(l7u, dup(gr), lF[1]);
    lW[PSI] = lW[PSI] + lF[4];
    lch2 = mad(lF[8], dup(R(2) * ch) * bx, lch2);
}

template <typename R>
ADJ_HD void p2c_adj2(const Pr<R>* W, R igm1, const Pr<R>* lU, Pr<R>* lW) {
    const Pr<R> r = W[RHO], u = W[PU], v = W[PV], w = W[PW], lE = lU[EN];
    const Pr<R> hv2 = dup(R(0.5)) * mad(w, w, mad(v, v, u * u));
    lW[RHO] = lW[RHO] + mad(lE, hv2, mad(lU[MZ], w, mad(lU[MY], v, mad(lU[MX], u, lU[RHO]))));
    lW[PU] = mad(mad(lE, u, lU[MX]), r, lW[PU]);
    lW[PV] = mad(mad(lE, v, lU[MY]), r, lW[PV]);
    lW[PW] = mad(mad(lE, w, lU[MZ]), r, lW[PW]);
    lW[BX] = lW[BX] + mad(lE, W[BX], lU[BX]);
    lW[BY] = lW[BY] + mad(lE, W[BY], lU[BY]);
    lW[BZ] = lW[BZ] + mad(lE, W[BZ], lU[BZ]);
    lW[PP] = mad(lE, dup(igm1), lW[PP]);
    lW[PSI] = lW[PSI] + lU[PSI];
}

// lU += (dW/dU)^T lW, with ir = 1 / rho
template <typename R>
ADJ_HD void c2p_adj2(const Pr<R>* W, const Pr<R>& ir, R gm1, const Pr<R>* lW, Pr<R>* lU) {
    const Pr<R> u = W[PU], v = W[PV], w = W[PW], q = dup(gm1) * lW[PP];
    const Pr<R> hv2 = dup(R(0.5)) * mad(w, w, mad(v, v, u * u));
    const Pr<R> t = mad(lW[PW], w, mad(lW[PV], v, lW[PU] * u));
    lU[EN] = lU[EN] + q;
    lU[MX] = lU[MX] + nmad(q, u, lW[PU] * ir);
    lU[MY] = lU[MY] + nmad(q, v, lW[PV] * ir);
    lU[MZ] = lU[MZ] + nmad(q, w, lW[PW] * ir);
    lU[RHO] = lU[RHO] + mad(q, hv2, nmad(t, ir, lW[RHO]));
    lU[BX] = lU[BX] + nmad(q, W[BX], lW[BX]);
    lU[BY] = lU[BY] + nmad(q, W[BY], lW[BY]);
    lU[BZ] = lU[BZ] + nmad(q, W[BZ], lW[BZ]);
    lU[PSI] = lU[PSI] + lW[PSI];
}

// x * 0 is 0 for a finite x and NaN otherwise
template <typename R>
ADJ_HD void physical2(const Pr<R>* V, bool& okx, bool& oky) {
    Pr<R> z = V[0] * dup(R(0));
#pragma unroll
    for (int k = 1; k < NV; ++k) z = mad(V[k], dup(R(0)), z);
    okx = V[RHO].x > R(1e-12) && V[PP].x > R(1e-12) && z.x == R(0);
    oky = V[RHO].y > R(1e-12) && V[PP].y > R(1e-12) && z.y == R(0);
}

// The limited slope and i = 1 / (a + b) where the slopes agree in sign, else 0
// (van Leer's derivatives are 2 (b i)^2 and 2 (a i)^2).
template <int LIM, typename R>
ADJ_HD R slope(R a, R b, R& i) {
    if (LIM == VANLEER) {
        const bool ok = a * b > R(0);
        i = ok ? rcp(ok ? a + b : R(1)) : R(0);
        return R(2) * a * (b * i);
    }
    i = R(0);
    return limit<LIM>(a, b);
}

// What the forward reconstruction of one cell leaves for its reverse.
template <typename R>
struct Recon {
    Pr<R> W[NV];   // face states before the half step (after their fallback)
    R D[NV];       // F_R - F_L
    R i[NV];       // slope's reciprocals
    bool okL, okR;    // the face states were physical
    bool okLs, okRs;  // the advanced states were
};

// MUSCL-Hancock predictor of a cell: S = (L*, R*) conserved, V their primitives,
// ir their 1 / rho.
template <int LIM, typename R>
ADJ_HD void recon2(const R* Wm, const R* Wc, const R* Wp, R dtd, R ch, R gm1, R igm1, Recon<R>& rc, Pr<R>* S, Pr<R>* V,
                   Pr<R>& ir) {
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        const R s = slope<LIM>(Wc[k] - Wm[k], Wp[k] - Wc[k], rc.i[k]);
        rc.W[k] = {Wc[k] - R(0.5) * s, Wc[k] + R(0.5) * s};
    }
    physical2(rc.W, rc.okL, rc.okR);
    if (!(rc.okL && rc.okR)) {
#pragma unroll
        for (int k = 0; k < NV; ++k) {
            if (!rc.okL) rc.W[k].x = Wc[k];
            if (!rc.okR) rc.W[k].y = Wc[k];
        }
    }
    Pr<R> U[NV], F[NV];
    p2c2(rc.W, igm1, U);
    flux2(U, rc.W, ch, F);
    const R h = R(0.5) * dtd;
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        rc.D[k] = F[k].y - F[k].x;
        S[k] = nmad(dup(h), dup(rc.D[k]), U[k]);
    }
    c2p2(S, gm1, V, ir);
    physical2(V, rc.okLs, rc.okRs);
    if (!(rc.okLs && rc.okRs)) {
#pragma unroll
        for (int k = 0; k < NV; ++k) {
            if (!rc.okLs) { S[k].x = U[k].x; V[k].x = rc.W[k].x; }
            if (!rc.okRs) { S[k].y = U[k].y; V[k].y = rc.W[k].y; }
        }
        ir = rcp(S[RHO]);
    }
}

// Reverse of recon2 for the cotangent lS of S.  Wm, Wc, Wp: the forward inputs;
// adds to lWm, lWc, lWp and the scalar cotangents of dtd and ch.
template <int LIM, typename R>
ADJ_HD void recon_adj2(const R* Wm, const R* Wc, const R* Wp, const Recon<R>& rc, R dtd, R ch, R igm1, R gr,
                       const Pr<R>* lS, R* lWm, R* lWc, R* lWp, R& ldtd, R& lch) {
    const R h = R(0.5) * dtd;
    Pr<R> lF[NV], lW[NV];
    R lh = R(0);
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        const R lD = (rc.okLs ? -lS[k].x : R(0)) - (rc.okRs ? lS[k].y : R(0));
        lF[k] = {-h * lD, h * lD};
        lh += lD * rc.D[k];
        lW[k] = dup(R(0));
    }
    ldtd += R(0.5) * lh;
    Pr<R> lch2 = dup(R(0));
    p2c_adj2(rc.W, igm1, lS, lW);
    flux_adj2(rc.W, ch, gr, lF, lW, lch2);
    lch += lch2.x + lch2.y;
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        const R ls = (rc.okR ? R(0.5) * lW[k].y : R(0)) - (rc.okL ? R(0.5) * lW[k].x : R(0));
        const R a = Wc[k] - Wm[k], b = Wp[k] - Wc[k];
        R la, lb;
        if (LIM == VANLEER) {
            const R t = R(2) * ls, p = b * rc.i[k], q = a * rc.i[k];
            la = t * p * p;
            lb = t * q * q;
        } else {
            la = lb = R(0);
            limit_adj<LIM>(a, b, ls, la, lb);
        }
        lWm[k] -= la;
        lWc[k] += lW[k].x + lW[k].y + (la - lb);
        lWp[k] += lb;
    }
}

// sqrt(x) and 1 / sqrt(x) for x > 0 (0 and 0 otherwise)
template <typename R>
ADJ_HD void root(R x, R& s, R& is) {
    s = x > R(0) ? sqrt(x) : R(0);
    is = x > R(0) ? rcp(s) : R(0);
}

// HLL flux of a face and its reverse at once.  U, W, ir: both sides (x = left);
// d = the cotangent of F over dtd (F's own is dtd d).  lU (both sides) is
// written; adds dtd-cotangent sum F . d to ldtd and the c_h cotangent to lch.
// The intermediate wave is what a face takes whenever c_h > 0 and both states
// are usable; any other face takes the general functions.
template <typename R>
ADJ_HD void hll_pair(const Pr<R>* U, const Pr<R>* W, const Pr<R>& ir, R ch, R g, R gm1, R gr, R dtd, const R* d,
                     Pr<R>* lU, R& ldtd, R& lch) {
    Pr<R> F[NV];
    flux2(U, W, ch, F);
    const Pr<R> a2 = dup(g) * W[PP] * ir;
    const Pr<R> b2 = mad(W[BZ], W[BZ], mad(W[BY], W[BY], W[BX] * W[BX])) * ir;
    const Pr<R> bn2 = W[BX] * W[BX] * ir, s = a2 + b2;
    const Pr<R> disc = nmad(dup(R(4)) * a2, bn2, s * s);
    Pr<R> rt, irt, cf, icf;
    root(disc.x, rt.x, irt.x);
    root(disc.y, rt.y, irt.y);
    const Pr<R> q = dup(R(0.5)) * (s + rt);
    root(q.x, cf.x, icf.x);
    root(q.y, cf.y, icf.y);
    const Pr<R> a = W[PU] - cf, b = W[PU] + cf;
    const R m1 = fmin(a.x, a.y), m2 = fmax(b.x, b.y);
    const R SL = fmin(m1, -ch), SR = fmax(m2, ch), D = SR - SL;
    const bool usable = W[RHO].x > R(0) && W[PP].x > R(0) && W[RHO].y > R(0) && W[PP].y > R(0) &&
                        (W[RHO].x * R(0) + W[PP].x * R(0)) + (W[RHO].y * R(0) + W[PP].y * R(0)) == R(0);
    if (!(usable && SL < R(0) && SR > R(0) && D >= R(1e-14))) {
        R UL[NV], UR[NV], f[NV], lF[NV], lL[NV], lR[NV];
#pragma unroll
        for (int k = 0; k < NV; ++k) { UL[k] = U[k].x; UR[k] = U[k].y; lF[k] = dtd * d[k]; lL[k] = lR[k] = R(0); }
        hll(UL, UR, ch, g, f);
        hll_adj(UL, UR, ch, g, lF, lL, lR, lch);
#pragma unroll
        for (int k = 0; k < NV; ++k) { ldtd += f[k] * d[k]; lU[k] = {lL[k], lR[k]}; }
        return;
    }
    const R iD = rcp(D);
    const R wL = SR * iD, wR = -SL * iD, wU = SL * wL;  // F = wL F_L + wR F_R + wU (U_R - U_L)
    R s0 = R(0), sd = R(0), s2 = R(0);
    Pr<R> lF[NV], lW[NV];
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        s0 += d[k] * F[k].x;
        sd += d[k] * (F[k].y - F[k].x);
        s2 += d[k] * (U[k].y - U[k].x);
        const R l = dtd * d[k];
        lF[k] = {l * wL, l * wR};
        lU[k] = {-(l * wU), l * wU};
        lW[k] = dup(R(0));
    }
    ldtd += s0 + wR * sd + wU * s2;  // sum F . d
    // dF/dS_R = -S_L (S_L dU - dF) / D^2, dF/dS_L = S_R (S_R dU - dF) / D^2
    const R lSR = dtd * iD * (wR * (SL * s2 - sd)), lSL = dtd * iD * (wL * (SR * s2 - sd));
    // S_L = min(a_L, a_R, -c_h), S_R = max(b_L, b_R, c_h): to the selected argument
    const bool fl = m1 <= -ch, fr = m2 >= ch, ll = a.x <= a.y, rl = b.x >= b.y;
    const Pr<R> tl = {fl && ll ? lSL : R(0), fl && !ll ? lSL : R(0)};
    const Pr<R> tr = {fr && rl ? lSR : R(0), fr && !rl ? lSR : R(0)};
    if (!fl) lch -= lSL;
    if (!fr) lch += lSR;
    lW[PU] = tl + tr;
    // c_f = sqrt((s + sqrt(s^2 - 4 a2 bn2)) / 2)
    const Pr<R> lq = dup(R(0.25)) * (tr - tl) * icf;  // half of the cotangent of (s + rt) / 2
    const Pr<R> ld = dup(R(0.5)) * lq * irt;
    const Pr<R> ls = mad(ld, dup(R(2)) * s, lq);
    const Pr<R> la2 = nmad(dup(R(4)) * bn2, ld, ls), lbn2 = dup(R(-4)) * a2 * ld;
    lW[PP] = la2 * dup(g) * ir;
    lW[RHO] = dup(R(0)) - mad(la2, a2, mad(ls, b2, lbn2 * bn2)) * ir;
    const Pr<R> t2 = dup(R(2)) * ir;
    lW[BX] = (ls + lbn2) * t2 * W[BX];
    lW[BY] = ls * t2 * W[BY];
    lW[BZ] = ls * t2 * W[BZ];
    Pr<R> lch2 = dup(R(0));
    flux_adj2(W, ch, gr, lF, lW, lch2);
    lch += lch2.x + lch2.y;
    c2p_adj2(W, ir, gm1, lW, lU);
}

// The same for HLLD (with its fallbacks and the GLM overwrite): the general
// functions, the forward flux once.
template <typename R>
ADJ_HD void hlld_pair(const Pr<R>* U, R ch, R g, R dtd, const R* d, Pr<R>* lU, R& ldtd, R& lch) {
    R UL[NV], UR[NV], f[NV], lF[NV], lL[NV], lR[NV];
#pragma unroll
    for (int k = 0; k < NV; ++k) { UL[k] = U[k].x; UR[k] = U[k].y; lF[k] = dtd * d[k]; lL[k] = lR[k] = R(0); }
    const bool fine = hlld_face(UL, UR, ch, g, f);
    hlld_face_adj(UL, UR, ch, g, fine, lF, lL, lR, lch);
#pragma unroll
    for (int k = 0; k < NV; ++k) { ldtd += f[k] * d[k]; lU[k] = {lL[k], lR[k]}; }
}

}  // namespace adj
}  // namespace mhd
