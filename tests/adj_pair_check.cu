// Host-side check of the paired adjoint functions (csrc/adj_pair.cuh) against
// the general ones they restate (csrc/adj_physics.cuh), for random states and
// cotangents: the HLL face with its reverse (every wave region, unusable
// states, c_h = 0) and the reconstruction with its reverse (both limiters,
// slopes that turn a face state non-physical, half steps that do).  The two
// evaluate the same formulas in another order, so each result may differ by
// rounding: 200 ulp of the sum of the absolute terms (under 100 operations).
// Built and run by test_adjoint_pair.py; no GPU.
#include <cmath>
#include <cstdio>
#include <limits>
#include <random>

#include "adj_pair.cuh"

using namespace mhd;
using namespace mhd::adj;

static std::mt19937_64 rng(7);
static double uni(double a, double b) { return std::uniform_real_distribution<double>(a, b)(rng); }
static int failures = 0, taken[8];

template <typename R>
static void close(const char* what, R got, R want, double scale) {
    const double tol = 200.0 * std::numeric_limits<R>::epsilon() * (1.0 + scale);
    const bool same_nan = std::isnan((double)got) && std::isnan((double)want);
    if (!same_nan && !(std::fabs((double)got - (double)want) <= tol) && failures++ < 20)
        std::printf("FAIL %s: %.17g against %.17g (scale %.3g)\n", what, (double)got, (double)want, scale);
}

template <typename R>
static void prim(R* W, double wild) {
    W[RHO] = (R)uni(0.3, 2.0); W[PU] = (R)uni(-wild, wild); W[PV] = (R)uni(-1, 1); W[PW] = (R)uni(-0.5, 0.5);
    W[BX] = (R)uni(-1, 1); W[BY] = (R)uni(-1, 1); W[BZ] = (R)uni(-0.5, 0.5); W[PP] = (R)uni(0.2, 2.0);
    W[PSI] = (R)uni(-0.1, 0.1);
}

template <typename R>
static void faces(const R g) {
    for (int t = 0; t < 4000; ++t) {
        R WL[NV], WR[NV], UL[NV], UR[NV], d[NV], lF[NV], lL[NV], lR[NV], f[NV];
        prim(WL, 1.0);
        prim(WR, 1.0);
        p2c(WL, g, UL);
        p2c(WR, g, UR);
        if (t % 11 == 3) UL[EN] = R(-1);          // negative pressure: the mean flux
        if (t % 11 == 5) UR[EN] = R(-0.5);
        if (t % 13 == 4) WR[RHO] = UR[RHO] = WL[RHO];
        const R ch = t % 17 == 6 ? R(0) : (R)uni(0.05, 3.0), dtd = (R)uni(0.05, 0.4);
        if (t % 17 == 6) { UL[MX] += R(4) * UL[RHO]; UR[MX] += R(4) * UR[RHO]; UL[EN] += R(20); UR[EN] += R(20); }
        double mag = 0.0;
        for (int k = 0; k < NV; ++k) {
            d[k] = (R)uni(-1, 1);
            lF[k] = dtd * d[k];
            lL[k] = lR[k] = R(0);
            mag += std::fabs((double)UL[k]) + std::fabs((double)UR[k]);
        }
        mag = mag * mag * (1.0 + (double)ch * ch) * 10.0;
        R lch0 = R(0), ld0 = R(0), lch1 = R(0), ld1 = R(0);
        hll(UL, UR, ch, g, f);
        hll_adj(UL, UR, ch, g, lF, lL, lR, lch0);
        for (int k = 0; k < NV; ++k) ld0 += f[k] * d[k];
        Pr<R> U2[NV], W2[NV], ir, lU[NV];
        for (int k = 0; k < NV; ++k) U2[k] = {UL[k], UR[k]};
        c2p2(U2, g - R(1), W2, ir);
        hll_pair(U2, W2, ir, ch, g, g - R(1), g / (g - R(1)), dtd, d, lU, ld1, lch1);
        for (int k = 0; k < NV; ++k) {
            close("hll lUL", lU[k].x, lL[k], mag);
            close("hll lUR", lU[k].y, lR[k], mag);
        }
        close("hll ldtd", ld1, ld0, mag);
        close("hll lch", lch1, lch0, mag);
    }
}

template <typename R, int LIM>
static void cells(const R g) {
    for (int t = 0; t < 4000; ++t) {
        R Wm[NV], Wc[NV], Wp[NV], L0[NV], R0[NV], lL[NV], lR[NV];
        prim(Wm, 1.0);
        prim(Wc, 1.0);
        prim(Wp, 1.0);
        if (t % 3 == 0)  // monotone data: slopes that do not vanish
            for (int k = 0; k < NV; ++k) { Wp[k] = Wc[k] + R(0.1) * (R)uni(0, 1); Wm[k] = Wc[k] - R(0.1) * (R)uni(0, 1); }
        if (t % 7 == 2) { Wc[PP] = R(1e-13); Wm[PP] = R(2e-13); Wp[PP] = R(5e-14); }  // under the floor: fallbacks
        if (t % 9 == 4) { Wc[PU] = R(3); Wm[PU] = R(-3); Wp[PU] = R(30); }             // half steps that go negative
        const R dtd = t % 9 == 4 ? R(3) : (R)uni(0.05, 0.4), ch = (R)uni(0.5, 2.0);
        double mag = 0.0;
        for (int k = 0; k < NV; ++k) {
            lL[k] = (R)uni(-1, 1);
            lR[k] = (R)uni(-1, 1);
            mag += std::fabs((double)Wm[k]) + std::fabs((double)Wc[k]) + std::fabs((double)Wp[k]);
        }
        mag = 100.0 * mag * mag * mag;
        recon<LIM>(Wm, Wc, Wp, dtd, ch, g, L0, R0);
        R a0[NV], b0[NV], c0[NV], a1[NV], b1[NV], c1[NV], ld0 = R(0), lc0 = R(0), ld1 = R(0), lc1 = R(0);
        zero(a0); zero(b0); zero(c0); zero(a1); zero(b1); zero(c1);
        Recon<R> rc;
        Pr<R> S[NV], V[NV], ir, lS[NV];
        const R gm1 = g - R(1), igm1 = R(1) / gm1;
        recon2<LIM>(Wm, Wc, Wp, dtd, ch, gm1, igm1, rc, S, V, ir);
        if (rc.okLs != rc.okRs || !rc.okLs) taken[2]++;
        if (!(rc.okL && rc.okR)) taken[1]++;
        taken[0]++;
        for (int k = 0; k < NV; ++k) lS[k] = {lL[k], lR[k]};
        // a state within rounding of a floor may take either side of it
        R W0[NV];
        bool edge = false;
        for (const R* s : {L0, R0}) {
            c2p(s, g, W0);
            edge = edge || std::fabs((double)W0[PP]) < 1e-4 * mag * std::numeric_limits<R>::epsilon();
        }
        if (edge) { taken[3]++; continue; }
        recon_adj<LIM>(Wm, Wc, Wp, dtd, ch, g, lL, lR, a0, b0, c0, ld0, lc0);
        recon_adj2<LIM>(Wm, Wc, Wp, rc, dtd, ch, igm1, g * igm1, lS, a1, b1, c1, ld1, lc1);
        for (int k = 0; k < NV; ++k) {
            close("recon L*", S[k].x, L0[k], mag);
            close("recon R*", S[k].y, R0[k], mag);
            close("recon lWm", a1[k], a0[k], mag);
            close("recon lWc", b1[k], b0[k], mag);
            close("recon lWp", c1[k], c0[k], mag);
        }
        close("recon ldtd", ld1, ld0, mag);
        close("recon lch", lc1, lc0, mag);
    }
}

int main() {
    for (double g : {5.0 / 3.0, 1.4, 2.0}) {
        faces<double>(g);
        faces<float>((float)g);
        cells<double, VANLEER>(g);
        cells<double, MINMOD>(g);
        cells<float, VANLEER>((float)g);
        cells<float, MINMOD>((float)g);
    }
    std::printf("%d cells, %d face fallbacks, %d half-step fallbacks, %d at a floor; %d failures\n", taken[0], taken[1],
                taken[2], taken[3], failures);
    return failures || taken[1] < 100 || taken[2] < 100 || taken[3] * 5 > taken[0] ? 1 : 0;
}
