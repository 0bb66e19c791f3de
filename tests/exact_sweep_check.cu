// Host-side comparison, bit for bit, of the sweeps' FP64 physics
// (csrc/phys_exact_sweep.cuh) with the reference-ordered functions it
// rearranges (csrc/phys_exact.cuh): reconstruction, the four solvers through the
// dispatcher and the CFL speed, in both directions.  States: ordinary ones;
// zero and negative-zero components; slopes and values of 1e-200 to 1e200
// (outside the short quotients' range); identical sides; negative pressure and
// density, infinities and NaN.  Built and run by test_exact_div.py; no GPU.
#include <cstdio>
#include <cstring>
#include <random>

#include "phys_exact_sweep.cuh"

using namespace mhd;
using namespace mhd::exact;

static std::mt19937_64 rng(5);
static double uni(double a, double b) { return std::uniform_real_distribution<double>(a, b)(rng); }
static int failures = 0;
static long long compared = 0;

static bool same(double a, double b) { return (std::isnan(a) && std::isnan(b)) || std::memcmp(&a, &b, 8) == 0; }
static void check(const char* what, int kind, const double* a, const double* b, int n) {
    for (int k = 0; k < n; ++k, ++compared)
        if (!same(a[k], b[k]) && failures++ < 20) std::printf("FAIL %s (kind %d, %d): %.17g against %.17g\n", what, kind, k, a[k], b[k]);
}

static void prim(int kind, double* W) {
    W[RHO] = uni(0.1, 3.0); W[PU] = uni(-2, 2); W[PV] = uni(-2, 2); W[PW] = uni(-1, 1);
    W[BX] = uni(-1.5, 1.5); W[BY] = uni(-1.5, 1.5); W[BZ] = uni(-1, 1); W[PP] = uni(0.02, 3.0); W[PSI] = uni(-0.2, 0.2);
    if (kind == 1) { W[PW] = 0.0; W[BZ] = -0.0; W[PSI] = 0.0; }
    if (kind == 2) { W[BX] = 0.0; W[BY] = rng() & 1 ? 0.0 : -0.0; W[BZ] = 0.0; W[PU] = -0.0; }
    if (kind == 3) for (int k : {(int)PV, (int)PW, (int)BY, (int)PSI}) W[k] *= std::pow(10.0, uni(-200, -60));
    if (kind == 4) for (int k : {(int)PU, (int)PP, (int)BZ}) W[k] *= std::pow(10.0, uni(20, 140));
    if (kind == 5) { W[RHO] *= std::pow(10.0, uni(-25, 25)); W[PP] *= std::pow(10.0, uni(-25, 25)); }
    if (kind == 6) { const double bad[4] = {-1.0, INFINITY, NAN, 0.0}; W[(int)(rng() % 9)] = bad[rng() % 4]; }
}

template <int DIR, int SOLVER>
static void face(int kind, const double* UL, const double* UR, double ch, double g) {
    double a[NV], b[NV];
    Side L, R;
    side_of(UL, g, L);
    side_of(UR, g, R);
    riemann_of<DIR, SOLVER>(L, R, ch, g, a);
    riemann<DIR, SOLVER>(UL, UR, ch, g, b);
    check(SOLVER == HLL ? "hll" : SOLVER == HLLC ? "hllc" : SOLVER == HLLD ? "hlld" : "force", kind, a, b, NV);
}

template <int DIR, int LIM>
static void cell(int kind, const double* Wm, const double* Wc, const double* Wp, double dtd, double ch, double g) {
    Side L, R;
    double l[NV], r[NV], V[NV];
    reconstruct_of<DIR, LIM>(Wm, Wc, Wp, dtd, ch, g, L, R);
    reconstruct<DIR, LIM>(Wm, Wc, Wp, dtd, ch, g, l, r);
    check("L*", kind, L.v, l, NV);
    check("R*", kind, R.v, r, NV);
    for (const Side* S : {&L, &R}) {
        c2p(S->v, g, V);
        const double w[4] = {V[PU], V[PV], V[PW], V[PP]}, ir = 1.0 / S->v[RHO];
        check("side primitives", kind, S->v + 9, w, 4);
        check("side 1/rho", kind, S->v + 13, &ir, 1);
    }
}

int main() {
    for (int t = 0; t < 120000; ++t) {
        const int kind = t % 8;
        const double g = (t / 8) % 3 == 0 ? 5.0 / 3.0 : (t / 8) % 3 == 1 ? 2.0 : 1.4;
        double Wm[NV], Wc[NV], Wp[NV], UL[NV], UR[NV];
        prim(kind, Wm);
        prim(kind, Wc);
        prim(kind, Wp);
        if (t % 3 == 0)  // close states: small slopes, weak waves
            for (int k = 0; k < NV; ++k) {
                const double e = std::pow(10.0, uni(-17, -1));
                Wm[k] = Wc[k] * (1 + e * uni(-1, 1));
                Wp[k] = Wc[k] * (1 + e * uni(-1, 1));
            }
        if (kind == 7)
            for (int k = 0; k < NV; ++k) Wm[k] = Wp[k] = Wc[k];
        const double dtd = uni(0.01, 0.6), ch = t % 29 == 0 ? 0.0 : uni(0.1, 4.0);
        cell<0, VANLEER>(kind, Wm, Wc, Wp, dtd, ch, g);
        cell<1, VANLEER>(kind, Wm, Wc, Wp, dtd, ch, g);
        cell<0, MINMOD>(kind, Wm, Wc, Wp, dtd, ch, g);
        cell<1, MINMOD>(kind, Wm, Wc, Wp, dtd, ch, g);
        p2c(Wm, g, UL);
        p2c(Wp, g, UR);
        if (t % 5 == 0) { UL[MX] += 8.0 * UL[RHO]; UR[MX] += 8.0 * UR[RHO]; UL[EN] += 200.0; UR[EN] += 200.0; }
        if (t % 7 == 0) UR[EN] = -std::fabs(UR[EN]);
        face<0, HLL>(kind, UL, UR, ch, g);
        face<1, HLL>(kind, UL, UR, ch, g);
        face<0, HLLC>(kind, UL, UR, ch, g);
        face<1, HLLC>(kind, UL, UR, ch, g);
        face<0, HLLD>(kind, UL, UR, ch, g);
        face<1, HLLD>(kind, UL, UR, ch, g);
        face<0, FORCE>(kind, UL, UR, ch, g);
        face<1, FORCE>(kind, UL, UR, ch, g);
        const double a = cell_speed_of(UL, g, ch), b = cell_speed(UL, g, ch);
        check("cell speed", kind, &a, &b, 1);
        for (double floor_ch : {0.5 * b, b, 1.0000001 * b, 3.0 * b}) {  // the fold from a floor under, at and over the speed
            if (!(floor_ch > 0.0)) continue;
            const double s = cell_speed(UL, g, floor_ch);
            double f = 0.0, want = 0.0 < s ? s : 0.0;
            fold_cell_speed(UL, g, floor_ch, f);
            check("fold", kind, &f, &want, 1);
        }
    }
    std::printf("%lld values, %d failures\n", compared, failures);
    return failures ? 1 : 0;
}
