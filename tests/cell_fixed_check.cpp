// Error of the fixed-point collision of a cell (csrc/cell_fixed.h) and of the same
// update in double, both against 113-bit arithmetic, over cells of the ranges the
// FP64 form meets.  Prints one line per kind of cell:
//   kind fixed_max fixed_rms double_max double_rms fluid_bits_equal fallbacks
// with errors relative to the cell's largest value (populations; P where it is larger).
//   usage: cell_fixed_check <cells per kind> <seed>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>

#include "cell_fixed.h"

#if defined(__aarch64__)
typedef long double quad;
#else
typedef __float128 quad;
#endif

static const int CX[19] = {0, -1, 0, 0, -1, -1, -1, -1, 0, 0, 1, 0, 0, 1, 1, 1, 1, 0, 0};
static const int CY[19] = {0, 0, -1, 0, -1, 1, 0, 0, -1, -1, 0, 1, 0, 1, -1, 0, 0, 1, 1};
static const int CZ[19] = {0, 0, 0, -1, 0, 0, -1, 1, -1, 1, 0, 0, 1, 0, 0, 1, -1, 1, -1};

// The update of k_collide.cu's collide_cell_fp64, in T (double: its operation
// order and fused multiply-adds; quad: exact enough to measure both).
static double mad(double a, double b, double c) { return std::fma(a, b, c); }
static quad mad(quad a, quad b, quad c) { return a * b + c; }

template <typename T>
static void collide(T (&f)[19], T omega, T B, const T (&up)[3], T (&F)[3]) {
    T s[9], d[9];
    for (int i = 1; i <= 9; ++i) {
        s[i - 1] = f[i] + f[i + 9];
        d[i - 1] = f[i + 9] - f[i];
    }
    const T rhoBar = f[0] + ((((s[0] + s[1]) + (s[2] + s[3])) + ((s[4] + s[5]) + (s[6] + s[7]))) + s[8]);
    T j[3] = {0, 0, 0};
    for (int k = 10; k < 19; ++k) {
        j[0] += CX[k] * d[k - 10];
        j[1] += CY[k] * d[k - 10];
        j[2] += CZ[k] * d[k - 10];
    }
    const T invRho = T(1) / (T(1) + rhoBar);
    const T jSqr = mad(j[2], j[2], mad(j[1], j[1], j[0] * j[0]));
    const T m15 = T(-1.5) * invRho;
    const T base = mad(m15, jSqr, rhoBar);
    const T rho = T(1) + rhoBar;
    T P[3];
    for (int a = 0; a < 3; ++a) P[a] = up[a] * rho;
    const T PSqr = mad(P[2], P[2], mad(P[1], P[1], P[0] * P[0]));
    const T dd = m15 * (jSqr - PSqr);
    const T alpha = mad(B, T(1) - omega, omega);
    const T om1B = omega * (T(1) - B);
    const T w0 = T(1) / T(3);
    const T g0 = f[0] - w0 * base;
    f[0] = mad(B, w0 * dd, mad(-om1B, g0, f[0]));
    T E[3] = {0, 0, 0};
    for (int k = 10; k < 19; ++k) {
        const int i = k - 9;
        const T t = k < 13 ? T(1) / T(18) : T(1) / T(36), t3 = T(3) * t;
        const T a45 = (T(4.5) * t) * invRho;
        const T cj = CX[k] * j[0] + CY[k] * j[1] + CZ[k] * j[2];
        const T C = mad(a45 * cj, cj, t * base);
        const T Lj = t3 * cj;
        const T gi = (f[i] - C) + Lj;
        const T gk = (f[k] - C) - Lj;
        const T cP = CX[k] * P[0] + CY[k] * P[1] + CZ[k] * P[2];
        const T m = cj - cP, p = cj + cP;
        const T Qd = mad(a45 * m, p, t * dd);
        const T L = t3 * m;
        const T e = d[i - 1] - t3 * p;
        f[i] = mad(B, (gk - Qd) + L, mad(-alpha, gi, f[i]));
        f[k] = mad(B, (gi - Qd) - L, mad(-alpha, gk, f[k]));
        E[0] += CX[k] * e;
        E[1] += CY[k] * e;
        E[2] += CZ[k] * e;
    }
    for (int a = 0; a < 3; ++a) F[a] = (B + B) * E[a];
}

// The update with a body force (k_collide.cu's collide_cell): BGK with the Guo force below
// full coverage, then the solid correction with the moments of the result, statement by
// statement (src/ibCompositeDynamics3D.hh:130-203).
template <typename T>
static void moments(const T (&f)[19], T& rb, T (&j)[3]) {
    rb = 0;
    j[0] = j[1] = j[2] = 0;
    for (int i = 0; i < 19; ++i) {
        rb += f[i];
        if (CX[i]) j[0] += CX[i] * f[i];
        if (CY[i]) j[1] += CY[i] * f[i];
        if (CZ[i]) j[2] += CZ[i] * f[i];
    }
}
template <typename T>
static T feq(int i, T rb, const T (&j)[3]) {
    const T t = i == 0 ? T(1) / T(3) : (i < 4 || (i > 9 && i < 13)) ? T(1) / T(18) : T(1) / T(36);
    const T cj = CX[i] * j[0] + CY[i] * j[1] + CZ[i] * j[2];
    const T jj = j[0] * j[0] + j[1] * j[1] + j[2] * j[2];
    return t * (rb + T(3) * cj + (T(4.5) * cj * cj - T(1.5) * jj) / (T(1) + rb));
}
template <typename T>
static void collide_force(T (&f)[19], T omega, const T (&g)[3], int n, T B, const T (&up)[3], T (&F)[3]) {
    T pre[19], rb, j[3];
    for (int i = 0; i < 19; ++i) pre[i] = f[i];
    moments(f, rb, j);
    if (n < 125) {
        const T rho = T(1) + rb;
        const T J[3] = {j[0] + T(0.5) * rho * g[0], j[1] + T(0.5) * rho * g[1], j[2] + T(0.5) * rho * g[2]};
        const T u[3] = {J[0] / rho, J[1] / rho, J[2] / rho};
        const T ug = u[0] * g[0] + u[1] * g[1] + u[2] * g[2];
        for (int i = 0; i < 19; ++i) {
            const T t = i == 0 ? T(1) / T(3) : (i < 4 || (i > 9 && i < 13)) ? T(1) / T(18) : T(1) / T(36);
            const T cg = CX[i] * g[0] + CY[i] * g[1] + CZ[i] * g[2], cu = CX[i] * u[0] + CY[i] * u[1] + CZ[i] * u[2];
            f[i] = (T(1) - omega) * f[i] + omega * feq<T>(i, rb, J) +
                   t * (T(1) - T(0.5) * omega) * rho * (T(3) * (cg - ug) + T(9) * cu * cg);
        }
        moments(f, rb, j);
    }
    F[0] = F[1] = F[2] = 0;
    if (n == 0) return;
    const T P[3] = {up[0] * (T(1) + rb), up[1] * (T(1) + rb), up[2] * (T(1) + rb)};
    f[0] = pre[0] + (T(1) - B) * (f[0] - pre[0]) + B * (feq<T>(0, rb, j) - feq<T>(0, rb, P));
    for (int i = 1; i < 10; ++i) {
        const int o = i + 9;
        const T bb = B * ((pre[o] - feq<T>(o, rb, j)) - (pre[i] - feq<T>(i, rb, P)));
        const T bo = B * ((pre[i] - feq<T>(i, rb, j)) - (pre[o] - feq<T>(o, rb, P)));
        f[i] = pre[i] + (T(1) - B) * (f[i] - pre[i]) + bb;
        f[o] = pre[o] + (T(1) - B) * (f[o] - pre[o]) + bo;
        F[0] -= CX[i] * (bb - bo);
        F[1] -= CY[i] * (bb - bo);
        F[2] -= CZ[i] * (bb - bo);
    }
}

struct Err {
    double mx = 0, sq = 0;
    long n = 0;
    void add(quad got, quad want, double scale) {
        const double e = std::fabs((double)(got - want)) / scale;
        mx = std::fmax(mx, e);
        sq += e * e;
        ++n;
    }
    double rms() const { return n ? std::sqrt(sq / n) : 0.0; }
};

int main(int argc, char** argv) {
    const long cells = argc > 1 ? std::atol(argv[1]) : 20000;
    std::mt19937_64 rng(argc > 2 ? std::atol(argv[2]) : 1);
    std::normal_distribution<double> N(0, 1);
    std::uniform_real_distribution<double> U(0, 1);
    struct Kind {
        const char* name;
        double rho, u, noise, up;   // density and velocity spread, non-equilibrium part, surface velocity spread
        bool solid;
        double g;                   // body force spread
    };
    const Kind kinds[] = {
        {"slow_fluid", 1e-5, 1e-4, 1e-7, 0, false, 0},      {"fluid", 1e-3, 1e-2, 1e-5, 0, false, 0},
        {"fast_fluid", 1e-2, 5e-2, 1e-3, 0, false, 0},      {"noise", 0, 0, 1e-3, 0, false, 0},
        {"faint_fluid", 1e-12, 1e-12, 1e-13, 0, false, 0},  {"solid", 1e-3, 1e-2, 1e-5, 1e-2, true, 0},
        {"slow_solid", 1e-5, 1e-4, 1e-7, 1e-4, true, 0},    {"fast_solid", 1e-2, 5e-2, 1e-3, 5e-2, true, 0},
        {"resting_bed", 1e-3, 1e-2, 1e-5, 0, true, 0},      {"far_outside", 0.5, 0.3, 1e-2, 0.3, true, 0},
        {"driven_fluid", 1e-3, 1e-2, 1e-5, 0, false, 1e-6}, {"driven_solid", 1e-3, 1e-2, 1e-5, 1e-2, true, 1e-6},
        {"pushed_fluid", 1e-3, 1e-2, 1e-5, 0, false, 1e-2}, {"pushed_solid", 1e-3, 1e-2, 1e-5, 1e-2, true, 1e-2},
    };
    for (const Kind& k : kinds) {
        Err fx, db, ffx, fdb;
        long bits = 0, out = 0;
        for (long c = 0; c < cells; ++c) {
            const double omega = 0.05 + 1.94 * U(rng);
            const double rb = k.rho * N(rng), u[3] = {k.u * N(rng), k.u * N(rng), k.u * N(rng)};
            double f[19], up[3] = {k.up * N(rng), k.up * N(rng), k.up * N(rng)};
            const double j2 = u[0] * u[0] + u[1] * u[1] + u[2] * u[2];
            for (int i = 0; i < 19; ++i) {
                const double t = i == 0 ? 1 / 3. : (i < 4 || (i > 9 && i < 13)) ? 1 / 18. : 1 / 36.;
                const double cj = CX[i] * u[0] + CY[i] * u[1] + CZ[i] * u[2];
                f[i] = t * (rb + 3 * cj + 4.5 * cj * cj - 1.5 * j2) + k.noise * N(rng);
            }
            const int n = k.solid ? 1 + (int)(U(rng) * 125) : 0;
            const double ooo = 1 / omega - 0.5, sf = n / 125.;
            const double B = n == 0 ? 0.0 : n >= 125 ? 1.0 : sf * ooo / ((1 - sf) + ooo);
            const double g[3] = {k.g * N(rng), k.g * N(rng), k.g * N(rng)};
            double a[19], b[19], Fa[3] = {0, 0, 0}, Fb[3];
            quad q[19], Fq[3], upq[3] = {up[0], up[1], up[2]};
            for (int i = 0; i < 19; ++i) { a[i] = b[i] = f[i]; q[i] = f[i]; }
            double scale = 0;
            for (int i = 0; i < 19; ++i) scale = std::fmax(scale, std::fabs(f[i]));
            for (double v : g) scale = std::fmax(scale, std::fabs(v) / 8);
            if (n) scale = std::fmax(scale, std::fmax(std::fabs(up[0]), std::fmax(std::fabs(up[1]), std::fabs(up[2]))) / 8);
            const bool force = k.g != 0;
            const quad gq[3] = {g[0], g[1], g[2]};
            if (force) {
                collide_force<quad>(q, omega, gq, n, B, upq, Fq);
                collide_force<double>(b, omega, g, n, B, up, Fb);
            } else {
                collide<quad>(q, omega, B, upq, Fq);
                collide<double>(b, omega, B, up, Fb);
            }
            auto fixed = [&](bool solid, double(&v)[19], int e, double(&F)[3]) {
                const lbdem::fixed::Relax rx = lbdem::fixed::relax_of(omega);
                const double w = solid && n ? B : 0.0, a0 = n ? up[0] : 0.0, a1 = n ? up[1] : 0.0, a2 = n ? up[2] : 0.0;
                if (force) lbdem::fixed::collide<true>(solid, v, e, rx, g[0], g[1], g[2], n == 125, w, a0, a1, a2, F);
                else lbdem::fixed::collide<false>(solid, v, e, rx, 0, 0, 0, n == 125, w, a0, a1, a2, F);
            };
            int e = lbdem::fixed::cell_exponent(f);
            if (n) e = lbdem::fixed::cell_exponent_up(e, up[0], up[1], up[2]);
            if (force) e = lbdem::fixed::cell_exponent_up(e, g[0], g[1], g[2]);
            if (!lbdem::fixed::fits(e)) { ++out; continue; }
            if (n) {
                fixed(true, a, e, Fa);
            } else {
                double a2[19], z[3];
                for (int i = 0; i < 19; ++i) a2[i] = a[i];
                fixed(false, a, e, Fa);
                fixed(true, a2, e, z);
                bool same = z[0] == 0 && z[1] == 0 && z[2] == 0;
                for (int i = 0; i < 19; ++i) same = same && std::memcmp(&a[i], &a2[i], 8) == 0;
                bits += same ? 0 : 1;
            }
            for (int i = 0; i < 19; ++i) {
                fx.add(a[i], q[i], scale);
                db.add(b[i], q[i], scale);
            }
            for (int d = 0; d < 3 && n; ++d) {
                ffx.add(Fa[d], Fq[d], scale);
                fdb.add(Fb[d], Fq[d], scale);
            }
        }
        std::printf("%s %.3e %.3e %.3e %.3e %.3e %.3e %.3e %.3e %ld %ld\n", k.name, fx.mx, fx.rms(), db.mx, db.rms(),
                    ffx.mx, ffx.rms(), fdb.mx, fdb.rms(), bits, out);
    }
    // exact zeros stay zero
    double z[19] = {}, F[3];
    const int e = lbdem::fixed::cell_exponent(z);
    bool zero = lbdem::fixed::fits(e);
    lbdem::fixed::collide<false>(false, z, e, lbdem::fixed::relax_of(1.7), 0, 0, 0, false, 0, 0, 0, 0, F);
    for (double v : z) zero = zero && v == 0.0;
    std::printf("zero %d\n", zero ? 1 : 0);
    // values outside the range are refused
    int refused = 0;
    for (double v : {0.04, 1e30, -(double)INFINITY, (double)NAN, 1e-300}) {
        double g[19] = {};
        g[7] = v;
        refused += lbdem::fixed::fits(lbdem::fixed::cell_exponent(g)) ? 0 : 1;
    }
    std::printf("refused %d\n", refused);
    return 0;
}
