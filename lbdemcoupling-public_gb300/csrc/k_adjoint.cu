// Reverse-mode (adjoint) step of the PSM lattice: gradients of a loss built
// from the per-particle forces and torques of a window of steps, with respect
// to the populations, the per-step particle velocities and angular velocities,
// the body force and the relaxation time tau.  The solid fraction and owner of
// every cell are held fixed over the window and are not differentiated.
//
// Forward map of one cell (what K1 computes, src/ibCompositeDynamics3D.hh:130-203,
// written as one function of the pre-collision populations f):
//   BGK with Guo forcing (n < 125):
//     rhoBar = sum f, j = sum c f, rho = 1 + rhoBar, r = 1/rho,
//     J = j + rho g / 2, u = J r, pre = (1 - omega/2) rho,
//     feq_k = t_k [rhoBar + 3 c_k.J + r (4.5 (c_k.J)^2 - 1.5 J.J)],
//     src_k = t_k pre [3 (c_k.g - u.g) + 9 (c_k.u)(c_k.g)],
//     f*_k = (1 - omega) f_k + omega feq_k + src_k          (f* = f when n = 125)
//   PSM (n > 0), moments rhoBar*, j* of f*, P = (1 + rhoBar*) uP:
//     out_k = (1 - B) f*_k + B (f_opp(k) - feq_opp(k)(j*) + feq_k(P))   k != 0
//     out_0 = (1 - B) f*_0 + B (f_0 + feq_0(j*) - feq_0(P))
//     F = -sum_{k=1..9} c_k (bb_k - bbOpp_k) = B (2 j - j* - P)
//   (feq(.) at rhoBar*, 1/(1 + rhoBar*)), and push streaming with half-way
//   bounce-back.  With uP = v + w x d (d: cell minus particle centre, minimum
//   image), tau entering through omega = 1/tau and B = sf ooo / ((1 - sf) + ooo),
//   ooo = tau - 1/2.
//
// The adjoint step, per cell x, given lambda_{t+1} (natural layout):
//   mu_k   = lambda_{t+1,k}(x + c_k), or lambda_{t+1,opp k}(x) beyond a wall
//            (transpose of push streaming),
//   a      = dL/dF of the owner particle at this step (+ w_T x arm for torques),
//   lambda_t(x) = (d out / d f)^T mu + (dF/df)^T a, and the parameter
//   gradients (d out / d theta)^T mu + (dF/d theta)^T a,
// evaluated by hand-written reverse differentiation of the formulas above.
#include "lbdem_internal.h"

namespace lbdem {
namespace {

constexpr unsigned FULLMASK = 0xffffffffu;
constexpr int ADJ_THREADS = 256;

template <typename T>
__device__ __forceinline__ T cdotT(int k, T a, T b, T c) {
    const int X = cx(k), Y = cy(k), Z = cz(k);
    T r = T(0);
    if (X) r = X > 0 ? a : -a;
    if (Y) r = Y > 0 ? r + b : r - b;
    if (Z) r = Z > 0 ? r + c : r - c;
    return r;
}

// 1/x: IEEE division in float; in double a float reciprocal refined by two
// Newton-Raphson steps r <- r (2 - x r) (relative error ~2^-23 -> ~2^-46 -> below
// double rounding), far cheaper than a double division on the narrow FP64 pipe.
__device__ __forceinline__ float recipT(float x) { return 1.0f / x; }
__device__ __forceinline__ double recipT(double x) {
    double r = (double)(1.0f / (float)x);
    r = r * (2.0 - x * r);
    return r * (2.0 - x * r);
}

template <typename T>
__device__ __forceinline__ T feqT(int k, T rb, T r, T c_dot, T sq) {
    return T(wt(k)) * (rb + T(3) * c_dot + r * (T(4.5) * c_dot * c_dot - T(1.5) * sq));
}

// Scalars of one cell's reverse pass; with them lambda_k (the adjoint of f_k) is
//   psm_k + (n == 125 ? phi_k : (1 - omega) phi_k + grb + c_k . gJ),
//   psm_k = B mu_opp(k) + 2 B (a . c_k),  phi_k = sB mu_k + grbs + c_k . gjs
// (n == 0: B = 0, sB = 1, grbs = gjs = 0), so the 19 values are formed while
// they are stored and never held together.
template <typename T>
struct CellAdj {
    T B, sB, grbs, gjs0, gjs1, gjs2;   // PSM part: adjoint of f* = sB mu + grbs + c . gjs
    T grb, gJ0, gJ1, gJ2;              // BGK part
};

// Reverse of one cell.  f: pre-collision populations; mu: adjoint of the
// post-collision populations; a: adjoint of the cell force.  Accumulates
// d/duP, d/dtau, d/dg and returns the scalars lambda is built from.
// general (warp-uniform: the warp holds a solid cell): a fluid cell takes the
// solid cells' path too, with B = 0, where it yields B = 0, sB = 1 and zero
// grbs, gjs, guP, so phi = mu and the same bits as the fluid path; the warp
// then runs one path instead of both.
template <typename T>
__device__ __forceinline__ CellAdj<T> adjoint_cell(const T (&f)[Q], const T (&mu)[Q], int n, bool general, T B,
                                                   T dBdtau, const T (&uP)[3], const T (&a)[3], T omega,
                                                   const T (&g)[3], T (&guP)[3], T& gtau, T (&gg)[3]) {
    CellAdj<T> R;
    // pre-collision moments
    T rb = T(0), j0 = T(0), j1 = T(0), j2 = T(0);
#pragma unroll
    for (int k = 0; k < Q; ++k) {
        rb += f[k];
        if (cx(k)) j0 += cx(k) > 0 ? f[k] : -f[k];
        if (cy(k)) j1 += cy(k) > 0 ? f[k] : -f[k];
        if (cz(k)) j2 += cz(k) > 0 ? f[k] : -f[k];
    }
    const T rho = T(1) + rb, r = recipT(rho);
    const T J0 = j0 + T(0.5) * rho * g[0], J1 = j1 + T(0.5) * rho * g[1], J2v = j2 + T(0.5) * rho * g[2];
    const T u0 = J0 * r, u1 = J1 * r, u2 = J2v * r;
    const T JJ = J0 * J0 + J1 * J1 + J2v * J2v;
    const T pre = (T(1) - T(0.5) * omega) * rho;
    const T ug = u0 * g[0] + u1 * g[1] + u2 * g[2];

    R.B = T(0); R.sB = T(1); R.grbs = T(0); R.gjs0 = T(0); R.gjs1 = T(0); R.gjs2 = T(0);
    guP[0] = guP[1] = guP[2] = T(0);
    if (n > 0 || general) {
        // moments of f* and S1 = sum mu_k f*_k
        T rbs = T(0), js0 = T(0), js1 = T(0), js2 = T(0), S1 = T(0);
        if (n == 125) {
            rbs = rb; js0 = j0; js1 = j1; js2 = j2;
#pragma unroll
            for (int k = 0; k < Q; ++k) S1 += mu[k] * f[k];
        } else {
#pragma unroll
            for (int k = 0; k < Q; ++k) {
                const T cJ = cdotT<T>(k, J0, J1, J2v);
                const T cu = cdotT<T>(k, u0, u1, u2), cg = cdotT<T>(k, g[0], g[1], g[2]);
                const T src = T(wt(k)) * pre * (T(3) * (cg - ug) + T(9) * cu * cg);
                const T fs = (T(1) - omega) * f[k] + omega * feqT<T>(k, rb, r, cJ, JJ) + src;
                rbs += fs;
                if (cx(k)) js0 += cx(k) > 0 ? fs : -fs;
                if (cy(k)) js1 += cy(k) > 0 ? fs : -fs;
                if (cz(k)) js2 += cz(k) > 0 ? fs : -fs;
                S1 += mu[k] * fs;
            }
        }
        R.B = B;
        R.sB = T(1) - B;
        const T rhos = T(1) + rbs, rs = recipT(rhos);
        const T Jq = js0 * js0 + js1 * js1 + js2 * js2;
        const T P0 = rhos * uP[0], P1 = rhos * uP[1], P2v = rhos * uP[2];
        const T PP = P0 * P0 + P1 * P1 + P2v * P2v;
        // F = B (2 j - j* - P)
        T gB = -S1 + a[0] * (T(2) * j0 - js0 - P0) + a[1] * (T(2) * j1 - js1 - P1) + a[2] * (T(2) * j2 - js2 - P2v);
        T gjs0 = -B * a[0], gjs1 = -B * a[1], gjs2 = -B * a[2];
        T gP0 = -B * a[0], gP1 = -B * a[1], gP2 = -B * a[2];
        // seeds e (of feq at j*) and E (of feq at P) of the B-weighted terms of out,
        // folded into the equilibria's reverse as they are formed
        T se = T(0), sE = T(0), grs = T(0);
        {
            const T q0 = feqT<T>(0, rbs, rs, T(0), Jq), s0 = feqT<T>(0, rbs, rs, T(0), PP);
            gB += mu[0] * (f[0] + q0 - s0);
            const T w = T(wt(0)), e0 = B * mu[0], E0 = -B * mu[0];
            se += w * e0;
            sE += w * E0;
            grs += w * (e0 * (-T(1.5) * Jq) + E0 * (-T(1.5) * PP));
        }
#pragma unroll
        for (int i = 1; i <= 9; ++i) {
            const int o = i + 9;
            const T w = T(wt(i));
            const T ci = cdotT<T>(i, js0, js1, js2);
            const T pi = cdotT<T>(i, P0, P1, P2v);
            const T qi = feqT<T>(i, rbs, rs, ci, Jq), qo = feqT<T>(o, rbs, rs, -ci, Jq);
            const T si = feqT<T>(i, rbs, rs, pi, PP), so = feqT<T>(o, rbs, rs, -pi, PP);
            gB += mu[i] * (f[o] - qo + si) + mu[o] * (f[i] - qi + so);
            const T ei = -B * mu[o], eo = -B * mu[i], Ei = B * mu[i], Eo = B * mu[o];
            se += w * (ei + eo);
            sE += w * (Ei + Eo);
            const T cq = T(4.5) * ci * ci - T(1.5) * Jq, pq = T(4.5) * pi * pi - T(1.5) * PP;
            grs += w * ((ei + eo) * cq + (Ei + Eo) * pq);
            // c_i w (e_i (3 + 9 rs c_i.j*) - e_o (3 - 9 rs c_i.j*)), c_o = -c_i
            const T aj = w * (ei * (T(3) + T(9) * rs * ci) - eo * (T(3) - T(9) * rs * ci));
            const T ap = w * (Ei * (T(3) + T(9) * rs * pi) - Eo * (T(3) - T(9) * rs * pi));
            if (cx(i)) { gjs0 += cx(i) > 0 ? aj : -aj; gP0 += cx(i) > 0 ? ap : -ap; }
            if (cy(i)) { gjs1 += cy(i) > 0 ? aj : -aj; gP1 += cy(i) > 0 ? ap : -ap; }
            if (cz(i)) { gjs2 += cz(i) > 0 ? aj : -aj; gP2 += cz(i) > 0 ? ap : -ap; }
        }
        // the -3 rs j* (resp. P) part of d feq / d j*, summed over k
        gjs0 -= T(3) * rs * se * js0; gjs1 -= T(3) * rs * se * js1; gjs2 -= T(3) * rs * se * js2;
        gP0 -= T(3) * rs * sE * P0; gP1 -= T(3) * rs * sE * P1; gP2 -= T(3) * rs * sE * P2v;
        // P = rho* uP, rs = 1/rho*, rho* = 1 + rbs
        T grhos = gP0 * uP[0] + gP1 * uP[1] + gP2 * uP[2];
        guP[0] = rhos * gP0; guP[1] = rhos * gP1; guP[2] = rhos * gP2;
        grhos -= rs * rs * grs;
        R.grbs = se + sE + grhos;
        R.gjs0 = gjs0; R.gjs1 = gjs1; R.gjs2 = gjs2;
        gtau += gB * dBdtau;
    }

    R.grb = T(0); R.gJ0 = T(0); R.gJ1 = T(0); R.gJ2 = T(0);
    if (n == 125) return R;   // no BGK: f* = f
    // BGK reverse with phi_k = sB mu_k + grbs + c_k . gjs.  Every term is a
    // weighted moment of phi of order <= 2 in c_k (feq and src are quadratic in
    // c_k), so the sums over k reduce to m0 = sum t_k phi_k, m1 = sum t_k phi_k c_k,
    // m2 = sum t_k phi_k c_k c_k^T, and sum phi_k f_k.
    T m0 = T(0), m1x = T(0), m1y = T(0), m1z = T(0);
    T mxx = T(0), myy = T(0), mzz = T(0), mxy = T(0), mxz = T(0), myz = T(0), sphf = T(0);
    auto moments = [&](auto phi_of) {
#pragma unroll
        for (int k = 0; k < Q; ++k) {
            const T phi = phi_of(k);
            sphf += phi * f[k];
            const T wp = T(wt(k)) * phi;
            m0 += wp;
            const int X = cx(k), Y = cy(k), Z = cz(k);
            if (X) { m1x += X > 0 ? wp : -wp; mxx += wp; }
            if (Y) { m1y += Y > 0 ? wp : -wp; myy += wp; }
            if (Z) { m1z += Z > 0 ? wp : -wp; mzz += wp; }
            if (X && Y) mxy += X * Y > 0 ? wp : -wp;
            if (X && Z) mxz += X * Z > 0 ? wp : -wp;
            if (Y && Z) myz += Y * Z > 0 ? wp : -wp;
        }
    };
    if (!general) moments([&](int k) { return mu[k]; });   // fluid cells only: phi = mu
    else moments([&](int k) { return R.sB * mu[k] + R.grbs + cdotT<T>(k, R.gjs0, R.gjs1, R.gjs2); });
    // m2 applied to J, u, g
    const T aJ0 = mxx * J0 + mxy * J1 + mxz * J2v, aJ1 = mxy * J0 + myy * J1 + myz * J2v,
            aJ2 = mxz * J0 + myz * J1 + mzz * J2v;
    const T ag0 = mxx * g[0] + mxy * g[1] + mxz * g[2], ag1 = mxy * g[0] + myy * g[1] + myz * g[2],
            ag2 = mxz * g[0] + myz * g[1] + mzz * g[2];
    const T au0 = mxx * u0 + mxy * u1 + mxz * u2, au1 = mxy * u0 + myy * u1 + myz * u2,
            au2 = mxz * u0 + myz * u1 + mzz * u2;
    const T JmJ = J0 * aJ0 + J1 * aJ1 + J2v * aJ2;
    const T quad = T(4.5) * JmJ - T(1.5) * JJ * m0;            // sum t phi (4.5 (c.J)^2 - 1.5 J.J)
    // sum phi_k feq_k - sum phi_k f_k
    T gom = rb * m0 + T(3) * (m1x * J0 + m1y * J1 + m1z * J2v) + r * quad - sphf;
    const T sh = omega * m0;                                       // sum t_k h_k, h = omega phi
    T gr = omega * quad;
    T gJ0 = omega * (T(3) * m1x + T(9) * r * aJ0), gJ1 = omega * (T(3) * m1y + T(9) * r * aJ1),
      gJ2 = omega * (T(3) * m1z + T(9) * r * aJ2);
    const T gpre = T(3) * (m1x * g[0] + m1y * g[1] + m1z * g[2]) - T(3) * ug * m0 +
                   T(9) * (u0 * ag0 + u1 * ag1 + u2 * ag2);
    const T swp = pre * m0;                                        // sum t_k pre phi_k
    T gu0 = T(9) * pre * ag0, gu1 = T(9) * pre * ag1, gu2 = T(9) * pre * ag2;
    T gg0 = pre * (T(3) * m1x + T(9) * au0), gg1 = pre * (T(3) * m1y + T(9) * au1),
      gg2 = pre * (T(3) * m1z + T(9) * au2);
    // the k-independent parts: -3 r J (sum t h), -3 g (sum t pre phi), -3 u (sum t pre phi)
    gJ0 -= T(3) * r * sh * J0; gJ1 -= T(3) * r * sh * J1; gJ2 -= T(3) * r * sh * J2v;
    gu0 -= T(3) * swp * g[0]; gu1 -= T(3) * swp * g[1]; gu2 -= T(3) * swp * g[2];
    gg0 -= T(3) * swp * u0; gg1 -= T(3) * swp * u1; gg2 -= T(3) * swp * u2;
    // pre = (1 - omega/2) rho
    gom -= T(0.5) * rho * gpre;
    T grho = (T(1) - T(0.5) * omega) * gpre;
    // u = J r
    gJ0 += r * gu0; gJ1 += r * gu1; gJ2 += r * gu2;
    gr += J0 * gu0 + J1 * gu1 + J2v * gu2;
    // J = j + rho g / 2
    grho += T(0.5) * (g[0] * gJ0 + g[1] * gJ1 + g[2] * gJ2);
    gg0 += T(0.5) * rho * gJ0; gg1 += T(0.5) * rho * gJ1; gg2 += T(0.5) * rho * gJ2;
    grho -= r * r * gr;
    R.grb = sh + grho;
    R.gJ0 = gJ0; R.gJ1 = gJ1; R.gJ2 = gJ2;
    gtau -= gom * omega * omega;   // omega = 1/tau
    gg[0] += gg0; gg[1] += gg1; gg[2] += gg2;
    return R;
}

// ---------------------------------------------------------------------------
// The same reverse in double, built from moments.  GB300 has two double lanes per clock
// per SM, and the sums above, written per direction, take about 600 double operations
// for a fluid cell and 1500 for a solid one (553 us a step at 64^3, against 264 here).  Every sum over the
// directions is a contraction of
//   M0 = sum t mu,  M1 = sum t mu c,  M2 = sum t mu c c,  sum mu_k f_k,  sum mu_k f_opp(k)
// with the cell's vectors (feq and the source are quadratic in c), so those are formed
// once per opposite pair and the rest is scalar algebra:
//   sum_k mu_k feq_k(rb, r, v) = rb M0 + 3 M1.v + r (4.5 v.M2.v - 1.5 v.v M0) =: q(v),
//   moments of f*: rbs = rb, j* = j + rho g (the Guo source adds rho g / 2 to the relaxed
//   J = j + rho g / 2), j below full coverage;
//   moments of phi = sB mu + grbs + c.gjs: with sum t = 1, sum t c c = 1/3,
//   m0 = sB M0 + grbs, m1 = sB M1 + gjs / 3, m2 = sB M2 + grbs / 3.
// The result is lambda_k = am mu_k + B mu_opp(k) + k0 + c_k.v.
struct CellAdjD {
    double am, B, k0, v0, v1, v2;
};
struct Moments2 {
    double m0, x, y, z, xx, yy, zz, xy, xz, yz;
};
// v.M2.v and the vector M2.v
__device__ __forceinline__ void apply2(const Moments2& m, double a, double b, double c, double& x, double& y,
                                       double& z) {
    x = fma(m.xz, c, fma(m.xy, b, m.xx * a));
    y = fma(m.yz, c, fma(m.yy, b, m.xy * a));
    z = fma(m.zz, c, fma(m.yz, b, m.xz * a));
}
__device__ __forceinline__ double dot3(double a, double b, double c, double x, double y, double z) {
    return fma(c, z, fma(b, y, a * x));
}

__device__ __forceinline__ CellAdjD adjoint_cell_double(const double (&f)[Q], const double (&mu)[Q], int n,
                                                        bool general, double B, double dBdtau, const double (&uP)[3],
                                                        const double (&a)[3], double omega, const double (&g)[3],
                                                        double (&guP)[3], double& gtau, double (&gg)[3]) {
    constexpr double t0 = 1.0 / 3.0, t1 = 1.0 / 18.0, t2 = 1.0 / 36.0;
    // pairs (k, i = k - 9), c_k = -c_i: sums and differences, then per axis a with the plane
    // (a, b): axis pair, c = e_a + e_b and c = e_a - e_b
    double rb = f[0], A = 0.0, D = 0.0;   // sum (mu_k + mu_i)(f_k + f_i), sum (mu_k - mu_i)(f_k - f_i)
    double jv[3] = {0.0, 0.0, 0.0}, P1[3], PP[3], PM[3], M1a[3], MP[3], MM[3];
#pragma unroll
    for (int ax = 0; ax < 3; ++ax) {
        // axis, plus and minus pairs of the planes (x, y), (y, z), (x, z)
        const int ka = 10 + ax, kp = ax == 0 ? 13 : (ax == 1 ? 17 : 15), km = kp + 1;
        const double pa = mu[ka] + mu[ka - 9], ma = mu[ka] - mu[ka - 9];
        const double pp = mu[kp] + mu[kp - 9], mp = mu[kp] - mu[kp - 9];
        const double pm = mu[km] + mu[km - 9], mm = mu[km] - mu[km - 9];
        const double sa = f[ka] + f[ka - 9], da = f[ka] - f[ka - 9];
        const double sp = f[kp] + f[kp - 9], dp = f[kp] - f[kp - 9];
        const double sm = f[km] + f[km - 9], dm = f[km] - f[km - 9];
        rb += sa + (sp + sm);
        A = fma(pm, sm, fma(pp, sp, fma(pa, sa, A)));
        D = fma(mm, dm, fma(mp, dp, fma(ma, da, D)));
        const int b1 = ax == 1 ? 1 : 0, b2 = ax == 0 ? 1 : 2;   // first and second axis of the plane
        jv[ax] += da;
        jv[b1] += dp + dm;
        jv[b2] += dp - dm;
        P1[ax] = pa;
        M1a[ax] = ma;
        PP[ax] = pp + pm;
        PM[ax] = pp - pm;
        MP[ax] = mp + mm;
        MM[ax] = mp - mm;
    }
    const double jx = jv[0], jy = jv[1], jz = jv[2];
    Moments2 M;   // planes: 0 (x, y), 1 (y, z), 2 (x, z)
    M.m0 = fma(t0, mu[0], fma(t1, (P1[0] + P1[1]) + P1[2], t2 * ((PP[0] + PP[1]) + PP[2])));
    M.x = fma(t1, M1a[0], t2 * (MP[0] + MP[2]));
    M.y = fma(t1, M1a[1], t2 * (MM[0] + MP[1]));
    M.z = fma(t1, M1a[2], t2 * (MM[1] + MM[2]));
    M.xx = fma(t1, P1[0], t2 * (PP[0] + PP[2]));
    M.yy = fma(t1, P1[1], t2 * (PP[0] + PP[1]));
    M.zz = fma(t1, P1[2], t2 * (PP[1] + PP[2]));
    M.xy = t2 * PM[0];
    M.yz = t2 * PM[1];
    M.xz = t2 * PM[2];
    const double m0f0 = mu[0] * f[0];
    const double smf = fma(0.5, A + D, m0f0), smo = fma(0.5, A - D, m0f0);

    const double rho = 1.0 + rb, r = recipT(rho), hr = 0.5 * rho;
    const double J0 = fma(hr, g[0], jx), J1 = fma(hr, g[1], jy), J2v = fma(hr, g[2], jz);
    const double u0 = J0 * r, u1 = J1 * r, u2 = J2v * r;
    const double JJ = dot3(J0, J1, J2v, J0, J1, J2v);
    const double pre = (1.0 - 0.5 * omega) * rho;
    const double ug = dot3(u0, u1, u2, g[0], g[1], g[2]);

    CellAdjD R;
    R.B = 0.0;
    double sB = 1.0, grbs = 0.0, gjs0 = 0.0, gjs1 = 0.0, gjs2 = 0.0, ta0 = 0.0, ta1 = 0.0, ta2 = 0.0;
    guP[0] = guP[1] = guP[2] = 0.0;
    double J20, J21, J22;   // M2.J
    apply2(M, J0, J1, J2v, J20, J21, J22);
    const double JMJ = dot3(J0, J1, J2v, J20, J21, J22);
    const double m1J = dot3(M.x, M.y, M.z, J0, J1, J2v);
    const double quadJ = fma(4.5, JMJ, -1.5 * JJ * M.m0);
    double mg0, mg1, mg2;   // M2.g
    apply2(M, g[0], g[1], g[2], mg0, mg1, mg2);
    const double m1g = dot3(M.x, M.y, M.z, g[0], g[1], g[2]);
    const double umg = dot3(u0, u1, u2, mg0, mg1, mg2);
    if (general) {
        const bool full = n == 125;
        // S1 = sum mu f*
        const double mfeq = fma(rb, M.m0, fma(3.0, m1J, r * quadJ));
        const double msrc = pre * fma(9.0, umg, fma(3.0, m1g, -3.0 * ug * M.m0));
        const double S1 = full ? smf : fma(1.0 - omega, smf, fma(omega, mfeq, msrc));
        const double hs = full ? 0.0 : rho;
        const double s0 = fma(hs, g[0], jx), s1 = fma(hs, g[1], jy), s2 = fma(hs, g[2], jz);   // j*
        const double Q0 = rho * uP[0], Q1 = rho * uP[1], Q2 = rho * uP[2];                       // P
        const double Jq = dot3(s0, s1, s2, s0, s1, s2), QQ = dot3(Q0, Q1, Q2, Q0, Q1, Q2);
        double ms0, ms1, ms2, mp0, mp1, mp2;   // M2.j*, M2.P
        apply2(M, s0, s1, s2, ms0, ms1, ms2);
        apply2(M, Q0, Q1, Q2, mp0, mp1, mp2);
        const double qs = fma(4.5, dot3(s0, s1, s2, ms0, ms1, ms2), -1.5 * Jq * M.m0);
        const double qp = fma(4.5, dot3(Q0, Q1, Q2, mp0, mp1, mp2), -1.5 * QQ * M.m0);
        const double dq = qp - qs;
        const double m1s = dot3(M.x, M.y, M.z, s0 + Q0, s1 + Q1, s2 + Q2);
        const double c0 = -1.5 * (Jq - QQ) * (t0 * mu[0]);   // mu_0 t_0 (-1.5)(j*.j* - P.P)
        // sum mu_k (f_opp - feq_opp(j*) + feq_k(P)) with the rest population's sign, F terms
        const double w = fma(r, fma(2.0, c0, dq), fma(3.0, m1s, smo));
        const double gB = (w - S1) + dot3(a[0], a[1], a[2], (2.0 * jx - s0) - Q0, (2.0 * jy - s1) - Q1,
                                          (2.0 * jz - s2) - Q2);
        R.B = B;
        sB = 1.0 - B;
        const double se = B * fma(2.0, t0 * mu[0], -M.m0);   // sum t e; sum t E = -se
        const double e3 = 3.0 * r * se, b3 = 3.0 * B, b9 = 9.0 * B * r;
        const double k0 = fma(b3, M.x, -B * a[0]), k1 = fma(b3, M.y, -B * a[1]), k2 = fma(b3, M.z, -B * a[2]);
        gjs0 = fma(-e3, s0, fma(-b9, ms0, k0));
        gjs1 = fma(-e3, s1, fma(-b9, ms1, k1));
        gjs2 = fma(-e3, s2, fma(-b9, ms2, k2));
        const double gP0 = fma(e3, Q0, fma(b9, mp0, k0)), gP1 = fma(e3, Q1, fma(b9, mp1, k1)),
                     gP2 = fma(e3, Q2, fma(b9, mp2, k2));
        const double grs = B * fma(2.0, c0, dq);
        grbs = fma(-r * r, grs, dot3(gP0, gP1, gP2, uP[0], uP[1], uP[2]));
        guP[0] = rho * gP0;
        guP[1] = rho * gP1;
        guP[2] = rho * gP2;
        gtau = fma(gB, dBdtau, gtau);
        ta0 = 2.0 * B * a[0];
        ta1 = 2.0 * B * a[1];
        ta2 = 2.0 * B * a[2];
    }
    if (n == 125) {   // no BGK: f* = f
        R.am = sB;
        R.k0 = grbs;
        R.v0 = gjs0 + ta0;
        R.v1 = gjs1 + ta1;
        R.v2 = gjs2 + ta2;
        return R;
    }
    // BGK reverse with the moments of phi: m0, m1, m2.J and m2.g (m2.u = m2.J r); fluid
    // cells have phi = mu (and get the same bits from the solid cells' expressions)
    double m0 = M.m0, m1x = M.x, m1y = M.y, m1z = M.z, sphf = smf;
    double aJ0 = J20, aJ1 = J21, aJ2 = J22, ag0 = mg0, ag1 = mg1, ag2 = mg2;
    if (general) {
        const double third = 1.0 / 3.0, g3 = third * grbs;
        m0 = fma(sB, M.m0, grbs);
        m1x = fma(sB, M.x, third * gjs0);
        m1y = fma(sB, M.y, third * gjs1);
        m1z = fma(sB, M.z, third * gjs2);
        sphf = fma(sB, smf, fma(grbs, rb, dot3(gjs0, gjs1, gjs2, jx, jy, jz)));
        aJ0 = fma(sB, J20, g3 * J0); aJ1 = fma(sB, J21, g3 * J1); aJ2 = fma(sB, J22, g3 * J2v);
        ag0 = fma(sB, mg0, g3 * g[0]); ag1 = fma(sB, mg1, g3 * g[1]); ag2 = fma(sB, mg2, g3 * g[2]);
    }
    double quad = quadJ, mJ = m1J, mg = m1g, uag = umg;
    if (general) {
        quad = fma(4.5, dot3(J0, J1, J2v, aJ0, aJ1, aJ2), -1.5 * JJ * m0);
        mJ = dot3(m1x, m1y, m1z, J0, J1, J2v);
        mg = dot3(m1x, m1y, m1z, g[0], g[1], g[2]);
        uag = dot3(u0, u1, u2, ag0, ag1, ag2);
    }
    double gom = fma(rb, m0, fma(3.0, mJ, fma(r, quad, -sphf)));   // sum phi feq - sum phi f
    const double gpre = fma(9.0, uag, fma(3.0, mg, -3.0 * ug * m0));
    const double swp3 = 3.0 * pre * m0, pre9 = 9.0 * pre, pre3 = 3.0 * pre;
    const double gu0 = fma(pre9, ag0, -swp3 * g[0]), gu1 = fma(pre9, ag1, -swp3 * g[1]),
                 gu2 = fma(pre9, ag2, -swp3 * g[2]);
    const double om3 = 3.0 * omega, om9r = 9.0 * omega * r, rsh = om3 * r * m0;
    const double gJ0 = fma(r, gu0, fma(-rsh, J0, fma(om9r, aJ0, om3 * m1x)));
    const double gJ1 = fma(r, gu1, fma(-rsh, J1, fma(om9r, aJ1, om3 * m1y)));
    const double gJ2 = fma(r, gu2, fma(-rsh, J2v, fma(om9r, aJ2, om3 * m1z)));
    const double p9r = pre9 * r;
    gg[0] += fma(hr, gJ0, fma(-swp3, u0, fma(p9r, aJ0, pre3 * m1x)));
    gg[1] += fma(hr, gJ1, fma(-swp3, u1, fma(p9r, aJ1, pre3 * m1y)));
    gg[2] += fma(hr, gJ2, fma(-swp3, u2, fma(p9r, aJ2, pre3 * m1z)));
    gom = fma(-hr, gpre, gom);   // pre = (1 - omega/2) rho
    const double gr = fma(omega, quad, dot3(J0, J1, J2v, gu0, gu1, gu2));
    const double grho = fma(-r * r, gr, fma(1.0 - 0.5 * omega, gpre, 0.5 * dot3(g[0], g[1], g[2], gJ0, gJ1, gJ2)));
    gtau -= gom * omega * omega;   // omega = 1/tau
    const double om1 = 1.0 - omega;
    R.am = om1;
    R.k0 = fma(omega, m0, grho);
    R.v0 = gJ0;
    R.v1 = gJ1;
    R.v2 = gJ2;
    if (general) {
        R.am = om1 * sB;
        R.k0 = fma(om1, grbs, R.k0);
        R.v0 = fma(om1, gjs0, gJ0) + ta0;
        R.v1 = fma(om1, gjs1, gJ1) + ta1;
        R.v2 = fma(om1, gjs2, gJ2) + ta2;
    }
    return R;
}

// Warp-segmented sum of six values per particle slot into out[key][6]
// (consecutive cells mostly share the owner).  All 32 lanes must call.
template <typename T>
__device__ __forceinline__ void reduce6(int key, T (&v)[6], double* __restrict__ out) {
    const unsigned solid = __ballot_sync(FULLMASK, key >= 0);
    if (solid == 0u) return;
    const int lane = threadIdx.x & 31;
    const int prevKey = __shfl_up_sync(FULLMASK, key, 1);
    const bool head = (lane == 0) || (prevKey != key);
    const unsigned heads = __ballot_sync(FULLMASK, head);
    const int segStart = 31 - __clz(heads & (FULLMASK >> (31 - lane)));
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
#pragma unroll
        for (int q = 0; q < 6; ++q) {
            const T o = __shfl_up_sync(FULLMASK, v[q], d);
            if (lane - d >= segStart) v[q] += o;
        }
    }
    const int nextKey = __shfl_down_sync(FULLMASK, key, 1);
    const bool tail = (lane == 31) || (nextKey != key);
    if (tail && key >= 0)
#pragma unroll
        for (int q = 0; q < 6; ++q) atomicAdd(out + 6 * (size_t)key + q, (double)v[q]);
}

// A run's rows in shared memory, made by one warp, one direction a lane: a load or store
// then takes one shared load and one multiply-add (FP32 step at 128^3: 155 us with the addresses
// formed at each, 138 so; FP64 at 64^3, bound by its double operations: 270 and 264).
// [f + k] the row that f_k is read from (f: even phase the run's own; odd phase slot opp k of
// row x - c_k), [mu + k] that of mu_k (slot k of row x + c_k), each followed by the entries
// for a z wall (the own row's slot, index z) and for the periodic z boundary; [out + k] the
// run's own row of lambda_out.  Beyond an x / y wall all three lead to the cell itself,
// whatever c_z did to its z.
constexpr int ROWS_F = 0, ROWS_MU = 3 * Q, ROWS_OUT = 6 * Q, ROWS_ALL = 7 * Q;
template <typename T, bool PER>
__device__ __forceinline__ void adjoint_rows(T** rows, const AdjointArgs<T>& A, int x, int y) {
    const int k = threadIdx.x & 31;
    const Geom& g = A.g;
    __syncwarp();   // the last run's reads
    if (k < Q) {
        const size_t N = g.N, own = ((size_t)x * g.ny + y) * g.nz;
        // row (x + dx, y + dy), or -1 beyond a wall
        auto row = [&](int dx, int dy) -> long long {
            int X = x + dx, Y = y + dy;
            if (X < 0 || X >= g.nx) X = PER || g.per[0] ? (X < 0 ? g.nx - 1 : 0) : -1;
            if (Y < 0 || Y >= g.ny) Y = PER || g.per[1] ? (Y < 0 ? g.ny - 1 : 0) : -1;
            return PER || (X >= 0 && Y >= 0) ? ((long long)X * g.ny + Y) * g.nz : -1;
        };
        auto entries = [&](T** t, T* base, int slot, int back, long long r, int c) {
            T* const self = base + ((size_t)back * N + own);
            T* const there = base + ((size_t)slot * N + (size_t)(r >= 0 ? r : 0));
            t[k] = PER || r >= 0 ? there : self - c;
            t[Q + k] = self;
            t[2 * Q + k] = PER || r >= 0 ? there : self + c * (g.nz - 1);
        };
        T* const f = const_cast<T*>(A.f);
        if (A.phase == 0) rows[ROWS_F + k] = f + ((size_t)k * N + own);
        else entries(rows + ROWS_F, f, opp(k), k, row(-cx(k), -cy(k)), -cz(k));
        entries(rows + ROWS_MU, const_cast<T*>(A.lam_in), k, opp(k), row(cx(k), cy(k)), cz(k));
        rows[ROWS_OUT + k] = A.lam_out + ((size_t)k * N + own);
    }
    __syncwarp();
}

// PER: every axis periodic (no wall cases in the neighbour lookups).
template <typename T, bool PER>
__global__ void __launch_bounds__(ADJ_THREADS, sizeof(T) == 4 ? 2 : 1) k_adjoint_step(const AdjointArgs<T> A) {
    __shared__ double s_red[ADJ_THREADS / 32][4];
    __shared__ T* s_rows[ADJ_THREADS / 32][ROWS_ALL];
    T** const rows = s_rows[threadIdx.x >> 5];
    const Geom g = A.g;
    T gtau = T(0), gg[3] = {T(0), T(0), T(0)};   // per-thread sums, widened once
    // one warp per 64-cell run of a z-row, in two passes of 32 cells: rows * runs
    // < 2^31 (nx * ny < 2^31 is checked at creation), so all index arithmetic
    // stays in 32 bits.  The run's solid cells are taken first (pass 0 holds as
    // many as fit): a pass with a solid cell runs the solid cells' path for every
    // lane, so gathering them leaves more passes on the fluid path.  A cell's
    // result does not depend on its pass.
    const int lane = threadIdx.x & 31;
    const int nzc = (g.nz + 63) >> 6;
    const long long nchunks = (long long)g.nx * g.ny * nzc;
    const long long wstride = (long long)gridDim.x * (ADJ_THREADS / 32);
    for (long long q = (long long)blockIdx.x * (ADJ_THREADS / 32) + (threadIdx.x >> 5); q < nchunks; q += wstride) {
        const int qi = (int)q;   // runs of 64 cells: < 2^31 for any lattice that fits in memory
        const int row = qi / nzc;
        const int zb = (qi - row * nzc) * 64;
        const int len = min(64, g.nz - zb);
        const int x = row / g.ny, y = row - x * g.ny;
        adjoint_rows<T, PER>(rows, A, x, y);
        const size_t rowc = (size_t)row * g.nz + zb;
        const uint32_t wl0 = lane < len ? A.vox[rowc + lane] : 0u;
        const uint32_t wl1 = lane + 32 < len ? A.vox[rowc + lane + 32] : 0u;
        const unsigned sol0 = __ballot_sync(FULLMASK, (wl0 & VOX_NMASK) != 0u);
        const unsigned sol1 = __ballot_sync(FULLMASK, (wl1 & VOX_NMASK) != 0u);
        const unsigned flu0 = __ballot_sync(FULLMASK, lane < len) & ~sol0;
        const unsigned flu1 = __ballot_sync(FULLMASK, lane + 32 < len) & ~sol1;
        const int ns0 = __popc(sol0), ns = ns0 + __popc(sol1);
        const int nf0 = __popc(flu0), nf = nf0 + __popc(flu1);
#pragma unroll 1
        for (int pass = 0; pass < 2; ++pass) {
            const int slot_l = 32 * pass + lane;
            int jr = -1;   // the cell of the run this lane takes in this pass
            if (slot_l < ns) jr = slot_l < ns0 ? nth_bit(sol0, slot_l) : 32 + nth_bit(sol1, slot_l - ns0);
            else if (slot_l - ns < nf)
                jr = slot_l - ns < nf0 ? nth_bit(flu0, slot_l - ns) : 32 + nth_bit(flu1, slot_l - ns - nf0);
            const bool general = ns > 32 * pass;   // warp-uniform: the pass holds a solid cell
            const int z = zb + jr;
            int key = -1;
            T pv[6] = {T(0), T(0), T(0), T(0), T(0), T(0)};
            if (jr >= 0) {
                const size_t c = (size_t)row * g.nz + z;
                // z - 1, z, z + 1 (wrapped; z itself beyond a wall) and their part of the row table
                int zs[3] = {z - 1, z, z + 1}, ts[3] = {0, 0, 0};
                const bool wrap = PER || g.per[2];
                if (z == 0) { zs[0] = wrap ? g.nz - 1 : z; ts[0] = wrap ? 2 * Q : Q; }
                if (z == g.nz - 1) { zs[2] = wrap ? 0 : z; ts[2] = wrap ? 2 * Q : Q; }
                auto at = [&](int tab, int k, int dz) -> T {
                    return rows[tab + k + (PER ? 0 : ts[dz + 1])][zs[dz + 1]];
                };
                T f[Q], mu[Q];
                if (A.phase == 0) {
#pragma unroll
                    for (int k = 0; k < Q; ++k) f[k] = rows[ROWS_F + k][z];
                } else {
                    // odd layout: f_k(x) in slot (opp k, x - c_k), or (k, x) when x - c_k is beyond a wall
#pragma unroll
                    for (int k = 0; k < Q; ++k) f[k] = at(ROWS_F, k, -cz(k));
                }
                // transpose of push streaming: mu_k = lambda_k(x + c_k), or lambda_opp k(x) beyond a wall
#pragma unroll
                for (int k = 0; k < Q; ++k) mu[k] = at(ROWS_MU, k, cz(k));
                const uint32_t w = A.vox[c];
                int n = min((int)(w & VOX_NMASK), 125);
                T uP[3] = {T(0), T(0), T(0)}, a[3] = {T(0), T(0), T(0)}, d[3] = {T(0), T(0), T(0)};
                T B = T(0), dBdtau = T(0);
                int slot = -1;
                if (n > 0) {
                    const int tag = (int)(w >> VOX_NBITS);
                    slot = tag <= A.max_tag ? A.tag2slot[tag] : -1;
                    if (slot < 0 || slot >= A.nslot) {
                        atomicOr(A.err, 0x8u);   // LBDEM_DEVERR_UNMAPPED_TAG
                        slot = -1;
                    } else {
                        const double* p = A.rec + (size_t)slot * REC_STRIDE;
                        // arm d = cell - centre, minimum image as in the force arm
                        // (src/ibProcessors3D.hh:230-243); the float form takes the
                        // centre's hi/lo split as the forward pass does
                        if (sizeof(T) == 8) {
                            d[0] = T((double)x - p[0]); d[1] = T((double)y - p[1]); d[2] = T((double)z - p[2]);
                        } else {
                            const float4* q4 = reinterpret_cast<const float4*>(A.xpf + (size_t)slot * XPF_STRIDE);
                            const float4 hq = q4[0], lq = q4[1];
                            d[0] = T(((float)x - hq.x) - hq.w);
                            d[1] = T(((float)y - hq.y) - lq.x);
                            d[2] = T(((float)z - hq.z) - lq.y);
                        }
                        const int ext[3] = {g.nx, g.ny, g.nz};
#pragma unroll
                        for (int q = 0; q < 3; ++q) {
                            const int h = ext[q] / 2;
                            if (d[q] > T(h)) d[q] -= T(ext[q]);
                            else if (d[q] < T(-h)) d[q] += T(ext[q]);
                        }
                        const T v0 = T(p[3]), v1 = T(p[4]), v2 = T(p[5]);
                        const T w0 = T(p[6]), w1 = T(p[7]), w2 = T(p[8]);
                        // uP = v + w x d (setValues, src/ibProcessors3D.hh:163-174)
                        uP[0] = v0 + (w1 * d[2] - w2 * d[1]);
                        uP[1] = v1 + (-w0 * d[2] + w2 * d[0]);
                        uP[2] = v2 + (w0 * d[1] - w1 * d[0]);
                        const double* wgt = A.w + (size_t)slot * 6;
                        const T wf0 = T(wgt[0]), wf1 = T(wgt[1]), wf2 = T(wgt[2]);
                        const T wt0 = T(wgt[3]), wt1 = T(wgt[4]), wt2 = T(wgt[5]);
                        // dL/dF_cell = w_F + w_T x d
                        a[0] = wf0 + (wt1 * d[2] - wt2 * d[1]);
                        a[1] = wf1 + (wt2 * d[0] - wt0 * d[2]);
                        a[2] = wf2 + (wt0 * d[1] - wt1 * d[0]);
                        B = A.btab[n];
                        const T sf = T(1.0 / 125.0) * T(n), den = (T(1) - sf) + (A.tauT - T(0.5));
                        dBdtau = n < 125 ? sf * (T(1) - sf) / (den * den) : T(0);
                    }
                }
                if (n > 0 && slot < 0) n = 0;
                T guP[3];
                const T gvec[3] = {A.g3[0], A.g3[1], A.g3[2]};
                if constexpr (sizeof(T) == 8) {
                    const CellAdjD R =
                        adjoint_cell_double(f, mu, n, general, B, dBdtau, uP, a, A.omega, gvec, guP, gtau, gg);
                    // lambda_k = am mu_k + B mu_opp(k) + k0 + c_k.v (a fluid cell has B = 0 and am = 1 - omega)
                    rows[ROWS_OUT][z] = fma(R.am, mu[0], fma(R.B, mu[0], R.k0));
#pragma unroll
                    for (int k = 10; k < Q; ++k) {
                        const int i = k - 9;
                        const double cv = cdotT<double>(k, R.v0, R.v1, R.v2);
                        const double hi = R.k0 + cv, lo = R.k0 - cv;
                        rows[ROWS_OUT + k][z] = fma(R.am, mu[k], general ? fma(R.B, mu[i], hi) : hi);
                        rows[ROWS_OUT + i][z] = fma(R.am, mu[i], general ? fma(R.B, mu[k], lo) : lo);
                    }
                } else {
                    const CellAdj<T> R =
                        adjoint_cell<T>(f, mu, n, general, B, dBdtau, uP, a, A.omega, gvec, guP, gtau, gg);
                    const T om1 = n == 125 ? T(1) : T(1) - A.omega;
                    if (!general) {   // fluid cells only: phi = mu, no solid terms
#pragma unroll
                        for (int k = 0; k < Q; ++k)
                            rows[ROWS_OUT + k][z] = om1 * mu[k] + (R.grb + cdotT<T>(k, R.gJ0, R.gJ1, R.gJ2));
                    } else {
                        // the fluid path's expression plus the solid terms (exactly zero for a fluid cell)
#pragma unroll
                        for (int k = 0; k < Q; ++k) {
                            const T phi = R.sB * mu[k] + R.grbs + cdotT<T>(k, R.gjs0, R.gjs1, R.gjs2);
                            T l = om1 * phi + (R.grb + cdotT<T>(k, R.gJ0, R.gJ1, R.gJ2));
                            l += R.B * mu[opp(k)] + T(2) * R.B * cdotT<T>(k, a[0], a[1], a[2]);
                            rows[ROWS_OUT + k][z] = l;
                        }
                    }
                }
                if (slot >= 0) {
                    key = slot;
                    pv[0] = guP[0]; pv[1] = guP[1]; pv[2] = guP[2];
                    // d/dw of w x d: d x guP
                    pv[3] = d[1] * guP[2] - d[2] * guP[1];
                    pv[4] = d[2] * guP[0] - d[0] * guP[2];
                    pv[5] = d[0] * guP[1] - d[1] * guP[0];
                }
            }
            reduce6(key, pv, A.gvel);
        }
    }
    // block sums of d/dg and d/dtau, one atomic per block and value
    const int warp = threadIdx.x >> 5;
    double v4[4] = {(double)gg[0], (double)gg[1], (double)gg[2], (double)gtau};
#pragma unroll
    for (int q = 0; q < 4; ++q)
        for (int o = 16; o > 0; o >>= 1) v4[q] += __shfl_down_sync(FULLMASK, v4[q], o);
    if (lane == 0)
#pragma unroll
        for (int q = 0; q < 4; ++q) s_red[warp][q] = v4[q];
    __syncthreads();
    if (threadIdx.x < 4) {
        double s = 0;
        for (int k = 0; k < ADJ_THREADS / 32; ++k) s += s_red[k][threadIdx.x];
        atomicAdd(A.gglob + threadIdx.x, s);
    }
}

// loss += sum_p w[p] . (F_p, T_p) for one step (ft: F (3 nslot) then T (3 nslot)).
__global__ void k_loss_step(const double* __restrict__ ft, const double* __restrict__ w, int n, int nslot,
                            double* __restrict__ loss) {
    double s = 0.0;
    for (int p = threadIdx.x; p < n; p += blockDim.x)
#pragma unroll
        for (int q = 0; q < 3; ++q)
            s += w[6 * (size_t)p + q] * ft[3 * (size_t)p + q] + w[6 * (size_t)p + 3 + q] * ft[3 * (size_t)nslot + 3 * (size_t)p + q];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(FULLMASK, s, o);
    __shared__ double part[32];
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0;
        for (int k = 0; k < (int)(blockDim.x >> 5); ++k) t += part[k];
        *loss += t;
    }
}

}  // namespace

template <typename T>
cudaError_t launch_adjoint_step(const AdjointArgs<T>& a, cudaStream_t s) {
    static std::atomic<int> cached[LBDEM_MAX_DEVICES];   // per device: grid size
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= LBDEM_MAX_DEVICES) return cudaErrorInvalidDevice;
    int blocks = cached[dev].load(std::memory_order_relaxed);
    if (blocks == 0) {
        int sms = 0, per_sm = 0;
        e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (e == cudaSuccess)
            e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_adjoint_step<T, false>, ADJ_THREADS, 0);
        if (e != cudaSuccess) return e;
        blocks = sms * (per_sm > 0 ? per_sm : 1);
        cached[dev].store(blocks, std::memory_order_relaxed);
    }
    const size_t need = (a.g.N + ADJ_THREADS - 1) / ADJ_THREADS;
    const unsigned grid = (unsigned)(need < (size_t)blocks ? (need > 0 ? need : 1) : (size_t)blocks);
    if (a.g.per[0] && a.g.per[1] && a.g.per[2])
        k_adjoint_step<T, true><<<grid, ADJ_THREADS, 0, s>>>(a);
    else
        k_adjoint_step<T, false><<<grid, ADJ_THREADS, 0, s>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_loss_step(const double* ft, const double* w, int n, int nslot, double* loss, cudaStream_t s) {
    k_loss_step<<<1, 256, 0, s>>>(ft, w, n, nslot, loss);
    return cudaGetLastError();
}

template cudaError_t launch_adjoint_step<float>(const AdjointArgs<float>&, cudaStream_t);
template cudaError_t launch_adjoint_step<double>(const AdjointArgs<double>&, cudaStream_t);

}  // namespace lbdem
