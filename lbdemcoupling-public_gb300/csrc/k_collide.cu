// K1: fused D3Q19 PSM collide-stream kernel with the per-particle force and
// torque reduction folded into the same pass.
//
// Replaces, per lattice step:
//   Palabos collideAndStream with IBcompositeDynamics<T,D3Q19>(BGK) in every
//   cell  -- src/ibCompositeDynamics3D.hh:130-203 (PSM collision, per-cell force)
//   SumForceTorque3D::process -- src/ibProcessors3D.hh:203-263 (sum F, r x F per id)
//
// Streaming is the in-place "AA" pattern on one population array:
//   even phase: cell x reads f_i from slot (i, x), writes f*_i to slot (opp i, x);
//   odd phase:  cell x reads f_i from slot (opp i, x - c_i), writes f*_i to slot
//               (i, x + c_i).
// Both phases read and write exactly the same set of slots per cell, so the
// update is race-free in place.  A neighbour beyond a wall (non-periodic axis)
// is replaced by the cell itself with the direction reversed: half-way
// bounce-back.  Periodic axes wrap.
//
// Lattices with 16-byte aligned rows and the FP64 form: persistent CTAs of 128 threads
// whose warps walk 64-cell z-segments.  The 19 population rows of a segment (plus, in the
// odd phase, the halo element of every c_z != 0 direction), the voxel words and
// (FP64 form, single lattice) the particle surface-velocity rows are staged in
// shared memory, double-buffered, so the next segment's bytes are in flight while the
// current one is collided: per-thread 16-byte cp.async with commit groups for
// the FP32 form, cp.async.bulk on an mbarrier for the FP64 form; rows that are not
// 16-byte aligned are copied in whole 16-byte chunks around the row (FP64, odd nz), or not
// staged at all (FP32, nz % 4 != 0: k_collide_direct, which also steps FP32 batches).  The
// staged pre-collision values double as fPre of the PSM update.  The FP32 form collides two cells per thread in packed
// f32x2 arithmetic (collide_segment_pairs) and recomputes the particle surface
// velocity of its solid cells from the owner particle's row of the float table
// (no per-cell velocity field); the FP64 form one cell per thread, BGK and solid
// correction in one pass in 64-bit fixed point (cell_fixed.h; a cell outside its range
// in double, collide_cell_fp64 or, with a body force, collide_cell), with the
// velocity setValues stored.  The same
// kernel steps many independent domains in one launch (batch mode).
#include "lbdem_internal.h"
#include "cell_fixed.h"

#include <cstddef>
#include <type_traits>

namespace lbdem {
namespace {

constexpr unsigned FULL = 0xffffffffu;

// 1/x (the FP64 form; the FP32 form uses __frcp_rn, identical to the IEEE division 1/x).
__device__ __forceinline__ double recip(double x) { return 1.0 / x; }

// c_i . (a, b, c) with the zero terms removed at compile time (0 * x is not
// foldable under IEEE rules, so the sum is built from the non-zero components).
template <typename T>
__device__ __forceinline__ T cdot(int i, T a, T b, T c) {
    const int X = cx(i), Y = cy(i), Z = cz(i);
    T r;
    if (X != 0) {
        r = X > 0 ? a : -a;
        if (Y != 0) r = Y > 0 ? r + b : r - b;
        if (Z != 0) r = Z > 0 ? r + c : r - c;
    } else if (Y != 0) {
        r = Y > 0 ? b : -b;
        if (Z != 0) r = Z > 0 ? r + c : r - c;
    } else if (Z != 0) {
        r = Z > 0 ? c : -c;
    } else {
        r = T(0);
    }
    return r;
}

template <typename T>
__device__ __forceinline__ void moments(const T (&f)[Q], T& rhoBar, T& jx, T& jy, T& jz) {
    rhoBar = ((f[0] + (f[1] + f[10])) + ((f[2] + f[11]) + (f[3] + f[12]))) +
             (((f[4] + f[13]) + (f[5] + f[14])) + ((f[6] + f[15]) + (f[7] + f[16]))) +
             ((f[8] + f[17]) + (f[9] + f[18]));
    jx = ((f[10] + f[13]) + (f[14] + f[15]) + f[16]) - ((f[1] + f[4]) + (f[5] + f[6]) + f[7]);
    jy = ((f[11] + f[13]) + (f[17] + f[18]) + f[5]) - ((f[2] + f[4]) + (f[8] + f[9]) + f[14]);
    jz = ((f[12] + f[15]) + (f[17] + f[7]) + f[9]) - ((f[3] + f[6]) + (f[8] + f[16]) + f[18]);
}

// Zeroth and first moments of a cell, rhoBar = sum f̄, j = sum c f̄, with 1/rho.
template <typename T>
struct Mom {
    T rhoBar, jx, jy, jz, invRho;
};

template <typename T>
__device__ __forceinline__ Mom<T> cell_moments(const T (&f)[Q]) {
    Mom<T> m;
    moments(f, m.rhoBar, m.jx, m.jy, m.jz);
    m.invRho = recip(T(1) + m.rhoBar);
    return m;
}

// BGK relaxation towards the second-order equilibrium
// feq_i = t_i [rhoBar + 3 c.j + invRho (4.5 (c.j)^2 - 1.5 j.j)], written per
// opposite pair (feq_i and feq_{i+9} differ only in the sign of 3 c.j), given
// the cell's pre-collision moments.
// With FORCE the Guo scheme is used (equilibrium momentum j + rho g / 2 plus
// the forcing term t_i (1 - omega/2) rho [3 (c - u).g + 9 (c.u)(c.g)]).
template <typename T, bool FORCE>
__device__ __forceinline__ void bgk(T (&f)[Q], const Mom<T>& m, T omega, T gx, T gy, T gz) {
    const T rhoBar = m.rhoBar, invRho = m.invRho;
    T jx = m.jx, jy = m.jy, jz = m.jz;
    const T rho = T(1) + rhoBar;
    if (FORCE) {
        const T h = T(0.5) * rho;
        jx += h * gx; jy += h * gy; jz += h * gz;
    }
    const T jSqr = jx * jx + jy * jy + jz * jz;
    const T base = rhoBar - T(1.5) * invRho * jSqr;
    const T om1 = T(1) - omega;
    const T q45 = T(4.5) * invRho;
    T ux = T(0), uy = T(0), uz = T(0), pre = T(0), ug = T(0);
    if (FORCE) {
        ux = jx * invRho; uy = jy * invRho; uz = jz * invRho;
        pre = (T(1) - T(0.5) * omega) * rho;
        ug = ux * gx + uy * gy + uz * gz;
    }
    f[0] = om1 * f[0] + (omega * T(wt(0))) * base;
    if (FORCE) f[0] += T(wt(0)) * pre * (T(-3) * ug);
#pragma unroll
    for (int i = 1; i <= 9; ++i) {
        const T cj = cdot(i, jx, jy, jz);
        const T ow = omega * T(wt(i));
        const T e = base + q45 * cj * cj;
        const T s = T(3) * cj;
        f[i] = om1 * f[i] + ow * (e + s);
        f[i + 9] = om1 * f[i + 9] + ow * (e - s);
        if (FORCE) {
            const T cu = cdot(i, ux, uy, uz);
            const T cg = cdot(i, gx, gy, gz);
            const T tp = T(wt(i)) * pre;
            // direction i: c = c_i ; direction i+9: c = -c_i
            f[i] += tp * (T(3) * (cg - ug) + T(9) * cu * cg);
            f[i + 9] += tp * (T(3) * (-cg - ug) + T(9) * cu * cg);
        }
    }
}

// Solid correction of a cell with n > 0 solid sub-cells,
// src/ibCompositeDynamics3D.hh:150-200.  On entry f holds the BGK
// post-collision state (fPre itself for n == 125, where B = 1 reduces the
// weighted update to fPre + bb exactly), m its moments, and pre(i) returns
// the pre-collision value fPre_i.  With feq (m) and the solid equilibrium
// feqS (rhoBar, uPart (1 + rhoBar)) written per opposite pair,
//   bb    = B ((fPre_o - feq_o) - (fPre_i - feqS_i)) = B (D + A + S)
//   bbOpp = B ((fPre_i - feq_i) - (fPre_o - feqS_o)) = B (A - D - S)
// with D = fPre_o - fPre_i, A = t_i (eS - eE), S = 3 t_i (c.j + c.uP), so the
// force term bb - bbOpp = 2 B (D + S).
template <typename T, typename Pre>
__device__ __forceinline__ void psm(T (&f)[Q], const Mom<T>& m, T up0, T up1, T up2, T B, const Pre& pre, T& Fx,
                                    T& Fy, T& Fz) {
    const T rhoBar = m.rhoBar, jx = m.jx, jy = m.jy, jz = m.jz, invRho = m.invRho;
    const T rho = T(1) + rhoBar;
    const T ux = up0 * rho, uy = up1 * rho, uz = up2 * rho;   // uPart (1 + rhoBar), :154
    const T q45 = T(4.5) * invRho;
    // eS - eE for c = 0: -1.5 invRho (uP^2 - j^2)
    const T dB = T(-1.5) * invRho * ((ux * ux + uy * uy + uz * uz) - (jx * jx + jy * jy + jz * jz));
    const T omB = T(1) - B;
    const T B2 = B + B;
    {
        const T p0 = pre(0);
        f[0] = p0 + omB * (f[0] - p0) - B * (T(wt(0)) * dB);   // B (feq_0 - feqS_0)
    }
    Fx = T(0); Fy = T(0); Fz = T(0);
#pragma unroll
    for (int i = 1; i <= 9; ++i) {
        const int o = i + 9;
        const T t = T(wt(i));
        const T cj = cdot(i, jx, jy, jz);
        const T cu = cdot(i, ux, uy, uz);
        const T A = t * (dB + q45 * ((cu - cj) * (cu + cj)));
        const T S = (T(3) * t) * (cj + cu);
        const T pi = pre(i), po = pre(o);
        const T D = po - pi;
        const T bb = B * (D + A + S);
        const T bbOpp = B * (A - D - S);
        f[i] = pi + omB * (f[i] - pi) + bb;
        f[o] = po + omB * (f[o] - po) + bbOpp;
        const T d = B2 * (D + S);                    // bb - bbOpp; F -= c_i (bb - bbOpp), :172-174
        if (cx(i) > 0) Fx -= d; else if (cx(i) < 0) Fx += d;
        if (cy(i) > 0) Fy -= d; else if (cy(i) < 0) Fy += d;
        if (cz(i) > 0) Fz -= d; else if (cz(i) < 0) Fz += d;
    }
}

// Collision of one cell with a body force given its pre-collision populations: BGK for
// every cell below full coverage (src/ibCompositeDynamics3D.hh:139-140), then the
// solid correction for cells with n > 0, with the moments of the post-collision
// populations (:146-148; the Guo force changes the momentum).  pre(i) returns fPre_i.
template <typename Pre>
__device__ __forceinline__ void collide_cell(double (&f)[Q], double omega, double gx, double gy, double gz, int n,
                                             double B, double up0, double up1, double up2, const Pre& pre,
                                             double (&F)[3]) {
    F[0] = F[1] = F[2] = 0.0;
    Mom<double> m = cell_moments(f);
    if (n < 125) bgk<double, true>(f, m, omega, gx, gy, gz);
    if (n > 0) {
        if (n < 125) m = cell_moments(f);
        psm<double>(f, m, up0, up1, up2, B, pre, F[0], F[1], F[2]);
    }
}

// ---------------------------------------------------------------------------
// FP64 form without a body force: the base BGK (src/ibCompositeDynamics3D.hh:139-140)
// and the solid correction (:150-200) of a cell in one pass over the opposite
// pairs (i = 1..9, k = i + 9, c_k = -c_i), written around the non-equilibrium
// parts g = fPre - feq.  With the solid equilibrium feqS at P = (1 + rhoBar) uPart
// (:154), Dl = feq - feqS and alpha = omega (1 - B) + B, the reference's
//   out = fPre + (1 - B)(fBGK - fPre) + bb,  fBGK = fPre - omega g,
// becomes
//   out_i = fPre_i - alpha g_i + B (g_k - Dl_i),   out_k = fPre_k - alpha g_k + B (g_i - Dl_k),
//   out_0 = fPre_0 - omega (1 - B) g_0 + B Dl_0     (the rest-population sign, :161, :185),
//   F -= c_i (bb - bbOpp) = c_k 2 B ((fPre_k - fPre_i) - 3 t c_k.(j + P))   (:172-174),
// where, with cj = c_k.j and cP = c_k.P,
//   feq_{k,i} = C +/- 3 t cj,  C = t (rhoBar + invRho (4.5 cj^2 - 1.5 j.j)),
//   Dl_{k,i} = Qd +/- 3 t (cj - cP),  Qd = t invRho (4.5 (cj - cP)(cj + cP) - 1.5 (j.j - P.P)),
//   Dl_0 = t_0 (-1.5 invRho (j.j - P.P)).
// n = 125 gives B = 1 (no BGK, alpha = 1), n = 0 gives B = 0 (the BGK result).
// The moments are those of fPre: without a body force BGK conserves them, and the
// reference's post-collision recomputation (:146-148) differs by rounding only.
// SOLID false (a warp without solid cells) leaves out the solid terms, 150 double operations
// instead of 270; a fluid cell gets the same bits either way, so results do not depend on
// which cells share a warp.
template <int AX>
__device__ __forceinline__ double pair_sum(const double (&d)[9]) {
    // sum_k c_k[AX] d[k - 10] over the directions k = 10..18 with c_k[AX] != 0, in k order
    double r = 0.0;
    bool any = false;
#pragma unroll
    for (int k = 10; k < Q; ++k) {
        const int c = AX == 0 ? cx(k) : (AX == 1 ? cy(k) : cz(k));
        if (c == 0) continue;
        const double v = d[k - 10];
        r = any ? (c > 0 ? r + v : r - v) : (c > 0 ? v : -v);
        any = true;
    }
    return r;
}

template <bool SOLID>
__device__ __forceinline__ void collide_cell_fp64(double (&f)[Q], double omega, double B, double up0, double up1,
                                                  double up2, double& Fx, double& Fy, double& Fz) {
    double d[9];
    double rhoBar;
    {
        double s[9];
#pragma unroll
        for (int i = 1; i <= 9; ++i) {
            s[i - 1] = f[i] + f[i + 9];
            d[i - 1] = f[i + 9] - f[i];
        }
        rhoBar = f[0] + ((((s[0] + s[1]) + (s[2] + s[3])) + ((s[4] + s[5]) + (s[6] + s[7]))) + s[8]);
    }
    const double jx = pair_sum<0>(d), jy = pair_sum<1>(d), jz = pair_sum<2>(d);
    const double invRho = recip(1.0 + rhoBar);
    const double jSqr = fma(jz, jz, fma(jy, jy, jx * jx));
    const double m15 = -1.5 * invRho;
    const double base = fma(m15, jSqr, rhoBar);
    double Px = 0.0, Py = 0.0, Pz = 0.0, dd = 0.0, alpha = omega, om1B = omega;
    if (SOLID) {
        const double rho = 1.0 + rhoBar;
        Px = up0 * rho; Py = up1 * rho; Pz = up2 * rho;
        const double PSqr = fma(Pz, Pz, fma(Py, Py, Px * Px));
        dd = m15 * (jSqr - PSqr);
        alpha = fma(B, 1.0 - omega, omega);
        om1B = omega * (1.0 - B);
    }
    {
        const double g0 = f[0] - wt(0) * base;
        f[0] = SOLID ? fma(B, wt(0) * dd, fma(-om1B, g0, f[0])) : fma(-omega, g0, f[0]);
    }
    double Ex = 0.0, Ey = 0.0, Ez = 0.0;
    bool fx0 = false, fy0 = false, fz0 = false;
#pragma unroll
    for (int k = 10; k < Q; ++k) {
        const int i = k - 9;
        const double t = wt(k), t3 = 3.0 * wt(k);
        const double a45 = (4.5 * wt(k)) * invRho;
        const double cj = cdot(k, jx, jy, jz);
        const double C = fma(a45 * cj, cj, t * base);
        const double Lj = t3 * cj;
        const double gi = (f[i] - C) + Lj;
        const double gk = (f[k] - C) - Lj;
        if (!SOLID) {
            f[i] = fma(-omega, gi, f[i]);
            f[k] = fma(-omega, gk, f[k]);
            continue;
        }
        const double cP = cdot(k, Px, Py, Pz);
        const double m = cj - cP, p = cj + cP;
        const double Qd = fma(a45 * m, p, t * dd);
        const double L = t3 * m;
        const double e = d[i - 1] - t3 * p;
        f[i] = fma(B, (gk - Qd) + L, fma(-alpha, gi, f[i]));
        f[k] = fma(B, (gi - Qd) - L, fma(-alpha, gk, f[k]));
        if (cx(k) != 0) { Ex = fx0 ? (cx(k) > 0 ? Ex + e : Ex - e) : (cx(k) > 0 ? e : -e); fx0 = true; }
        if (cy(k) != 0) { Ey = fy0 ? (cy(k) > 0 ? Ey + e : Ey - e) : (cy(k) > 0 ? e : -e); fy0 = true; }
        if (cz(k) != 0) { Ez = fz0 ? (cz(k) > 0 ? Ez + e : Ez - e) : (cz(k) > 0 ? e : -e); fz0 = true; }
    }
    const double B2 = B + B;
    Fx = SOLID ? B2 * Ex : 0.0;
    Fy = SOLID ? B2 * Ey : 0.0;
    Fz = SOLID ? B2 * Ez : 0.0;
}

// Per-cell force and torque added to the particle's sums (FP64 form): six
// double atomics per solid cell, resolved in L2 instead of a warp scan on the
// FP64 pipe.
__device__ __forceinline__ void add_cell_force(const CollideArgs<double>& a, int slot, const double (&v)[6]) {
    double* Fp = a.ft + 3 * (size_t)slot;
    double* Tp = a.ft + 3 * (size_t)a.nslot + 3 * (size_t)slot;
    atomicAdd(Fp + 0, v[0]); atomicAdd(Fp + 1, v[1]); atomicAdd(Fp + 2, v[2]);
    atomicAdd(Tp + 0, v[3]); atomicAdd(Tp + 1, v[4]); atomicAdd(Tp + 2, v[5]);
}

// ---------------------------------------------------------------------------
// FP32 form: two cells per thread in packed f32x2 arithmetic (sm_100 family
// add/sub/mul/fma .f32x2), the cells z and z + 1 of one row.  The same update as
// collide_cell, arranged per opposite pair around the direction k = i + 9 (every
// c_k has a non-negative first non-zero component, so c_k . v needs no
// negation), with two algebraically equal rewrites:
//   * the solid correction is applied as f + B ((fPre - f) + X), which leaves a
//     fluid cell (B = 0) exactly unchanged, so a pair mixing a fluid and a solid
//     cell runs it for both without a select;
//   * with the Guo force the solid correction's momentum is the BGK post-collision
//     momentum j + rho g (exact in arithmetic) instead of a second moment sum.
// Rounding differs from the FP64 form at the float level.
struct F2 {
    unsigned long long r;
};
__device__ __forceinline__ F2 pk(float a, float b) {
    F2 v;
    asm("mov.b64 %0, {%1, %2};" : "=l"(v.r) : "f"(a), "f"(b));
    return v;
}
__device__ __forceinline__ F2 bc(float a) { return pk(a, a); }
__device__ __forceinline__ float2 upk(F2 v) {
    float2 o;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(o.x), "=f"(o.y) : "l"(v.r));
    return o;
}
__device__ __forceinline__ F2 operator+(F2 a, F2 b) {
    F2 d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d.r) : "l"(a.r), "l"(b.r));
    return d;
}
__device__ __forceinline__ F2 operator-(F2 a, F2 b) {
    F2 d;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d.r) : "l"(a.r), "l"(b.r));
    return d;
}
__device__ __forceinline__ F2 operator*(F2 a, F2 b) {
    F2 d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d.r) : "l"(a.r), "l"(b.r));
    return d;
}
// a * b + c, one rounding
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) {
    F2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d.r) : "l"(a.r), "l"(b.r), "l"(c.r));
    return d;
}

// c_k . (a, b, c) for k >= 10 (first non-zero component of c_k is +1)
template <int K>
__device__ __forceinline__ F2 cdotk(F2 a, F2 b, F2 c) {
    constexpr int X = cx(K), Y = cy(K), Z = cz(K);
    static_assert(X > 0 || (X == 0 && (Y > 0 || (Y == 0 && Z > 0))), "direction with a negative lead");
    if constexpr (X != 0) {
        if constexpr (Y != 0) return Y > 0 ? a + b : a - b;
        else if constexpr (Z != 0) return Z > 0 ? a + c : a - c;
        else return a;
    } else if constexpr (Y != 0) {
        if constexpr (Z != 0) return Z > 0 ? b + c : b - c;
        else return b;
    } else {
        return c;
    }
}
// the same with uniform scalars
template <int K>
__device__ __forceinline__ float cdotk_s(float a, float b, float c) {
    return (float)cx(K) * a + (float)cy(K) * b + (float)cz(K) * c;
}

struct Mom2 {
    F2 rhoBar, jx, jy, jz, invRho;
};

__device__ __forceinline__ Mom2 moments2(const F2 (&f)[Q]) {
    Mom2 m;
    m.rhoBar = ((f[0] + (f[1] + f[10])) + ((f[2] + f[11]) + (f[3] + f[12]))) +
               (((f[4] + f[13]) + (f[5] + f[14])) + ((f[6] + f[15]) + (f[7] + f[16]))) +
               ((f[8] + f[17]) + (f[9] + f[18]));
    m.jx = ((f[10] + f[13]) + (f[14] + f[15]) + f[16]) - ((f[1] + f[4]) + (f[5] + f[6]) + f[7]);
    m.jy = ((f[11] + f[13]) + (f[17] + f[18]) + f[5]) - ((f[2] + f[4]) + (f[8] + f[9]) + f[14]);
    m.jz = ((f[12] + f[15]) + (f[17] + f[7]) + f[9]) - ((f[3] + f[6]) + (f[8] + f[16]) + f[18]);
    const float2 rb = upk(m.rhoBar);
    m.invRho = pk(__frcp_rn(1.f + rb.x), __frcp_rn(1.f + rb.y));
    return m;
}

template <bool FORCE>
__device__ __forceinline__ void bgk2(F2 (&f)[Q], const Mom2& m, float omega, float gx, float gy, float gz) {
    const F2 one = bc(1.f);
    const F2 rho = one + m.rhoBar, invRho = m.invRho;
    F2 jx = m.jx, jy = m.jy, jz = m.jz;
    if (FORCE) {
        const F2 h = bc(0.5f) * rho;
        jx = fma2(h, bc(gx), jx); jy = fma2(h, bc(gy), jy); jz = fma2(h, bc(gz), jz);
    }
    const F2 jSqr = fma2(jz, jz, fma2(jy, jy, jx * jx));
    const F2 base = fma2(bc(-1.5f) * invRho, jSqr, m.rhoBar);
    const F2 om1 = bc(1.f - omega);
    const F2 q45 = bc(4.5f) * invRho;
    F2 ux{}, uy{}, uz{}, pre{}, ug{};
    if (FORCE) {
        ux = jx * invRho; uy = jy * invRho; uz = jz * invRho;
        pre = bc(1.f - 0.5f * omega) * rho;
        ug = fma2(uz, bc(gz), fma2(uy, bc(gy), ux * bc(gx)));
    }
    f[0] = fma2(om1, f[0], bc(omega * (float)wt(0)) * base);
    if (FORCE) f[0] = f[0] - bc(3.f * (float)wt(0)) * (pre * ug);
    auto pair = [&](auto kc) {
        constexpr int k = decltype(kc)::value, i = k - 9;
        const F2 cj = cdotk<k>(jx, jy, jz);          // c_k . j = -c_i . j
        const F2 ow = bc(omega * (float)wt(k));
        const F2 e = fma2(q45 * cj, cj, base);
        const F2 s = bc(3.f) * cj;
        f[i] = fma2(om1, f[i], ow * (e - s));
        f[k] = fma2(om1, f[k], ow * (e + s));
        if (FORCE) {
            const F2 cu = cdotk<k>(ux, uy, uz);
            const float cg = cdotk_s<k>(gx, gy, gz);
            const F2 tp = bc((float)wt(k)) * pre;
            const F2 X = fma2(bc(9.f * cg), cu, bc(-3.f) * ug);
            f[i] = fma2(tp, X - bc(3.f * cg), f[i]);
            f[k] = fma2(tp, X + bc(3.f * cg), f[k]);
        }
    };
    pair(std::integral_constant<int, 10>{}); pair(std::integral_constant<int, 11>{});
    pair(std::integral_constant<int, 12>{}); pair(std::integral_constant<int, 13>{});
    pair(std::integral_constant<int, 14>{}); pair(std::integral_constant<int, 15>{});
    pair(std::integral_constant<int, 16>{}); pair(std::integral_constant<int, 17>{});
    pair(std::integral_constant<int, 18>{});
}

// Solid correction of both cells (a no-op for a cell with B = 0), with the
// momentum exchange accumulated in (Fx, Fy, Fz); pre(i) returns the pair's fPre_i.
template <typename Pre>
__device__ __forceinline__ void psm2(F2 (&f)[Q], F2 rhoBar, F2 jx, F2 jy, F2 jz, F2 invRho, F2 up0, F2 up1, F2 up2,
                                     F2 B, const Pre& pre, F2& Fx, F2& Fy, F2& Fz) {
    const F2 rho = bc(1.f) + rhoBar;
    const F2 ux = up0 * rho, uy = up1 * rho, uz = up2 * rho;
    const F2 q45 = bc(4.5f) * invRho;
    const F2 dB = (bc(-1.5f) * invRho) * (fma2(uz, uz, fma2(uy, uy, ux * ux)) - fma2(jz, jz, fma2(jy, jy, jx * jx)));
    {
        const F2 p0 = pre(0);
        f[0] = fma2(B, (p0 - f[0]) - bc((float)wt(0)) * dB, f[0]);
    }
    const F2 B2 = B + B;
    Fx = bc(0.f); Fy = bc(0.f); Fz = bc(0.f);
    auto pair = [&](auto kc) {
        constexpr int k = decltype(kc)::value, i = k - 9;
        const F2 t = bc((float)wt(k));
        const F2 cj = cdotk<k>(jx, jy, jz);
        const F2 cu = cdotk<k>(ux, uy, uz);
        const F2 A = t * fma2(q45, (cu - cj) * (cu + cj), dB);
        const F2 Sk = bc(3.f * (float)wt(k)) * (cj + cu);
        const F2 pi = pre(i), pkk = pre(k);
        const F2 E = (pkk - pi) - Sk;
        f[i] = fma2(B, (pi - f[i]) + (A + E), f[i]);
        f[k] = fma2(B, (pkk - f[k]) + (A - E), f[k]);
        const F2 d = B2 * E;                          // F += c_k (bb - bbOpp)
        if constexpr (cx(k) > 0) Fx = Fx + d;
        if constexpr (cy(k) > 0) Fy = Fy + d; else if constexpr (cy(k) < 0) Fy = Fy - d;
        if constexpr (cz(k) > 0) Fz = Fz + d; else if constexpr (cz(k) < 0) Fz = Fz - d;
    };
    pair(std::integral_constant<int, 10>{}); pair(std::integral_constant<int, 11>{});
    pair(std::integral_constant<int, 12>{}); pair(std::integral_constant<int, 13>{});
    pair(std::integral_constant<int, 14>{}); pair(std::integral_constant<int, 15>{});
    pair(std::integral_constant<int, 16>{}); pair(std::integral_constant<int, 17>{});
    pair(std::integral_constant<int, 18>{});
}

// bgk2 followed by psm2 in one pass over the opposite pairs (the same operations
// in the same order, so the same bits): the pre-collision pair is still in
// registers when its correction is applied, so fPre is not re-read.  Used with a
// body force for unaligned rows (batch); aligned rows keep the two passes, which
// measured faster there (without a body force both take collide_g2).  Per pair
// k = i + 9 (c_k = -c_i), with the solid
// equilibrium at P = (1 + rhoBar) uPart and fb the BGK result:
//   A = t (dB + 4.5 invRho ((c_k.P)^2 - (c_k.j)^2)),  S = 3 t c_k.(j + P),
//   E = (fPre_k - fPre_i) - S,
//   f_i = fb_i + B ((fPre_i - fb_i) + (A + E)),  f_k = fb_k + B ((fPre_k - fb_k) + (A - E)),
//   F += c_k 2 B E      (src/ibCompositeDynamics3D.hh:150-200, regrouped).  hs = (n < 125) rho
// per cell (FORCE: the solid correction's momentum j + hs g).  A cell with B = 0
// comes out exactly as bgk2 leaves it.
template <bool FORCE>
__device__ __forceinline__ void bgk_psm2(F2 (&f)[Q], const Mom2& m, float omega, float gx, float gy, float gz, F2 hs,
                                         F2 up0, F2 up1, F2 up2, F2 B, F2& Fx, F2& Fy, F2& Fz) {
    const F2 one = bc(1.f);
    const F2 rho = one + m.rhoBar, invRho = m.invRho;
    // BGK constants (bgk2)
    F2 jx = m.jx, jy = m.jy, jz = m.jz;
    if (FORCE) {
        const F2 h = bc(0.5f) * rho;
        jx = fma2(h, bc(gx), jx); jy = fma2(h, bc(gy), jy); jz = fma2(h, bc(gz), jz);
    }
    const F2 jSqr = fma2(jz, jz, fma2(jy, jy, jx * jx));
    const F2 base = fma2(bc(-1.5f) * invRho, jSqr, m.rhoBar);
    const F2 om1 = bc(1.f - omega);
    const F2 q45 = bc(4.5f) * invRho;
    F2 ux{}, uy{}, uz{}, pre{}, ug{};
    if (FORCE) {
        ux = jx * invRho; uy = jy * invRho; uz = jz * invRho;
        pre = bc(1.f - 0.5f * omega) * rho;
        ug = fma2(uz, bc(gz), fma2(uy, bc(gy), ux * bc(gx)));
    }
    // solid-correction constants
    F2 sjx = m.jx, sjy = m.jy, sjz = m.jz;
    if (FORCE) {
        sjx = fma2(hs, bc(gx), sjx); sjy = fma2(hs, bc(gy), sjy); sjz = fma2(hs, bc(gz), sjz);
    }
    const F2 rhoS = bc(1.f) + m.rhoBar;
    const F2 px = up0 * rhoS, py = up1 * rhoS, pz = up2 * rhoS;
    const F2 q45S = bc(4.5f) * invRho;
    const F2 dB = (bc(-1.5f) * invRho) * (fma2(pz, pz, fma2(py, py, px * px)) - fma2(sjz, sjz, fma2(sjy, sjy, sjx * sjx)));
    {
        const F2 p0 = f[0];
        F2 b0 = fma2(om1, f[0], bc(omega * (float)wt(0)) * base);
        if (FORCE) b0 = b0 - bc(3.f * (float)wt(0)) * (pre * ug);
        f[0] = fma2(B, (p0 - b0) - bc((float)wt(0)) * dB, b0);
    }
    const F2 B2 = B + B;
    Fx = bc(0.f); Fy = bc(0.f); Fz = bc(0.f);
    auto pair = [&](auto kc) {
        constexpr int k = decltype(kc)::value, i = k - 9;
        const F2 pi = f[i], pkk = f[k];
        // BGK of the pair
        const F2 cj = cdotk<k>(jx, jy, jz);
        const F2 ow = bc(omega * (float)wt(k));
        const F2 e = fma2(q45 * cj, cj, base);
        const F2 s = bc(3.f) * cj;
        F2 bi = fma2(om1, pi, ow * (e - s));
        F2 bk = fma2(om1, pkk, ow * (e + s));
        if (FORCE) {
            const F2 cu = cdotk<k>(ux, uy, uz);
            const float cg = cdotk_s<k>(gx, gy, gz);
            const F2 tp = bc((float)wt(k)) * pre;
            const F2 X = fma2(bc(9.f * cg), cu, bc(-3.f) * ug);
            bi = fma2(tp, X - bc(3.f * cg), bi);
            bk = fma2(tp, X + bc(3.f * cg), bk);
        }
        // solid correction of the pair
        const F2 t = bc((float)wt(k));
        const F2 cjS = cdotk<k>(sjx, sjy, sjz);
        const F2 cu = cdotk<k>(px, py, pz);
        const F2 A = t * fma2(q45S, (cu - cjS) * (cu + cjS), dB);
        const F2 Sk = bc(3.f * (float)wt(k)) * (cjS + cu);
        const F2 E = (pkk - pi) - Sk;
        f[i] = fma2(B, (pi - bi) + (A + E), bi);
        f[k] = fma2(B, (pkk - bk) + (A - E), bk);
        const F2 d = B2 * E;
        if constexpr (cx(k) > 0) Fx = Fx + d;
        if constexpr (cy(k) > 0) Fy = Fy + d; else if constexpr (cy(k) < 0) Fy = Fy - d;
        if constexpr (cz(k) > 0) Fz = Fz + d; else if constexpr (cz(k) < 0) Fz = Fz - d;
    };
    pair(std::integral_constant<int, 10>{}); pair(std::integral_constant<int, 11>{});
    pair(std::integral_constant<int, 12>{}); pair(std::integral_constant<int, 13>{});
    pair(std::integral_constant<int, 14>{}); pair(std::integral_constant<int, 15>{});
    pair(std::integral_constant<int, 16>{}); pair(std::integral_constant<int, 17>{});
    pair(std::integral_constant<int, 18>{});
}

// FP32 form without a body force: BGK and the solid correction of both cells
// in one pass, the formulation of collide_cell_fp64 in packed pairs (around
// g = fPre - feq; alpha = omega (1 - B) + B; see there).  fPre is f itself on
// entry, so nothing is re-read from the stage.  SOLID false (no solid cell in
// the warp) leaves out the solid terms; a fluid cell (B = 0, uP = 0) gets the
// same bits either way.
template <bool SOLID>
__device__ __forceinline__ void collide_g2(F2 (&f)[Q], const Mom2& m, float omega, F2 up0, F2 up1, F2 up2, F2 B,
                                           F2& Fx, F2& Fy, F2& Fz) {
    const F2 invRho = m.invRho;
    const F2 jSqr = fma2(m.jz, m.jz, fma2(m.jy, m.jy, m.jx * m.jx));
    const F2 m15 = bc(-1.5f) * invRho;
    const F2 base = fma2(m15, jSqr, m.rhoBar);
    const F2 nom = bc(-omega);
    F2 Px = bc(0.f), Py = bc(0.f), Pz = bc(0.f), dd = bc(0.f), nalpha = nom, nom1B = nom;
    if (SOLID) {
        const F2 rho = bc(1.f) + m.rhoBar;
        Px = up0 * rho; Py = up1 * rho; Pz = up2 * rho;
        const F2 PSqr = fma2(Pz, Pz, fma2(Py, Py, Px * Px));
        dd = m15 * (jSqr - PSqr);
        nalpha = fma2(B, bc(omega - 1.f), nom);     // -(omega (1 - B) + B)
        nom1B = fma2(B, bc(omega), nom);            // -omega (1 - B)
    }
    {
        const F2 g0 = f[0] - bc((float)wt(0)) * base;
        f[0] = SOLID ? fma2(B, bc((float)wt(0)) * dd, fma2(nom1B, g0, f[0])) : fma2(nom, g0, f[0]);
    }
    F2 Ex = bc(0.f), Ey = bc(0.f), Ez = bc(0.f);
    auto pair = [&](auto kc) {
        constexpr int k = decltype(kc)::value, i = k - 9;
        const F2 t = bc((float)wt(k)), t3 = bc(3.f * (float)wt(k));
        const F2 a45 = bc(4.5f * (float)wt(k)) * invRho;
        const F2 cj = cdotk<k>(m.jx, m.jy, m.jz);
        const F2 C = fma2(a45 * cj, cj, t * base);
        const F2 Lj = t3 * cj;
        const F2 gi = (f[i] - C) + Lj;
        const F2 gk = (f[k] - C) - Lj;
        if (SOLID) {
            const F2 cP = cdotk<k>(Px, Py, Pz);
            const F2 mm = cj - cP, pp = cj + cP;
            const F2 Qd = fma2(a45 * mm, pp, t * dd);
            const F2 L = t3 * mm;
            const F2 e = (f[k] - f[i]) - t3 * pp;
            f[i] = fma2(B, (gk - Qd) + L, fma2(nalpha, gi, f[i]));
            f[k] = fma2(B, (gi - Qd) - L, fma2(nalpha, gk, f[k]));
            if constexpr (cx(k) > 0) Ex = Ex + e;
            if constexpr (cy(k) > 0) Ey = Ey + e; else if constexpr (cy(k) < 0) Ey = Ey - e;
            if constexpr (cz(k) > 0) Ez = Ez + e; else if constexpr (cz(k) < 0) Ez = Ez - e;
        } else {
            f[i] = fma2(nom, gi, f[i]);
            f[k] = fma2(nom, gk, f[k]);
        }
    };
    pair(std::integral_constant<int, 10>{}); pair(std::integral_constant<int, 11>{});
    pair(std::integral_constant<int, 12>{}); pair(std::integral_constant<int, 13>{});
    pair(std::integral_constant<int, 14>{}); pair(std::integral_constant<int, 15>{});
    pair(std::integral_constant<int, 16>{}); pair(std::integral_constant<int, 17>{});
    pair(std::integral_constant<int, 18>{});
    const F2 B2 = B + B;
    Fx = B2 * Ex; Fy = B2 * Ey; Fz = B2 * Ez;
}

// float -> double by bit manipulation (exact for normal numbers; subnormal
// floats become signed zero).  Keeps the conversion off GB300's narrow FP64 pipe.
__device__ __forceinline__ double widen(float x) {
    const uint32_t b = __float_as_uint(x);
    const uint32_t s = b & 0x80000000u, e = (b >> 23) & 0xffu, m = b & 0x7fffffu;
    if (e == 0) return __hiloint2double((int)s, 0);
    const uint32_t ed = e == 0xffu ? 0x7ffu : e + 896u;   // rebias 127 -> 1023
    return __hiloint2double((int)(s | (ed << 20) | (m >> 3)), (int)(m << 29));
}

// Per-cell force and torque of a solid cell (SumForceTorque3D,
// src/ibProcessors3D.hh:203-263): particle slot of the owner tag and the
// terms F, r x F with the minimum-image arm of :230-243.  Returns the slot or -1.
// The terms F and r x F of a cell with arm (dx, dy, dz) before the minimum image
// (integer half extents of g, src/ibProcessors3D.hh:230-243).
template <typename T>
__device__ __forceinline__ void arm_terms(T dx, T dy, T dz, const Geom& g, T Fx, T Fy, T Fz, T (&v)[6]) {
    const int nx = g.nx, ny = g.ny, nz = g.nz;
    const int hx = nx / 2, hy = ny / 2, hz = nz / 2;
    // doubles are compared as integers (same order for a non-negative bound), off the
    // FP64 pipe
    auto above = [](T d, int h) -> bool {
        if constexpr (sizeof(T) == 8) return __double_as_longlong(d) > __double_as_longlong((double)h);
        else return d > T(h);
    };
    if (above(dx, hx)) dx -= T(nx); else if (above(-dx, hx)) dx += T(nx);
    if (above(dy, hy)) dy -= T(ny); else if (above(-dy, hy)) dy += T(ny);
    if (above(dz, hz)) dz -= T(nz); else if (above(-dz, hz)) dz += T(nz);
    v[0] = Fx; v[1] = Fy; v[2] = Fz;
    v[3] = dy * Fz - dz * Fy;
    v[4] = -dx * Fz + dz * Fx;
    v[5] = dx * Fy - dy * Fx;
}

__device__ __forceinline__ int cell_force_terms(const CollideArgs<double>& a, uint32_t w, int x, int y, int z,
                                                double Fx, double Fy, double Fz, double (&v)[6]) {
    if ((w & VOX_NMASK) == 0) return -1;
    const int tag = (int)(w >> VOX_NBITS);
    const int slot = tag <= a.max_tag ? __ldg(a.tag2slot + tag) : -1;
    if (slot < 0 || slot >= a.nslot) {
        atomicOr(a.err, 0x8u);   // LBDEM_DEVERR_UNMAPPED_TAG
        return -1;
    }
    const double* p = a.rec + (size_t)slot * REC_STRIDE;
    const double dx = (double)x - __ldg(p + 0), dy = (double)y - __ldg(p + 1), dz = (double)z - __ldg(p + 2);
    arm_terms(dx, dy, dz, a.g, Fx, Fy, Fz, v);
    return slot;
}

// Warp-segmented sum over runs of equal particle slot (consecutive cells along
// z mostly belong to the same sphere), one set of double atomics per run.
// Must be reached by all 32 lanes.
template <typename T>
__device__ __forceinline__ void reduce_forces(const CollideArgs<T>& a, int key, T (&v)[6]) {
    const unsigned solid = __ballot_sync(FULL, key >= 0);
    if (solid == 0u) return;
    const int lane = threadIdx.x & 31;
    const int first = __shfl_sync(FULL, key, __ffs(solid) - 1);
    if (__all_sync(FULL, key < 0 || key == first)) {
        // one particle in the group: butterfly sum, lane 0 adds
#pragma unroll
        for (int d = 16; d > 0; d >>= 1)
#pragma unroll
            for (int k = 0; k < 6; ++k) v[k] += __shfl_xor_sync(FULL, v[k], d);
        if (lane == 0) {
            double* Fp = a.ft + 3 * (size_t)first;
            double* Tp = a.ft + 3 * (size_t)a.nslot + 3 * (size_t)first;
            atomicAdd(Fp + 0, widen(v[0])); atomicAdd(Fp + 1, widen(v[1])); atomicAdd(Fp + 2, widen(v[2]));
            atomicAdd(Tp + 0, widen(v[3])); atomicAdd(Tp + 1, widen(v[4])); atomicAdd(Tp + 2, widen(v[5]));
        }
        return;
    }
    const int prevKey = __shfl_up_sync(FULL, key, 1);
    const bool head = (lane == 0) || (prevKey != key);
    const unsigned heads = __ballot_sync(FULL, head);
    const int segStart = 31 - __clz(heads & (FULL >> (31 - lane)));
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
#pragma unroll
        for (int k = 0; k < 6; ++k) {
            const T o = __shfl_up_sync(FULL, v[k], d);
            if (lane - d >= segStart) v[k] += o;
        }
    }
    const int nextKey = __shfl_down_sync(FULL, key, 1);
    const bool tail = (lane == 31) || (nextKey != key);
    if (tail && key >= 0) {
        double* Fp = a.ft + 3 * (size_t)key;
        double* Tp = a.ft + 3 * (size_t)a.nslot + 3 * (size_t)key;
        atomicAdd(Fp + 0, widen(v[0])); atomicAdd(Fp + 1, widen(v[1])); atomicAdd(Fp + 2, widen(v[2]));
        atomicAdd(Tp + 0, widen(v[3])); atomicAdd(Tp + 1, widen(v[4])); atomicAdd(Tp + 2, widen(v[5]));
    }
}

// FP32 form: force and torque of the cells of one row segment, reduced per run
// of equal owner (keyed by the owner's particle slot, which the cells' surface
// velocity already looked up).  Every cell of a
// particle lies within its radius of the particle's nearest image, so along a
// row the minimum-image arm of cell z is arm(zc) + (z - zc) e_z for any point
// zc of the segment (where the cells' nearest images differ, images_differ(), the arms are
// taken per cell), and
//   sum_cells arm x F = arm(zc) x sum F + sum (z - zc) e_z x F,
// with e_z x F = (-F_y, F_x, 0).  Per cell the kernel accumulates
// v = (F, -(z - zc) F_y, (z - zc) F_x); the lane that ends a run (the last
// lane of a run of equal slots, or the first solid lane when one slot covers the
// warp) takes the arm of its own cell zr from the particle's row,
// arm(zc) = arm(zr) - (zr - zc) e_z, and adds F and arm(zc) x F + (v3, v4, 0).
__device__ __forceinline__ void finish_run(const CollideArgs<float>& a, int slot, const float (&v)[5], int sx, int sy,
                                           int zr, int zc, const float4& rh, float rl0, float rl1, bool have) {
    // the lane's own table row when it is the run's owner's (loaded for the velocity)
    float4 h = rh, l = make_float4(rl0, rl1, 0.f, 0.f);
    if (!have) {
        const float4* p = reinterpret_cast<const float4*>(a.xpf + (size_t)slot * XPF_STRIDE);
        h = __ldg(p);
        l = __ldg(p + 1);
    }
    float dx = ((float)sx - h.x) - h.w;
    float dy = ((float)sy - h.y) - l.x;
    float dz = ((float)zr - h.z) - l.y;
    const int nx = a.g.nx, ny = a.g.ny, nz = a.g.nz;
    const int hx = nx / 2, hy = ny / 2, hz = nz / 2;
    if (dx > (float)hx) dx -= (float)nx; else if (dx < (float)-hx) dx += (float)nx;
    if (dy > (float)hy) dy -= (float)ny; else if (dy < (float)-hy) dy += (float)ny;
    if (dz > (float)hz) dz -= (float)nz; else if (dz < (float)-hz) dz += (float)nz;
    dz -= (float)(zr - zc);
    double* Fp = a.ft + 3 * (size_t)slot;
    double* Tp = a.ft + 3 * (size_t)a.nslot + 3 * (size_t)slot;
    // few lanes get here: the hardware conversion is cheaper than widen()
    atomicAdd(Fp + 0, (double)v[0]); atomicAdd(Fp + 1, (double)v[1]); atomicAdd(Fp + 2, (double)v[2]);
    atomicAdd(Tp + 0, (double)((dy * v[2] - dz * v[1]) + v[3]));
    atomicAdd(Tp + 1, (double)((dz * v[0] - dx * v[2]) + v[4]));
    atomicAdd(Tp + 2, (double)(dx * v[1] - dy * v[0]));
}

// Warp reduction of v over runs of equal key (owner slot, -1: no solid cell);
// zr is a cell of the lane's run.  Must be reached by all 32 lanes.
__device__ __forceinline__ void reduce_runs(const CollideArgs<float>& a, int key, float (&v)[5], int zr, int sx,
                                            int sy, int zc, const float4& rh, float rl0, float rl1, int rslot) {
    const unsigned solid = __ballot_sync(FULL, key >= 0);
    if (solid == 0u) return;
    const int lane = threadIdx.x & 31;
    const int lead = __ffs(solid) - 1;
    const int first = __shfl_sync(FULL, key, lead);
    if (__all_sync(FULL, key < 0 || key == first)) {
#pragma unroll
        for (int d = 16; d > 0; d >>= 1)
#pragma unroll
            for (int k = 0; k < 5; ++k) v[k] += __shfl_xor_sync(FULL, v[k], d);
        if (lane == lead) finish_run(a, first, v, sx, sy, zr, zc, rh, rl0, rl1, rslot == first);
        return;
    }
    const int prevKey = __shfl_up_sync(FULL, key, 1);
    const bool head = (lane == 0) || (prevKey != key);
    const unsigned heads = __ballot_sync(FULL, head);
    const int segStart = 31 - __clz(heads & (FULL >> (31 - lane)));
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
#pragma unroll
        for (int k = 0; k < 5; ++k) {
            const float o = __shfl_up_sync(FULL, v[k], d);
            if (lane - d >= segStart) v[k] += o;
        }
    }
    const int nextKey = __shfl_down_sync(FULL, key, 1);
    const bool tail = (lane == 31) || (nextKey != key);
    if (tail && key >= 0) finish_run(a, key, v, sx, sy, zr, zc, rh, rl0, rl1, rslot == key);
}

__device__ __forceinline__ int wrap_minus(int v, int n, int per) { return v > 0 ? v - 1 : (per ? n - 1 : -1); }
__device__ __forceinline__ int wrap_plus(int v, int n, int per) { return v < n - 1 ? v + 1 : (per ? 0 : -1); }
__device__ __forceinline__ int pick(int c, int m, int v, int p) { return c < 0 ? m : (c > 0 ? p : v); }

// ---------------------------------------------------------------------------
// Staged persistent kernel: every warp runs its own double-buffered pipeline
// over SEGW-cell z-segments (no block-wide barriers, so a warp with solid
// cells does not hold up the others).
constexpr int WARPS = COLLIDE_BLOCK / 32;    // warps per CTA
constexpr int DIRECT_BLOCK = 128;              // threads per CTA of k_collide_direct
constexpr int DIRECT_BLOCKS_PER_SM = 4;
// Per-CTA tables in dynamic shared memory behind the warps' stages.
// FP32 form, single lattice: a copy of the tag -> slot map when the tags fit below
// TAGMAP_SMEM - 1, holding -1 for a tag with no particle in the list and for every entry
// past max_tag (the last one included), so that a lookup is one shared load at
// min(tag, TAGMAP_SMEM - 1) with no tests between the cell's voxel word and the owner's
// table row; then B(n) (128 floats).
constexpr int TAGMAP_SMEM = 2048;
constexpr size_t TAGMAP_BYTES = sizeof(int) * TAGMAP_SMEM + sizeof(float) * 128;
// Batch mode: each CTA keeps the first segment of every domain in shared memory when
// there are at most SEG0_SMEM domains (the per-segment domain search reads it there).
constexpr int SEG0_SMEM = 2048;
constexpr size_t SEG0_BYTES = sizeof(int) * SEG0_SMEM;
constexpr int SEGW = COLLIDE_SEGW;          // cells per warp segment (2 per lane)
constexpr int WAIT_LIMIT = 1 << 22;         // bounded mbarrier wait (iterations of try_wait)
constexpr int PROBE_WAIT = 64;              // the timeout test hook's wait (iterations)

// Surface-velocity rows are staged by the FP64 form of a single lattice only.
template <typename T, bool BATCH>
__host__ __device__ constexpr bool stage_up() { return !BATCH && sizeof(T) == 8; }

// 16-byte aligned, so that every warp's stage (at warp * sizeof) keeps the bulk
// copies' shared-memory destinations on 16-byte boundaries.
template <typename T, bool STAGE_UP = true>
struct alignas(16) WarpStage {
    static constexpr int V = 16 / (int)sizeof(T);   // elements per 16 bytes
    static constexpr int UW = STAGE_UP ? SEGW + V : 1;
    static constexpr int W = SEGW + 2 * V;          // row: V halo | (lead) SEGW core | V halo
    T f[2][Q][W];
    uint32_t vox[2][SEGW + 4];
    T up[2][3][UW];        // particle surface velocity rows of the segment (when staged)
    long long row[2][sizeof(T) == 8 ? 9 : 1];   // FP64: element offset of row (x + dx, y + dy) at [3 (dx + 1) + dy + 1]; -1 beyond a wall
    T* out[2][sizeof(T) == 8 ? 3 * Q : Q + 1];   // output rows (see issue_segment, issue_segment_lsu)
    const T* src[sizeof(T) == 8 ? 1 : Q + 1];    // FP32: source rows of the segment being issued
    int geo[2][8];         // x, y, z0, len, domain, source rows inside, voxel lead of the segment in buffer b
    unsigned long long lead[2];   // unaligned rows: lead elements of row i at bits 2i, voxel row at bits 38,
                                  // surface-velocity row d at bits 40 + 2d
    unsigned long long bar[2];
};

static_assert(sizeof(WarpStage<float, true>) % 16 == 0 && sizeof(WarpStage<float, false>) % 16 == 0 &&
                  sizeof(WarpStage<double, true>) % 16 == 0 && sizeof(WarpStage<double, false>) % 16 == 0,
              "per-warp stages must keep 16-byte alignment");
static_assert(offsetof(WarpStage<float>, vox) % 16 == 0 && offsetof(WarpStage<float>, up) % 16 == 0 &&
                  offsetof(WarpStage<double>, vox) % 16 == 0 && offsetof(WarpStage<double>, up) % 16 == 0,
              "bulk-copy destinations on 16-byte boundaries");

// Where the FP32 form's per-CTA tables lie: behind the warps' stages.
constexpr size_t STAGED_TABLES = WARPS * sizeof(WarpStage<float, false>);

__host__ __device__ constexpr int row_slot(int dx, int dy) { return 3 * (dx + 1) + dy + 1; }

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(unsigned long long* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(unsigned long long* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void mbar_arrive(unsigned long long* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(unsigned long long* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_addr(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// Bounded wait: false if the phase did not complete within `limit` tries.
__device__ __forceinline__ bool mbar_wait(unsigned long long* bar, uint32_t parity, int limit = WAIT_LIMIT) {
    for (int k = 0; k < limit; ++k)
        if (mbar_try_wait(bar, parity)) return true;
    return false;
}
// Global -> shared bulk copy completing on an mbarrier (16-byte aligned, size % 16 == 0).
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes, unsigned long long* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_addr(dst)),
                 "l"(src), "r"(bytes), "r"(smem_addr(bar))
                 : "memory");
}

// Directions with c_z != 0 (they need a halo element in the odd phase).
constexpr uint32_t ZDIRS = 1u << 3 | 1u << 6 | 1u << 7 | 1u << 8 | 1u << 9 | 1u << 12 | 1u << 15 | 1u << 16 | 1u << 17 |
                           1u << 18;
__device__ __forceinline__ int zdir(int k) {
    // {3, 6, 7, 8, 9, 12, 15, 16, 17, 18} packed in 5-bit fields
    constexpr unsigned long long D = 3ull | 6ull << 5 | 7ull << 10 | 8ull << 15 | 9ull << 20 | 12ull << 25 |
                                     15ull << 30 | 16ull << 35 | 17ull << 40 | 18ull << 45;
    return (int)((D >> (5 * k)) & 31u);
}

struct SegGeo {
    int x, y, z0, len;
    int xm, xp, ym, yp;     // neighbour rows along x and y (-1: beyond a wall)
};

// dz divides by the z-segments per row, dy by ny (CollideArgs::dz, dy).  PER: all
// axes periodic (known at compile time).
template <bool PER = false>
__device__ __forceinline__ SegGeo seg_geo(const Geom& g, long long seg, const DivMagic& dz, const DivMagic& dy) {
    SegGeo s;
    // 32-bit arithmetic: a lattice holds fewer than 2^31 segments (launch checks)
    const unsigned sg = (unsigned)seg;
    const unsigned row = fast_div(sg, dz);
    const int zs = (int)(sg - row * dz.d);
    s.x = (int)fast_div(row, dy);
    s.y = (int)(row - (unsigned)s.x * dy.d);
    s.z0 = zs * SEGW;
    s.len = min(SEGW, g.nz - s.z0);
    s.xm = wrap_minus(s.x, g.nx, PER ? 1 : g.per[0]); s.xp = wrap_plus(s.x, g.nx, PER ? 1 : g.per[0]);
    s.ym = wrap_minus(s.y, g.ny, PER ? 1 : g.per[1]); s.yp = wrap_plus(s.y, g.ny, PER ? 1 : g.per[1]);
    return s;
}

// Row (x + dx, y + dy) as an element offset, or -1 beyond a wall.
template <bool PER = false>
__device__ __forceinline__ long long row_off(const Geom& g, const SegGeo& s, int dx, int dy) {
    const int X = pick(dx, s.xm, s.x, s.xp), Y = pick(dy, s.ym, s.y, s.yp);
    if (!PER && (X < 0 || Y < 0)) return -1;
    return ((long long)X * g.ny + Y) * g.nz;
}

// An 8-byte copy by this thread, counted on an mbarrier whose count has room for one
// arrival of each lane (cp_arrive).
__device__ __forceinline__ void cp8(void* dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_addr(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_arrive(unsigned long long* bar) {
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_addr(bar)) : "memory");
}

// FP64 form: issued by one warp for its segment into buffer b:
//   lanes 0..18:  population rows (even: own row, slot i; odd: row x - c_i,
//                 slot opp i, or own row slot i when that row is beyond a wall);
//   lanes 19..28: odd phase, aligned rows: the 16-byte chunk holding the halo
//                 element of the (lane-19)-th c_z != 0 direction;
//   lane 29:      voxel words of the segment (from the 16-byte boundary below; the lead
//                 is published);
//   lanes 29-31:  (second copy) the segment's particle surface-velocity rows.
// Odd phase, walls (not PER): what is half-way bounced back is staged where the cell
// looks for it, one place on along c_z: own rows of c_z != 0 directions whose source
// row lies beyond a wall, and the halo element at a z wall, with 8-byte copies (about one
// row in fifteen of a 60 x 60 section).  Telling the cases apart at every read and store
// instead cost a third more instructions than the even phase: 60x60x180 box with walls,
// odd phase 117 us, 92 so (even 79); periodic 128^3 suspension, whose stores now take
// their row from the table st.out, 397 to 359 us (even 322).
// MIS (rows not 16-byte aligned, odd nz, every batch): a row lies in the stage behind its
// lead, the elements between it and the 16-byte boundary below; the leads are published in
// st.lead.  Even phase: the copy starts at that boundary and is rounded up to whole chunks
// (the allocations carry 64 bytes of tail padding).  Odd phase: the halo elements lie where
// such chunks would write, so the whole chunks inside the row go out as a bulk copy, and
// its cut ends and the halo elements as 8-byte copies (put in place by hand after the copy,
// between the stage's two warps: 60x60x179 box, odd phase 98 us, 88 so).
// Lanes 0..9 also publish the segment geometry for the compute pass.
// Output rows of the odd phase, st.out: the value of direction opp(i) of cell z goes to
// [i] + z + c_z (the row that direction i was read from), at a z wall to [Q + i] + z (own
// row), and across the periodic z boundary to [2 Q + i] + the wrapped z + c_z.  For a row
// beyond a wall all three lead to slot i of the cell itself.
template <bool ODD, bool PER, bool MIS, bool STAGE_UP>
__device__ __forceinline__ void issue_segment(const CollideArgs<double>& a, WarpStage<double, STAGE_UP>& st, int b,
                                                long long seg, int dom) {
    using T = double;
    constexpr int V = WarpStage<T>::V;
    const int lane = threadIdx.x & 31;
    const Geom& g = a.g;
    const SegGeo s = seg_geo<PER>(g, seg, a.dz, a.dy);
    const size_t N = g.N;
    const long long own = ((long long)s.x * g.ny + s.y) * g.nz;
    if (lane < 9) st.row[b][lane] = row_off<PER>(g, s, lane / 3 - 1, lane % 3 - 1);

    if (lane == 9) {
        st.geo[b][0] = s.x; st.geo[b][1] = s.y; st.geo[b][2] = s.z0; st.geo[b][3] = s.len; st.geo[b][4] = dom;
    }
    const T* src = nullptr;
    void* dst = nullptr;
    uint32_t bytes = 0;
    uint32_t lead = 0;
    bool in = true;       // the lane's source row lies inside the lattice
    bool bounce = false;  // the lane's halo element is bounced back at a z wall
    if (lane < Q) {
        const int i = lane;
        const size_t slot = (size_t)i * N + (size_t)own;
        size_t off = slot;
        if (ODD && i != 0) {
            const long long r = row_off<PER>(g, s, -cx(i), -cy(i));
            in = PER || r >= 0;
            if (in) off = (size_t)opp(i) * N + (size_t)r;
        }
        if (ODD) {
            const int c = in ? 0 : cz(i);
            st.out[b][i] = a.fo + off + c;
            if (!PER) {
                st.out[b][Q + i] = a.fo + slot;
                st.out[b][2 * Q + i] = a.fo + off - c * (g.nz - 1);
            }
        }
        src = a.f + off + s.z0;
        dst = &st.f[b][i][V];
        if (MIS && !ODD) {
            lead = (uint32_t)(((uintptr_t)src & 15u) / sizeof(T));
            src -= lead;
            bytes = (uint32_t)(((lead + (uint32_t)s.len + V - 1) / V) * 16u);
        } else if (MIS && (in || cz(i) == 0)) {
            static_assert(V == 2, "a cut end is one element");
            lead = (uint32_t)(((uintptr_t)src & 15u) / sizeof(T));
            T* const cells = &st.f[b][i][V + lead];
            const int rest = s.len - (int)lead;
            if (lead) cp8(cells, src);
            if (rest & 1) cp8(cells + s.len - 1, src + s.len - 1);
            if (cz(i) != 0) {
                const int e = cz(i) > 0 ? 0 : s.len - 1;   // the cell that reads the halo element
                int zh = s.z0 + e - cz(i);
                if (zh < 0 || zh >= g.nz) zh = g.per[2] ? (zh < 0 ? g.nz - 1 : 0) : -1;
                cp8(cells + e - cz(i), zh >= 0 ? a.f + off + zh : a.f + slot + s.z0 + e);
            }
            src += lead;
            dst = cells + lead;
            bytes = (uint32_t)(rest / 2) * 16u;
        } else if (!MIS && (!ODD || PER || in || cz(i) == 0)) {
            bytes = (uint32_t)(s.len * sizeof(T));
        }
    } else if (ODD && !MIS && lane < Q + 10) {
        const int i = zdir(lane - Q);
        const long long r = row_off<PER>(g, s, -cx(i), -cy(i));
        if (PER || r >= 0) {
            int zc;      // first element of the 16-byte chunk (-1: beyond a z wall)
            if (cz(i) > 0) {
                zc = s.z0 - V;
                if (zc < 0) zc = PER || g.per[2] ? zc + g.nz : -1;
                dst = &st.f[b][i][0];
            } else {
                zc = s.z0 + s.len;
                if (zc >= g.nz) zc = PER || g.per[2] ? zc - g.nz : -1;
                dst = &st.f[b][i][V + s.len];
            }
            if (PER || zc >= 0) {
                src = a.f + (size_t)opp(i) * N + (size_t)r + zc;
                bytes = 16;
            } else {
                bounce = true;
            }
        }
    } else if (lane == Q + 10) {
        const uint32_t* vs = a.vox + own + s.z0;
        const uint32_t vlead = (uint32_t)(((uintptr_t)vs & 15u) / 4u);
        bytes = ((vlead + (uint32_t)s.len + 3u) / 4u) * 16u;
        src = reinterpret_cast<const T*>(vs - vlead);
        dst = &st.vox[b][0];
        st.geo[b][6] = (int)vlead;
    }
    // lanes 29, 30, 31: the surface-velocity rows (components 2, 0, 1) as a second copy
    const T* src2 = nullptr;
    void* dst2 = nullptr;
    uint32_t bytes2 = 0, lead2 = 0;
    const int ud = lane == Q + 10 ? 2 : lane - (Q + 11);
    if (STAGE_UP && lane >= Q + 10) {
        src2 = a.up + (size_t)ud * N + own + s.z0;
        dst2 = &st.up[b][ud][0];
        if (MIS) {
            lead2 = (uint32_t)(((uintptr_t)src2 & 15u) / sizeof(T));
            src2 -= lead2;
            bytes2 = (uint32_t)(((lead2 + (uint32_t)s.len + V - 1) / V) * 16u);
        } else {
            bytes2 = (uint32_t)(s.len * sizeof(T));
        }
    }
    if (MIS) {
        const uint32_t lo = __reduce_or_sync(FULL, lane < 16 ? lead << (2 * lane) : 0u);
        const uint32_t hi = __reduce_or_sync(FULL, ((lane >= 16 && lane < Q) ? lead << (2 * (lane - 16)) : 0u) |
                                                       ((STAGE_UP && lane >= Q + 10) ? lead2 << (8 + 2 * ud) : 0u));
        if (lane == 0) st.lead[b] = (unsigned long long)lo | ((unsigned long long)hi << 32);
    }
    if constexpr (ODD && !PER) {
        if (bounce) {
            const int i = zdir(lane - Q);
            if (cz(i) > 0) cp8(&st.f[b][i][V - 1], a.f + (size_t)i * N + (size_t)own);
            else cp8(&st.f[b][i][V + s.len], a.f + (size_t)i * N + (size_t)own + (g.nz - 1));
        }
        for (unsigned m = ~__ballot_sync(FULL, in) & ZDIRS; m; m &= m - 1u) {
            const int i = __ffs(m) - 1;
            const T* p = a.f + (size_t)i * N + (size_t)own + s.z0;
            for (int j = lane; j < s.len; j += 32) cp8(&st.f[b][i][V - cz(i) + j], p + j);
        }
        cp_arrive(&st.bar[b]);
    }
    const uint32_t total = __reduce_add_sync(FULL, bytes + bytes2);
    __syncwarp();   // the lanes' geometry writes come before lane 0's arrival
    if (lane == 0) mbar_arrive_expect_tx(&st.bar[b], total);
    __syncwarp();
    if (bytes) bulk_g2s(dst, src, bytes, &st.bar[b]);
    if (bytes2) bulk_g2s(dst2, src2, bytes2, &st.bar[b]);
}

// ---------------------------------------------------------------------------
// Staging of aligned rows (nz % 4 == 0) with per-thread 16-byte cp.async
// through the load/store path: a segment's rows go out as many small copies
// (19 population rows, the voxel row, the surface-velocity rows and up to 10
// halo chunks), and bulk copies of that size are bounded by the per-operation
// rate of the bulk-copy unit rather than by DRAM.  Completion is tracked per
// thread with commit groups (one group per segment).
__device__ __forceinline__ void cp16(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int P>
__device__ __forceinline__ void cp_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(P) : "memory");
}

template <typename Fn, int... Ts>
__device__ __forceinline__ void unroll_seq(std::integer_sequence<int, Ts...>, Fn&& fn) {
    (fn(std::integral_constant<int, Ts>{}), ...);
}

// The rows' addresses are formed once per segment, by one lane each, and kept in shared
// memory: st.src[i] is the segment's source row of direction i (even: slot i of the own
// row; odd: slot opp i of row x - c_i, or slot i of the own row beyond a wall), and
// st.out[b][i] the same row of the output, which is where the value of direction opp(i)
// goes.  (A copy or store then takes one shared load and one multiply-add.  With the
// addresses formed at each of them a periodic 256^3 suspension took 445 / 545 us, even /
// odd phase; so 433 / 530.)
template <typename T, bool ODD, bool PER, bool STAGE_UP>
__device__ __forceinline__ void issue_segment_lsu(const CollideArgs<T>& a, WarpStage<T, STAGE_UP>& st, int b,
                                                  long long seg) {
    constexpr int V = WarpStage<T>::V;   // elements per 16-byte chunk
    constexpr int CPR = SEGW / V;        // chunks per row of a segment
    constexpr int RPI = 32 / CPR;        // rows per warp pass
    static_assert(CPR * RPI == 32, "a warp pass covers whole rows");
    const int lane = threadIdx.x & 31;
    const Geom& g = a.g;
    const SegGeo s = seg_geo<PER>(g, seg, a.dz, a.dy);
    const size_t N = g.N;
    const size_t own = ((size_t)s.x * g.ny + s.y) * g.nz;
    bool in = true;   // the lane's source row lies inside the lattice
    if (lane < Q) {
        const int i = lane;
        size_t off = (size_t)i * N + own;
        if (ODD && i != 0) {
            const long long r = row_off<PER>(g, s, -cx(i), -cy(i));
            in = PER || r >= 0;
            if (in) off = (size_t)opp(i) * N + (size_t)r;
        }
        st.src[i] = a.f + off + s.z0;
        st.out[b][i] = a.fo + off + s.z0;
    }
    if (lane == Q) {
        st.geo[b][0] = s.x; st.geo[b][1] = s.y; st.geo[b][2] = s.z0; st.geo[b][3] = s.len;
    }
    if (ODD && !PER) {
        const unsigned rows = __ballot_sync(FULL, in);
        if (lane == 0) st.geo[b][5] = (int)rows;
    }
    __syncwarp();
    const int c = lane % CPR, sub = lane / CPR;
    const bool cin = c * V < s.len;   // rows of aligned lattices end on a chunk boundary
    // population rows: pass t covers directions t * RPI + sub
#pragma unroll
    for (int t = 0; t < (Q + RPI - 1) / RPI; ++t) {
        const int i = t * RPI + sub;
        if (cin && (RPI * (t + 1) <= Q || i < Q)) cp16(&st.f[b][i][V + c * V], st.src[i] + c * V);
    }
    // then: voxel row (SEGW / 4 chunks), surface-velocity rows (3 CPR), halo chunks
    // (odd phase, 10) -- in that order, so that only the first pass mixes two kinds
    constexpr int NH = ODD ? 10 : 0, NV = SEGW / 4, NU = STAGE_UP ? 3 * CPR : 0;
    constexpr int NX = NH + NV + NU;
#pragma unroll
    for (int kk = lane; kk < ((NX + 31) / 32) * 32; kk += 32) {
        // item order voxel, velocity, halo, mapped onto the halo-first numbering below
        const int k = kk < NV + NU ? kk + NH : kk - (NV + NU);
        if (kk >= NX) continue;
        if (k < NH) {
            const int i = zdir(k);
            if (!PER && row_off(g, s, -cx(i), -cy(i)) < 0) continue;
            int zc;     // first element of the chunk holding the halo (-1: beyond a z wall)
            T* dst;
            if (cz(i) > 0) {
                zc = s.z0 - V;
                if (zc < 0) zc = (PER || g.per[2]) ? zc + g.nz : -1;
                dst = &st.f[b][i][0];
            } else {
                zc = s.z0 + s.len;
                if (zc >= g.nz) zc = (PER || g.per[2]) ? zc - g.nz : -1;
                dst = &st.f[b][i][V + s.len];
            }
            if (zc >= 0) cp16(dst, st.src[i] + (zc - s.z0));
        } else if (k < NH + NV) {
            const int cv = k - NH;
            if (cv * 4 < s.len) cp16(&st.vox[b][cv * 4], a.vox + own + s.z0 + cv * 4);
        } else if (k < NX) {
            const int u = k - NH - NV, d = u / CPR, cu = u % CPR;
            if (STAGE_UP && cu * V < s.len)
                cp16(&st.up[b][d][cu * V], a.up + (size_t)d * N + own + s.z0 + cu * V);
        }
    }
    cp_commit();
}

// The FP32 form's per-CTA tables (see TAGMAP_SMEM), OFF bytes into dynamic shared
// memory; NO_TABLES: none, B(n) and the map are read from global memory.  (Addressed from
// the array itself: through a stored pointer the compiler takes generic loads.)
constexpr size_t NO_TABLES = ~(size_t)0;
template <size_t OFF>
struct PairTables {
    bool map;   // the tags fit the copy of the map
    __device__ __forceinline__ static int* base() {
        extern __shared__ __align__(16) unsigned char smem_raw[];
        return reinterpret_cast<int*>(smem_raw + OFF);
    }
    __device__ __forceinline__ static float* btab() { return reinterpret_cast<float*>(base() + TAGMAP_SMEM); }
    // Filled by the CTA's threads (TAGMAP_BYTES); the caller synchronizes.
    __device__ __forceinline__ void load(const CollideArgs<float>& a) {
        map = a.max_tag < TAGMAP_SMEM - 1;
        if (map)
            for (int k = threadIdx.x; k < TAGMAP_SMEM; k += blockDim.x) {
                const int v = k <= a.max_tag ? __ldg(a.tag2slot + k) : -1;
                base()[k] = (v >= 0 && v < a.nslot) ? v : -1;
            }
        for (int k = threadIdx.x; k < 126; k += blockDim.x) btab()[k] = __ldg(a.btab + k);
    }
};
// What the collision of a lane's two cells leaves for the force sums: the momentum
// exchange, the owners' slots (-1: none) and the centre part of the table row that the
// velocity lookup read (slot vslot).
struct PairForce {
    F2 Fx, Fy, Fz;
    int s0, s1, vslot;
    bool unmapped;   // a solid cell whose tag names no particle (reported, left out of the sums)
    float4 rh;
    float rl0, rl1;
};

// Collision of a lane's two cells (x, ya, za) and (x, yb, zb) with the voxel words w0,
// w1 (0 for a lane slot without a cell): f in, f out, for k_collide_direct.  The same
// operations as in collide_segment_pairs, so a cell gets the same bits in both.
// BGK runs for every cell, the fully covered ones included (their solid correction with
// B = 1 returns fPre + bb up to rounding), so that a cell's result does not depend on the
// cell it is paired with; the solid terms run in warps that hold a solid cell.  Must be
// reached by all 32 lanes.
template <bool FORCE, size_t OFF>
__device__ __forceinline__ void collide_pair(const CollideArgs<float>& a, const Geom& g, const PairTables<OFF>& tb,
                                             F2 (&f)[Q], uint32_t w0, uint32_t w1, int x, int ya, int za, int yb,
                                             int zb, PairForce& o) {
    const int n0 = min((int)(w0 & VOX_NMASK), 125), n1 = min((int)(w1 & VOX_NMASK), 125);
    const F2 B = OFF != NO_TABLES ? pk(tb.btab()[n0], tb.btab()[n1]) : pk(__ldg(a.btab + n0), __ldg(a.btab + n1));
    const Mom2 m = moments2(f);
    o.Fx = o.Fy = o.Fz = bc(0.f);
    o.s0 = o.s1 = o.vslot = -1;
    o.unmapped = false;
    o.rh = make_float4(0.f, 0.f, 0.f, 0.f);
    o.rl0 = o.rl1 = 0.f;
    // owner slots (from the CTA's shared copy of the map when it has one)
    auto owner = [&](uint32_t w) -> int {
        const int tag = (int)(w >> VOX_NBITS);
        if (OFF != NO_TABLES && tb.map) return tb.base()[min(tag, TAGMAP_SMEM - 1)];
        // global map: an unconditional load at the clamped tag, tested afterwards
        const int slot = __ldg(a.tag2slot + min(tag, a.max_tag));
        return (tag <= a.max_tag && slot >= 0 && slot < a.nslot) ? slot : -1;
    };
    o.s0 = n0 > 0 ? owner(w0) : -1;
    o.s1 = n1 > 0 ? owner(w1) : -1;
    // particle surface velocity of the lane's solid cells, recomputed from the owner
    // particle's row of the float table (one row when both cells belong to the same
    // particle); every lane of the warp loads a row (slot 0 for a lane without a solid
    // cell, whose velocities stay zero): no branch ahead of the load
    F2 u0 = bc(0.f), u1 = bc(0.f), u2 = bc(0.f);
    auto solid_velocity = [&]() {
        float ua[3] = {0.f, 0.f, 0.f}, ub[3] = {0.f, 0.f, 0.f};
        const int sl = o.s0 >= 0 ? o.s0 : o.s1;
        {
            const TableRow r = load_row(a.xpf, max(sl, 0));
            o.rh = r.a;
            o.rl0 = r.b.x;
            o.rl1 = r.b.y;
            o.vslot = sl;
            const RowPart rp = row_part(r, x, ya, g);
            if (o.s0 >= 0) cell_part(r, rp, za, g, ua[0], ua[1], ua[2]);
            if (sl >= 0 && o.s1 == sl) {
                if (yb != ya) cell_part(r, row_part(r, x, yb, g), zb, g, ub[0], ub[1], ub[2]);
                else cell_part(r, rp, zb, g, ub[0], ub[1], ub[2]);
            }
        }
        if (o.s1 >= 0 && o.s1 != sl) row_velocity(load_row(a.xpf, o.s1), x, yb, zb, g, ub[0], ub[1], ub[2]);
        u0 = pk(ua[0], ub[0]);
        u1 = pk(ua[1], ub[1]);
        u2 = pk(ua[2], ub[2]);
    };
    // FORCE: the solid correction's momentum is the BGK post-collision one, j + rho g,
    // for the cells that ran BGK
    auto hsol = [&]() -> F2 {
        return pk(n0 < 125 ? 1.f : 0.f, n1 < 125 ? 1.f : 0.f) * (bc(1.f) + m.rhoBar);
    };
    if (__any_sync(FULL, n0 > 0 || n1 > 0)) {   // one pass
        solid_velocity();
        if constexpr (FORCE)
            bgk_psm2<FORCE>(f, m, a.omega, a.g3[0], a.g3[1], a.g3[2], hsol(), u0, u1, u2, B, o.Fx, o.Fy, o.Fz);
        else
            collide_g2<true>(f, m, a.omega, u0, u1, u2, B, o.Fx, o.Fy, o.Fz);
    } else {
        if constexpr (FORCE) bgk2<FORCE>(f, m, a.omega, a.g3[0], a.g3[1], a.g3[2]);
        else collide_g2<false>(f, m, a.omega, u0, u1, u2, B, o.Fx, o.Fy, o.Fz);
    }
    o.unmapped = (n0 > 0 && o.s0 < 0) || (n1 > 0 && o.s1 < 0);
}

// Force and torque of a lane's two cells with per-cell arms (cells of one owner may lie in
// several rows, or wrap around a periodic row), reduced over the warp per run of equal
// owner; v0, v1: the lane slots that hold a cell.  Must be reached by all 32 lanes.
__device__ __forceinline__ void forces_by_cell(const CollideArgs<float>& a, const Geom& g, const PairForce& o,
                                               int x, int ya, int za, int yb, int zb, bool apart) {
    if (o.unmapped) atomicOr(a.err, 0x8u);   // LBDEM_DEVERR_UNMAPPED_TAG
    const int ka = o.s0, kb = o.s1;
    if (!__any_sync(FULL, ka >= 0 || kb >= 0)) return;
    const float2 fx = upk(o.Fx), fy = upk(o.Fy), fz = upk(o.Fz);
    auto terms = [&](int slot, int y, int z, float cfx, float cfy, float cfz, float (&v)[6]) {
        float4 h = o.rh;
        float lx = o.rl0, lz = o.rl1;
        if (slot != o.vslot) {
            const float4* p = reinterpret_cast<const float4*>(a.xpf + (size_t)slot * XPF_STRIDE);
            h = __ldg(p);
            const float4 l = __ldg(p + 1);
            lx = l.x;
            lz = l.y;
        }
        // centre = hi + lo in float: (x - hi) - lo is the arm to ~1 ulp
        arm_terms(((float)x - h.x) - h.w, ((float)y - h.y) - lx, ((float)z - h.z) - lz, g, cfx, cfy, cfz, v);
    };
    float va[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f}, vb[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    if (ka >= 0) terms(ka, ya, za, fx.x, fy.x, fz.x, va);
    if (kb >= 0) terms(kb, yb, zb, fx.y, fy.y, fz.y, vb);
    const bool one = !apart && __all_sync(FULL, ka < 0 || kb < 0 || ka == kb);   // one reduction for both cells
    if (one) {
#pragma unroll
        for (int q = 0; q < 6; ++q) va[q] += vb[q];
    }
#pragma unroll 1
    for (int pass = 0; pass < (one ? 1 : 2); ++pass) {   // a single reduction site, as below
        float v[6];
#pragma unroll
        for (int q = 0; q < 6; ++q) v[q] = pass == 0 ? va[q] : vb[q];
        reduce_forces(a, pass == 0 ? (one && ka < 0 ? kb : ka) : kb, v);
    }
}
// Force and torque of the two cells of a lane in one row segment, reduced per run of
// equal owner (finish_run), arms from the segment's middle point zc; the two cells go
// through one warp reduction when their owners agree.  Must be reached by all 32 lanes.
__device__ __forceinline__ void forces_by_run(const CollideArgs<float>& a, const PairForce& o, int x, int ya, int yb,
                                              int zc, int za, int zb, bool apart) {
    if (o.unmapped) atomicOr(a.err, 0x8u);   // LBDEM_DEVERR_UNMAPPED_TAG
    const int ka = o.s0, kb = o.s1;
    if (!__any_sync(FULL, ka >= 0 || kb >= 0)) return;
    const float2 fx = upk(o.Fx), fy = upk(o.Fy), fz = upk(o.Fz);
    const float da = (float)(za - zc), db = (float)(zb - zc);
    float va[5] = {fx.x, fy.x, fz.x, -da * fy.x, da * fx.x};
    float vb[5] = {fx.y, fy.y, fz.y, -db * fy.y, db * fx.y};
#pragma unroll
    for (int q = 0; q < 5; ++q) {
        if (ka < 0) va[q] = 0.f;
        if (kb < 0) vb[q] = 0.f;
    }
    const bool one = !apart && __all_sync(FULL, ka < 0 || kb < 0 || ka == kb);   // one reduction for both cells
    if (one) {
#pragma unroll
        for (int q = 0; q < 5; ++q) va[q] += vb[q];
    }
    // a single reduction site (the batch kernels' loop bodies are large enough for
    // instruction-cache misses to cost more than the loop)
#pragma unroll 1
    for (int pass = 0; pass < (one ? 1 : 2); ++pass) {
        float v[5];
#pragma unroll
        for (int q = 0; q < 5; ++q) v[q] = pass == 0 ? va[q] : vb[q];
        const bool second = pass == 1 || (one && ka < 0);   // the run's cells are the b cells
        reduce_runs(a, second ? kb : ka, v, second ? zb : za, x, second ? yb : ya, zc, o.rh, o.rl0, o.rl1, o.vslot);
    }
}
// Whether a segment of len cells can hold cells of one particle whose arms take the minimum
// image (integer half extent) differently: across the periodic boundary the two ends of a
// chord are nz less the chord apart, so there are solid cells that far apart, and between
// walls an arm has to exceed half the row.  s: an owner slot of the lane (-1: none), whose
// cells are j = 2 l, 2 l + 1 (ADJ) or l, l + 32.  Must be reached by all 32 lanes.
// (Registers, launch constants and two votes only: a load from the batch's table here took
// 1 % of the time of 512 channels.)
template <bool ADJ>
__device__ __forceinline__ bool images_can_differ(const Geom& g, int reach, int len, int s) {
    const int j = ADJ ? 2 * (threadIdx.x & 31) : threadIdx.x & 31;
    const int apart = g.per[2] ? g.nz - 2 * reach : (g.nz / 2 < reach ? 0 : len);
    return len > apart && __any_sync(FULL, s >= 0 && j < len - apart) &&
           __any_sync(FULL, s >= 0 && j >= apart - (ADJ ? 1 : 32));
}
// Whether they do.  Out of line; must be reached by all 32 lanes.
__device__ __noinline__ bool images_differ(const CollideArgs<float>& a, int s0, int s1, int vslot, float zh, float zl,
                                           int za, int zb) {
    const float half = (float)(a.g.nz / 2);
    auto image = [&](int slot, int z) -> int {
        if (slot < 0) return 0;
        float h = zh, l = zl;   // the centre's z in the row that the velocity lookup read
        if (slot != vslot) {
            const float* p = a.xpf + (size_t)slot * XPF_STRIDE;
            h = __ldg(p + 2);
            l = __ldg(p + 5);
        }
        const float d = ((float)z - h) - l;
        return d > half ? 1 : (d < -half ? -1 : 0);
    };
    const int i0 = image(s0, za), i1 = image(s1, zb);
    unsigned m0 = __ballot_sync(FULL, i0 != 0), m1 = __ballot_sync(FULL, i1 != 0);
    while (m0 | m1) {   // one particle at a time: its cells have the image of its first one
        const int lead = __ffs(m0 ? m0 : m1) - 1;
        const int slot = __shfl_sync(FULL, m0 ? s0 : s1, lead), first = __shfl_sync(FULL, m0 ? i0 : i1, lead);
        if (__any_sync(FULL, (s0 == slot && i0 != first) || (s1 == slot && i1 != first))) return true;
        m0 &= ~__ballot_sync(FULL, s0 == slot);
        m1 &= ~__ballot_sync(FULL, s1 == slot);
    }
    return false;
}
// forces_by_cell out of line, for the rare segments of the row kernels.
__device__ __noinline__ void forces_by_cell_far(const CollideArgs<float>& a, PairForce o, int x, int ya, int za,
                                                int yb, int zb, bool apart) {
    forces_by_cell(a, a.g, o, x, ya, za, yb, zb, apart);
}

// FP32 compute pass over one staged segment of a lattice with 16-byte aligned rows, two
// cells per lane in packed pairs: lane l takes the adjacent cells j = 2 l, 2 l + 1,
// whose staged values and destination slots are 8-byte aligned pairs, so loads
// and stores are 64-bit (in the odd phase the c_z != 0 directions land one slot
// over and are moved one lane over with a shuffle).
// Force and torque are reduced per run of equal owner (reduce_runs); the two
// cells of a lane go through one warp reduction when their owners agree.
template <bool ODD, bool FORCE, bool PER, bool STAGE_UP>
__device__ __forceinline__ void collide_segment_pairs(const CollideArgs<float>& a, WarpStage<float, STAGE_UP>& st,
                                                      int b, int sx, int sy, int z0, int len, uint32_t srcrow,
                                                      const PairTables<STAGED_TABLES>& tb) {
    constexpr int V = WarpStage<float>::V;
    const int lane = threadIdx.x & 31;
    const Geom& g = a.g;
    const size_t N = g.N;
    const int j0 = 2 * lane, j1 = j0 + 1;
    const bool v0 = j0 < len, v1 = j1 < len;
    const int za = z0 + j0, zb = z0 + j1;

    // staged values of direction i for the lane's two cells
    auto at2 = [&](int i) -> F2 {
        const int shift = (ODD && cz(i) != 0 && (PER || ((srcrow >> i) & 1u))) ? cz(i) : 0;
        const float* p = &st.f[b][i][V - shift];
        if ((shift & 1) == 0) {
            const float2 t = *reinterpret_cast<const float2*>(p + j0);
            return pk(t.x, t.y);
        }
        return pk(p[j0], p[j1]);
    };
    F2 f[Q];
#pragma unroll
    for (int i = 0; i < Q; ++i) f[i] = at2(i);
    const uint32_t w0 = v0 ? st.vox[b][j0] : 0u, w1 = v1 ? st.vox[b][j1] : 0u;
    const int n0 = min((int)(w0 & VOX_NMASK), 125), n1 = min((int)(w1 & VOX_NMASK), 125);
    const F2 B = pk(tb.btab()[n0], tb.btab()[n1]);

    // BGK runs for every cell, the fully covered ones included (their solid
    // correction with B = 1 returns fPre + bb up to rounding), so that a cell's
    // result does not depend on the cell it is paired with.
    const Mom2 m = moments2(f);
    F2 Fx = bc(0.f), Fy = bc(0.f), Fz = bc(0.f);
    // particle surface velocity of the lane's solid cells, recomputed from the
    // owner particle's row of the float table (one row when both cells belong to
    // the same particle), read after the BGK arithmetic.  (Looking the owners up
    // before the moment sums, or prefetching the rows, measured slower.)
    // owner slots (from the CTA's shared copy of the map when it has one)
    auto owner = [&](uint32_t w) -> int {
        const int tag = (int)(w >> VOX_NBITS);
        if (tb.map) return tb.base()[min(tag, TAGMAP_SMEM - 1)];
        // global map: an unconditional load at the clamped tag, tested afterwards
        const int slot = __ldg(a.tag2slot + min(tag, a.max_tag));
        return (tag <= a.max_tag && slot >= 0 && slot < a.nslot) ? slot : -1;
    };
    const int s0 = n0 > 0 ? owner(w0) : -1;
    const int s1 = n1 > 0 ? owner(w1) : -1;
    F2 up[3] = {bc(0.f), bc(0.f), bc(0.f)};
    // the centre part of the row the velocity read (slot vslot), kept for the force flush
    float4 vrh = make_float4(0.f, 0.f, 0.f, 0.f);
    float vrl0 = 0.f, vrl1 = 0.f;
    int vslot = -1;
    auto solid_velocity = [&]() {
        float ua[3] = {0.f, 0.f, 0.f}, ub[3] = {0.f, 0.f, 0.f};
        const int sl = s0 >= 0 ? s0 : s1;
        {
            // every lane of the warp loads a row (slot 0 for a lane without a solid
            // cell, whose velocities stay zero): no branch ahead of the load
            const TableRow r = load_row(a.xpf, max(sl, 0));
            vrh = r.a; vrl0 = r.b.x; vrl1 = r.b.y; vslot = sl;
            const RowPart rp = row_part(r, sx, sy, g);
            if (s0 >= 0) cell_part(r, rp, za, g, ua[0], ua[1], ua[2]);
            if (sl >= 0 && s1 == sl) cell_part(r, rp, zb, g, ub[0], ub[1], ub[2]);
        }
        if (s1 >= 0 && s1 != sl) row_velocity(load_row(a.xpf, s1), sx, sy, zb, g, ub[0], ub[1], ub[2]);
#pragma unroll
        for (int d = 0; d < 3; ++d) up[d] = pk(ua[d], ub[d]);
    };
    // FORCE: the solid correction's momentum is the BGK post-collision one, j + rho g,
    // for the cells that ran BGK
    auto hsol = [&]() -> F2 {
        return FORCE ? pk(n0 < 125 ? 1.f : 0.f, n1 < 125 ? 1.f : 0.f) * (bc(1.f) + m.rhoBar) : bc(0.f);
    };
    if constexpr (!FORCE) {
        // one pass; the solid terms only in warps that hold a solid cell
        if (__any_sync(FULL, n0 > 0 || n1 > 0)) {
            solid_velocity();
            collide_g2<true>(f, m, a.omega, up[0], up[1], up[2], B, Fx, Fy, Fz);
        } else {
            collide_g2<false>(f, m, a.omega, up[0], up[1], up[2], B, Fx, Fy, Fz);
        }
    } else {
        bgk2<FORCE>(f, m, a.omega, a.g3[0], a.g3[1], a.g3[2]);
        if (n0 > 0 || n1 > 0) {
            const F2 hs = hsol();
            const F2 sjx = fma2(hs, bc(a.g3[0]), m.jx), sjy = fma2(hs, bc(a.g3[1]), m.jy),
                     sjz = fma2(hs, bc(a.g3[2]), m.jz);
            solid_velocity();
            psm2(f, m.rhoBar, sjx, sjy, sjz, m.invRho, up[0], up[1], up[2], B, at2, Fx, Fy, Fz);
        }
    }

    // Stores (aligned rows only, the launcher sends others to k_collide_direct)
    // the lane's two cells in place in a row
    auto put_cells = [&](float* row, F2 v) {
        const float2 t = upk(v);
        // segments hold a multiple of 4 cells, so both cells of a pair are valid together,
        // and every pair of slots is 8-byte aligned
        if (v0) *reinterpret_cast<float2*>(row + j0) = t;
    };
    const size_t own = ((size_t)sx * g.ny + sy) * g.nz;
    put_cells(st.out[b][0], f[0]);
    // Odd phase, c_z != 0: each cell goes to slot z + c_z.  Slots (j0, j0 + 1) receive cells
    // (j0 - 1, j0) (c_z = +1) or (j0 + 1, j0 + 2) (c_z = -1), one lane over; the first and
    // the last lane store one value alone: the pair that is cut off by the segment's end, and
    // the cell whose slot lies outside it (wrapped, or bounced back at a z wall).  Both go out
    // in one predicated store: as branches of those two lanes they cost a warp one divergence
    // per direction (256^3 odd phase 530 us, 496 so = 78 % of the copy rate).
    const int last = len / 2 - 1;
    const bool pair_p = lane > 0 && v0, pair_m = lane < last, single = lane == 0 || lane == last;
    const int per_z = PER ? 1 : g.per[2];
    const int zdp = wrap_plus(z0 + len - 1, g.nz, per_z), zdm = wrap_minus(z0, g.nz, per_z);
    const int single_p = lane == 0 ? 1 : zdp - z0, single_m = lane == 0 ? zdm - z0 : j0;
#pragma unroll
    for (int i = 1; i < Q; ++i) {
        // row x + c_i; beyond an x / y wall the cell's own (bounce back in place)
        float* const row = st.out[b][opp(i)];
        if (!ODD || cz(i) == 0 || (!PER && !((srcrow >> opp(i)) & 1u))) {
            put_cells(row, f[i]);
            continue;
        }
        const float2 t = upk(f[i]);
        float* q = row + (cz(i) > 0 ? single_p : single_m);
        if (cz(i) > 0) {
            const float o = __shfl_up_sync(FULL, t.y, 1);
            if (pair_p) *reinterpret_cast<float2*>(row + j0) = make_float2(o, t.x);
            if (!PER && zdp < 0 && lane != 0) q = a.fo + (size_t)opp(i) * N + own + z0 + len - 1;
        } else {
            const float o = __shfl_down_sync(FULL, t.x, 1);
            if (pair_m) *reinterpret_cast<float2*>(row + j0) = make_float2(t.y, o);
            if (!PER && zdm < 0 && lane == 0) q = a.fo + (size_t)opp(i) * N + own;
        }
        if (single) *q = lane == 0 ? t.x : t.y;
    }

    const float2 fx = upk(Fx), fy = upk(Fy), fz = upk(Fz);
    if (a.cf) {
        const size_t ca = own + za, cb = own + zb;
        if (v0) { a.cf[ca] = fx.x; a.cf[N + ca] = fy.x; a.cf[2 * N + ca] = fz.x; }
        if (v1) { a.cf[cb] = fx.y; a.cf[N + cb] = fy.y; a.cf[2 * N + cb] = fz.y; }
    }
    if (((PER || g.per[2]) && len == g.nz) ||
        (images_can_differ<true>(g, a.reach, len, max(s0, s1)) &&
         images_differ(a, s0, s1, vslot, vrh.z, vrl1, za, zb))) {
        // the segment is a whole z-periodic row, or holds both ends of a chord that wraps
        // around: the arms are taken per cell
        forces_by_cell_far(a, PairForce{Fx, Fy, Fz, s0, s1, vslot, (n0 > 0 && s0 < 0) || (n1 > 0 && s1 < 0), vrh, vrl0, vrl1},
                           sx, sy, za, sy, zb, false);
        return;
    }
    // runs of equal owner, arms from the segment's middle point zc
    const int zc = z0 + SEGW / 2;
    // keys: the owners' particle slots; a solid cell whose tag names no particle is
    // reported and left out
    const int ka = v0 ? s0 : -1;
    const int kb = v1 ? s1 : -1;
    if ((v0 && n0 > 0 && s0 < 0) || (v1 && n1 > 0 && s1 < 0)) atomicOr(a.err, 0x8u);   // LBDEM_DEVERR_UNMAPPED_TAG
    const float da = (float)(za - zc), db = (float)(zb - zc);
    float va[5] = {fx.x, fy.x, fz.x, -da * fy.x, da * fx.x};
    float vb[5] = {fx.y, fy.y, fz.y, -db * fy.y, db * fx.y};
#pragma unroll
    for (int q = 0; q < 5; ++q) {
        if (ka < 0) va[q] = 0.f;
        if (kb < 0) vb[q] = 0.f;
    }
    if (__all_sync(FULL, ka < 0 || kb < 0 || ka == kb)) {
        const int key = ka >= 0 ? ka : kb;
#pragma unroll
        for (int q = 0; q < 5; ++q) va[q] += vb[q];
        reduce_runs(a, key, va, ka >= 0 ? za : zb, sx, sy, zc, vrh, vrl0, vrl1, vslot);
    } else {
        reduce_runs(a, ka, va, za, sx, sy, zc, vrh, vrl0, vrl1, vslot);
        reduce_runs(a, kb, vb, zb, sx, sy, zc, vrh, vrl0, vrl1, vslot);
    }
}

// ---------------------------------------------------------------------------
// FP32 form without staging: lattices whose rows are not 16-byte aligned, and
// every batch.  Lane l takes the cells l and l + 32 of a 64-cell segment and reads and
// writes global memory directly: every access is a coalesced 32-bit one whatever its
// alignment.  (Staged, such rows cost a
// bulk copy per row with its own lead, and halo elements put in place by hand: even / odd
// phase of a 71x67x243 channel 34.8 / 54.7 us staged, 32.4 / 35.5 us here = 82 / 75 % of
// the copy bandwidth; of 512 batched channels, 75.6 M cells, 2.80 / 5.27 and 2.61 /
// 3.08 ms.)  16 warps per SM at 128 registers; 20 or 24 spill and are slower.
// Odd phase: a cell's source and target rows come from a table of the segment in shared
// memory, with entries for the cells at a z wall or wrap, so that an access is one
// shared load and one multiply-add (slots formed from the cell's index at each access, and
// again with tests in warps at a wall: 3.40 ms for the 512 channels).
// A segment lies in a z-row, or, in the even phase of a batch, which touches only each
// cell's own slots, in an x-plane across its z-rows (the plane view: the lanes are filled
// whatever the row length; force and torque then take per-cell arms).
struct DirectCell {
    unsigned own;      // index in the domain, also of its voxel word
    int y, z;
    int zn[2];         // odd phase: z - 1, z + 1 (wrapped; z itself beyond a wall)
    int t[2];          // and their part of the row table: 0, Q at a wall, 2 Q wrapped
};
// Odd phase: slot that direction I of the cell is read from: slot opp I of the neighbour at
// x - c_I, or the cell's own slot I beyond a wall.  The value that streams along I goes to
// the slot of opp I: in the AA pattern a cell reads and writes the same slots.  T: the
// segment's row table (direct_rows).
template <int I>
__device__ __forceinline__ float* direct_slot(float* const* T, const DirectCell& c) {
    if constexpr (cz(I) == 0) return T[I] + c.z;
    else return T[I + c.t[cz(I) > 0 ? 0 : 1]] + c.zn[cz(I) > 0 ? 0 : 1];
}
// The row table of a segment of row (x, y), made by one warp, one direction a lane:
// [i] the row that direction i is read from, [Q + i] the cells' own (at a z wall), [2 Q + i]
// that row again (across the periodic z boundary).  Beyond an x / y wall all three lead to
// slot i of the cell itself, whatever c_z did to its z.
__device__ __forceinline__ void direct_rows(float** T, float* F, const Geom& g, int x, int y) {
    const int i = threadIdx.x & 31;
    __syncwarp();   // the last segment's reads
    if (i < Q) {
        const unsigned own = ((unsigned)x * (unsigned)g.ny + (unsigned)y) * (unsigned)g.nz;
        float* const slot = F + ((size_t)i * g.N + own);
        const int X = pick(cx(i), wrap_plus(x, g.nx, g.per[0]), x, wrap_minus(x, g.nx, g.per[0]));
        const int Y = pick(cy(i), wrap_plus(y, g.ny, g.per[1]), y, wrap_minus(y, g.ny, g.per[1]));
        if (i != 0 && X >= 0 && Y >= 0) {
            float* const row = F + ((size_t)opp(i) * g.N + ((unsigned)X * (unsigned)g.ny + (unsigned)Y) * (unsigned)g.nz);
            T[i] = row;
            T[2 * Q + i] = row;
        } else {
            T[i] = slot + cz(i);
            T[2 * Q + i] = slot - cz(i) * (g.nz - 1);
        }
        T[Q + i] = slot;
    }
    __syncwarp();
}

template <bool ODD, bool FORCE, bool BATCH>
__global__ void __launch_bounds__(DIRECT_BLOCK, DIRECT_BLOCKS_PER_SM)
k_collide_direct(const CollideArgs<float> a1, long long nseg, const CollideArgs<float>* __restrict__ dargs,
                 const int* __restrict__ seg0, int ndom) {
    constexpr bool PLANE = BATCH && !ODD;
    constexpr bool ROWS2 = BATCH && ODD;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int lane = threadIdx.x & 31;
    // row tables: input, and output or (batch, in place) the second row's
    __shared__ float* rows[ODD ? DIRECT_BLOCK / 32 : 1][2][ODD ? 3 * Q : 1];
    float** const Tin = rows[ODD ? threadIdx.x >> 5 : 0][0];
    float** const Tout = rows[ODD ? threadIdx.x >> 5 : 0][1];
    PairTables<BATCH ? NO_TABLES : 0> tb{false};
    const int* sseg0 = nullptr;   // batch: the CTA's copy of seg0 (ndom <= SEG0_SMEM)
    if constexpr (BATCH) {
        int* m = reinterpret_cast<int*>(smem_raw);
        if (ndom <= SEG0_SMEM) {
            for (int k = threadIdx.x; k < ndom; k += blockDim.x) m[k] = __ldg(seg0 + k);
            sseg0 = m;
        }
    } else {
        tb.load(a1);
        if (a1.probe_timeout) {
            // test hook: every warp meets a wait that runs out (as in k_collide_staged), reports
            // it and leaves; this kernel has no waits of its own
            __shared__ unsigned long long probe[DIRECT_BLOCK / 32];
            if (lane == 0) mbar_init(&probe[threadIdx.x >> 5], 1);
            __syncthreads();
            if (!mbar_wait(&probe[threadIdx.x >> 5], 0u, PROBE_WAIT) && lane == 0) atomicOr(a1.err, 0x20u);
            return;
        }
    }
    __syncthreads();
    const unsigned warps = gridDim.x * (DIRECT_BLOCK / 32);
    for (unsigned seg = blockIdx.x * (DIRECT_BLOCK / 32) + (threadIdx.x >> 5); seg < (unsigned)nseg; seg += warps) {
        int d = 0, first = 0;
        if constexpr (BATCH) {
            if (sseg0) {
                int lo = 0, hi = ndom - 1;
                while (lo < hi) {
                    const int mid = (lo + hi + 1) >> 1;
                    if (sseg0[mid] <= (int)seg) lo = mid;
                    else hi = mid - 1;
                }
                d = lo;
                first = sseg0[d];
            } else {
                d = find_domain(seg0, ndom, (int)seg);
                first = __ldg(seg0 + d);
            }
        }
        const CollideArgs<float>& a = BATCH ? dargs[d] : a1;
        // PLANE: a.g is the plane view (one row of ny nz cells per x), g the domain itself
        Geom g = a.g;
        if (PLANE) {
            g.ny = a.flat_ny;
            g.nz = a.flat_nz;
        }
        const unsigned N = (unsigned)g.N;   // 19 N floats fit the memory, so N < 2^32
        const unsigned sg = seg - (unsigned)first;
        const unsigned row = fast_div(sg, a.dz);
        int z0 = (int)(sg - row * a.dz.d) * SEGW;
        const int x = (int)fast_div(row, a.dy);
        int y = (int)(row - (unsigned)x * a.dy.d);
        unsigned rowbase = row * (unsigned)a.g.nz;
        bool two = false;    // the lane's second cell lies in the next row
        bool there = true;   // the segment's row exists
        if (ROWS2 && tails_paired(g.nz)) {
            // `row` is a pair of rows, dz divides by the pair's segments: the full ones of each
            // row, then both tails
            const int full = g.nz / SEGW;
            int k = z0 / SEGW;
            two = k == 2 * full;
            y *= 2;
            if (two) k = full;
            else if (k >= full) { k -= full; ++y; }
            z0 = k * SEGW;
            there = y < g.ny;
            if (!there) --y;
            rowbase = ((unsigned)x * (unsigned)g.ny + (unsigned)y) * (unsigned)g.nz;
        }
        const int hz = two ? 0 : 32;   // z of a lane's second cell, from its first
        float* F = a.fo;
        const float* Fin = a.f;
        if constexpr (ODD) {
            direct_rows(Tin, const_cast<float*>(Fin), g, x, y);
            if (BATCH && two) direct_rows(Tout, F, g, x, min(y + 1, g.ny - 1));
            if (!BATCH && F != Fin) direct_rows(Tout, F, g, x, y);
        }
        DirectCell c[2];
        bool valid[2];
        uint32_t w[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int p = z0 + lane + hz * h;
            valid[h] = p < a.g.nz;
            const int pc = valid[h] ? p : a.g.nz - 1;   // a lane slot past the row reads its last cell
            DirectCell& q = c[h];
            q.own = rowbase + (unsigned)pc;
            q.y = y;
            if (ROWS2) {
                valid[h] = valid[h] && there;
                if (two && h == 1) {
                    if (y + 1 < g.ny) {
                        q.y = y + 1;
                        q.own += (unsigned)g.nz;
                    } else {
                        valid[1] = false;
                    }
                }
            }
            w[h] = a.vox[q.own];
            q.z = pc;
            if (PLANE) {
                q.y = (int)fast_div((unsigned)pc, a.dnz);
                q.z = pc - q.y * g.nz;
            }
            if (ODD) {
                q.zn[0] = pc - 1;
                q.zn[1] = pc + 1;
                q.t[0] = q.t[1] = 0;
                if (pc == 0) { q.zn[0] = g.per[2] ? g.nz - 1 : pc; q.t[0] = g.per[2] ? 2 * Q : Q; }
                if (pc == g.nz - 1) { q.zn[1] = g.per[2] ? 0 : pc; q.t[1] = g.per[2] ? 2 * Q : Q; }
            }
        }
        // rows of the lane's second cells (a batch steps in place: its output rows too)
        float* const* const T1 = ROWS2 && two ? Tout : Tin;
        F2 f[Q];
        if constexpr (!ODD) {
#pragma unroll
            for (int i = 0; i < Q; ++i) {
                const float* r = Fin + (unsigned long long)i * N;
                f[i] = pk(r[c[0].own], r[c[1].own]);
            }
        } else {
            unroll_seq(std::make_integer_sequence<int, Q>{}, [&](auto ic) {
                constexpr int i = decltype(ic)::value;
                f[i] = pk(*direct_slot<i>(Tin, c[0]), *direct_slot<i>(T1, c[1]));
            });
        }
        PairForce o;
        collide_pair<FORCE>(a, g, tb, f, valid[0] ? w[0] : 0u, valid[1] ? w[1] : 0u, x, c[0].y, c[0].z, c[1].y, c[1].z,
                            o);
        if constexpr (!ODD) {
#pragma unroll
            for (int i = 0; i < Q; ++i) {
                float* r = F + (unsigned long long)opp(i) * N;
                const float2 t = upk(f[i]);
                if (valid[0]) r[c[0].own] = t.x;
                if (valid[1]) r[c[1].own] = t.y;
            }
        } else {
            float* const* const O0 = !BATCH && F != Fin ? Tout : Tin;
            float* const* const O1 = BATCH ? T1 : O0;
            unroll_seq(std::make_integer_sequence<int, Q>{}, [&](auto ic) {
                constexpr int i = decltype(ic)::value;
                const float2 t = upk(f[i]);
                if (valid[0]) *direct_slot<opp(i)>(O0, c[0]) = t.x;
                if (valid[1]) *direct_slot<opp(i)>(O1, c[1]) = t.y;
            });
        }
        if (a.cf) {
            const float2 fx = upk(o.Fx), fy = upk(o.Fy), fz = upk(o.Fz);
            if (valid[0]) { a.cf[c[0].own] = fx.x; a.cf[(size_t)N + c[0].own] = fy.x; a.cf[2 * (size_t)N + c[0].own] = fz.x; }
            if (valid[1]) { a.cf[c[1].own] = fx.y; a.cf[(size_t)N + c[1].own] = fy.y; a.cf[2 * (size_t)N + c[1].own] = fz.y; }
        }
        if (PLANE) {
            forces_by_cell(a, g, o, x, c[0].y, c[0].z, c[1].y, c[1].z, false);
        } else if ((g.per[2] && g.nz <= SEGW) ||
                   (images_can_differ<false>(g, a1.reach, min(g.nz - z0, SEGW), max(o.s0, o.s1)) &&
                    images_differ(a, o.s0, o.s1, o.vslot, o.rh.z, o.rl1, z0 + lane, z0 + lane + hz))) {
            // the segment is a whole z-periodic row, or holds both ends of a chord that wraps
            // around: the arms are taken per cell
            forces_by_cell_far(a, o, x, y, z0 + lane, c[1].y, z0 + lane + hz, two);
        } else {
            forces_by_run(a, o, x, y, c[1].y, z0 + SEGW / 2, z0 + lane, z0 + lane + hz, two);
        }
    }
}

// ---------------------------------------------------------------------------
// FP64 form: one staged cell (lane's cell j of the segment in
// buffer b), evaluated in fixed point (cell_fixed.h) from the stage and stored.
// The loop bodies cover the three direction pairs of one axis and run three times
// (the axes are cycled in between), over values kept in the stage: fully unrolled
// the update is 5000 instructions, and the warps, each at another place of it, then
// wait for the instruction cache 80 % of the time.
// MIS: rows not aligned (see issue_segment).
template <bool ODD, bool PER, bool MIS, bool STAGE_UP>
struct StagedCell {
    static constexpr int ROW = WarpStage<double, STAGE_UP>::W;
    WarpStage<double, STAGE_UP>& st;
    double* base;         // cell j of direction 0's staged row, without the row's lead
    double* fo;           // output populations
    const double* upf;    // surface-velocity field (read directly where it is not staged)
    unsigned N;           // cells (19 N doubles fit the memory, so N < 2^32)
    int b, z;
    size_t c;
    int zm, zp;           // z - 1 and z + 1 (wrapped; z itself beyond a wall)
    int tm, tp;           // and their part of the output rows: 0, Q at a wall, 2 Q wrapped
    unsigned long long lead;

    __device__ __forceinline__ StagedCell(const CollideArgs<double>& a, WarpStage<double, STAGE_UP>& stage, int buf,
                                          int j, int z0, unsigned long long leads)
        : st(stage), base(&stage.f[buf][0][WarpStage<double>::V + j]), fo(a.fo), upf(a.up), N((unsigned)a.g.N), b(buf),
          z(z0 + j), c((size_t)stage.row[buf][row_slot(0, 0)] + (z0 + j)), zm(z - 1), zp(z + 1), tm(0), tp(0),
          lead(leads) {
        const bool wrap = PER || a.g.per[2];
        if (z == 0) { zm = wrap ? a.g.nz - 1 : z; tm = wrap ? 2 * Q : Q; }
        if (z == a.g.nz - 1) { zp = wrap ? 0 : z; tp = wrap ? 2 * Q : Q; }
    }
    // the staged value of direction i (c_z = cz), the cell's own place in the stage
    __device__ __forceinline__ double* at(int i, int cz) const {
        int off = i * ROW;
        if (ODD) off -= cz;
        if (MIS) off += (int)((lead >> (2 * i)) & 3u);
        return base + off;
    }
    __device__ __forceinline__ double up(int d, int j) const {
        if (!STAGE_UP) return __ldg(upf + (size_t)d * N + c);
        const int m = MIS ? (int)((lead >> (40 + 2 * d)) & 3u) : 0;
        return st.up[b][d][m + j];
    }
    // where the post-collision value of direction i (opposite o, c_z = cz) goes: in both
    // phases the row that direction o was read from, one cell on in the odd phase
    __device__ __forceinline__ double* slot(int o, int cz) const {
        if (!ODD) return fo + c + (unsigned long long)(unsigned)o * N;
        const int zd = pick(cz, zm, z, zp), t = PER ? 0 : pick(cz, tm, 0, tp);
        return st.out[b][o + t] + zd;
    }
};

// The double routine for a cell outside the fixed-point range, out of line.  SOLID false: for
// the lanes of a warp without solid cells (128^3 fluid of density 1.12: 550 us a step, 1076
// with the solid terms; with a body force both forms run them for solid cells only).
template <bool FORCE, bool SOLID, typename Cell>
__device__ __noinline__ void collide_cell_double(Cell s, double omega, double g0,
                                                 double g1, double g2, int n, double B, double u0, double u1,
                                                 double u2, double (&F)[3]) {
    double f[Q];
#pragma unroll
    for (int i = 0; i < Q; ++i) f[i] = *s.at(i, cz(i));
    if constexpr (FORCE) collide_cell(f, omega, g0, g1, g2, n, B, u0, u1, u2, [&](int i) { return *s.at(i, cz(i)); }, F);
    else collide_cell_fp64<SOLID>(f, omega, B, u0, u1, u2, F[0], F[1], F[2]);
    s.fo[s.c] = f[0];
#pragma unroll
    for (int i = 1; i < Q; ++i) *s.slot(opp(i), cz(i)) = f[i];
}

template <bool ODD, bool FORCE, bool PER, bool MIS, bool STAGE_UP>
__device__ __forceinline__ void collide_cell_staged(const CollideArgs<double>& a, WarpStage<double, STAGE_UP>& st,
                                                    int b, int j, int z0, unsigned long long lead,
                                                    uint32_t w, bool solid, double (&F)[3]) {
    using fixed::i64;
    const StagedCell<ODD, PER, MIS, STAGE_UP> s(a, st, b, j, z0, lead);
    // the cell's unit
    double* const p0 = s.at(0, 0);
    int e = __double2hiint(*p0) & 0x7ff00000;
#pragma unroll
    for (int i = 1; i < Q; ++i) e = max(e, __double2hiint(*s.at(i, cz(i))) & 0x7ff00000);
    e >>= 20;
    double B = 0.0, u0 = 0.0, u1 = 0.0, u2 = 0.0;
    const int n = min((int)(w & VOX_NMASK), 125);
    if (n > 0) {
        B = __ldg(a.btab + n);
        u0 = s.up(0, j);
        u1 = s.up(1, j);
        u2 = s.up(2, j);
        e = fixed::cell_exponent_up(e, u0, u1, u2);
    }
    if (FORCE) e = fixed::cell_exponent_up(e, a.g3[0], a.g3[1], a.g3[2]);
    if (!fixed::fits(e)) {
        if (FORCE || solid) collide_cell_double<FORCE, true>(s, a.omega, a.g3[0], a.g3[1], a.g3[2], n, B, u0, u1, u2, F);
        else collide_cell_double<FORCE, FORCE>(s, a.omega, 0.0, 0.0, 0.0, 0, 0.0, 0.0, 0.0, 0.0, F);
        return;
    }
    e = max(e, fixed::EMAX_LO);
    // populations in units (back into the stage), and their sums
    const i64 X0 = fixed::to_fixed<4>(*p0, e);
    fixed::Sums sum{X0, {0, 0, 0}};
    // direction q of cycle a, as in fixed::dir_of, with its c_z and target row slot
    auto dir = [](int q, int a, int dg) { return q < 2 ? (q == 0 ? 10 : 1) + a : (q == 2 ? 13 : q == 3 ? 4 : q == 4 ? 14 : 5) + dg; };
    auto dir_z = [](int q, int a) {
        const int zc = q < 2 ? (a == 2 ? 1 : 0) : (a > 0 ? 1 : 0);
        return q == 0 || q == 2 || q == 5 ? zc : -zc;
    };
#pragma unroll 1
    for (int t = 0, dg = 0; t < 3; dg = t == 0 ? 4 : 2, ++t) {
        i64 x[6];
#pragma unroll
        for (int q = 0; q < 6; ++q) {
            double* p = s.at(dir(q, t, dg), dir_z(q, t));
            x[q] = fixed::to_fixed<4>(*p, e);
            *reinterpret_cast<i64*>(p) = x[q];
        }
        fixed::add_three(sum, x, t == 2);
    }
    fixed::Cell cell = fixed::cell_setup<FORCE>(solid, sum, e, fixed::relax_of(a.omega), a.g3[0], a.g3[1], a.g3[2],
                                                n == 125, B, u0, u1, u2, F);
    *s.slot(0, 0) = fixed::update_rest<FORCE>(solid, cell, X0, e);
#pragma unroll 1
    for (int t = 0, dg = 0; t < 3; dg = t == 0 ? 4 : 2, ++t) {
        fixed::update_three<FORCE>(
            solid, cell, t == 2,
            [&](int q) { return *reinterpret_cast<const i64*>(s.at(dir(q, t, dg), dir_z(q, t))); }, e,
            [&](int q, double v) { *s.slot(dir(q ^ 1, t, dg), dir_z(q, t)) = v; });
    }
}

// Warps per stage.  The FP64 form gives each segment to two
// warps, one 32-cell pass each: the stages of 8 warps fill the SM's shared memory, and
// with two warps per scheduler the integer chains of a cell left half of the issue
// slots empty.  The two take the longer (solid) pass in turn and do not wait for
// each other at the end of a segment: a buffer is handed back through a barrier, so the warp with the shorter pass goes on to the next segment.
template <typename T>
__host__ __device__ constexpr int stage_warps() { return sizeof(T) == 8 ? 2 : 1; }

// PER: every axis periodic (no wall cases; shifts and neighbour rows are fixed).
// MIS: rows not 16-byte aligned (see issue_segment).
// BATCH: segments of many domains, numbered domain after domain (seg0[d] is
// the first segment of domain d); every domain has its own CollideArgs.
template <typename T, bool ODD, bool FORCE, bool PER, bool MIS, bool BATCH>
__global__ void __launch_bounds__(COLLIDE_BLOCK, sizeof(T) == 4 ? 4 : 2 * stage_warps<T>())
k_collide_staged(const CollideArgs<T> a1, long long nseg, const CollideArgs<T>* __restrict__ dargs,
                 const int* __restrict__ seg0, int ndom) {
    constexpr int V = WarpStage<T>::V;
    // FP64 form: surface-velocity rows staged with the populations for a single
    // lattice; the many short rows of a batch read them directly (three more small
    // copies per segment cost more there than the loads they replace).  The FP32
    // form keeps no velocity field (it recomputes the velocity per solid cell).
    constexpr bool STAGE_UP = stage_up<T, BATCH>();
    // FP32 form, aligned rows of a single lattice: staging by per-thread cp.async
    constexpr bool LSU = sizeof(T) == 4 && !MIS && !BATCH;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    // SW warps share a stage: warp `sub` of group `group`
    constexpr int SW = stage_warps<T>();
    constexpr int GROUPS = WARPS / SW;
    // a buffer's arrivals: the bytes of its bulk copies, and every lane's own copies
    constexpr uint32_t ARRIVALS = sizeof(T) == 8 && ODD && !PER ? 33 : 1;
    const int group = warp / SW, sub = warp % SW;
    WarpStage<T, STAGE_UP>& st = reinterpret_cast<WarpStage<T, STAGE_UP>*>(smem_raw)[group];
    __shared__ unsigned long long probe[WARPS];   // the test hook's barrier (never completes)
    // a shared stage's barriers: buffer b left by both warps
    __shared__ unsigned long long shared_bar[SW > 1 ? GROUPS : 1][2];
    if (lane == 0) {
        if (sub == 0) {
            mbar_init(&st.bar[0], ARRIVALS);
            mbar_init(&st.bar[1], ARRIVALS);
            if (SW > 1)
                for (int q = 0; q < 2; ++q) mbar_init(&shared_bar[group][q], SW);
        }
        mbar_init(&probe[warp], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (SW > 1) __syncthreads();
    else __syncwarp();
    PairTables<STAGED_TABLES> tb{false};
    if constexpr (sizeof(T) == 4) {
        tb.load(a1);
        __syncthreads();   // every warp of the CTA reaches it (before any leaves)
    }
    const int* sseg0 = nullptr;   // batch: the CTA's copy of seg0 (ndom <= SEG0_SMEM)
    if constexpr (BATCH) {
        int* m = reinterpret_cast<int*>(smem_raw + GROUPS * sizeof(WarpStage<T, STAGE_UP>));
        if (ndom <= SEG0_SMEM) {
            for (int k = threadIdx.x; k < ndom; k += blockDim.x) m[k] = __ldg(seg0 + k);
            sseg0 = m;
        }
        __syncthreads();   // every warp of the CTA reaches it (before any leaves)
    }
    const long long stride = (long long)gridDim.x * GROUPS;
    long long seg = (long long)blockIdx.x * GROUPS + group;
    if (seg >= nseg) return;   // both warps of a shared stage
    auto issue = [&](int buf, long long sg) {
        if constexpr (LSU) {
            issue_segment_lsu<T, ODD, PER, STAGE_UP>(a1, st, buf, sg);
        } else if constexpr (BATCH) {
            int d, first;
            if (sseg0) {
                int lo = 0, hi = ndom - 1;
                while (lo < hi) {
                    const int mid = (lo + hi + 1) >> 1;
                    if (sseg0[mid] <= (int)sg) lo = mid;
                    else hi = mid - 1;
                }
                d = lo;
                first = sseg0[d];
            } else {
                d = find_domain(seg0, ndom, (int)sg);
                first = __ldg(seg0 + d);
            }
            const CollideArgs<T>& A = dargs[d];
            issue_segment<ODD, PER, MIS, STAGE_UP>(A, st, buf, sg - first, d);
        } else {
            issue_segment<ODD, PER, MIS, STAGE_UP>(a1, st, buf, sg, 0);
        }
    };
    // segment k of the stage (buffer b = k & 1) is issued by warp k % SW, one segment
    // ahead; with two warps the same warp takes its first (solid) pass
    if (sub == 0) issue(0, seg);
    uint32_t phase = 0;   // bit b: parity expected next on buffer b
    uint32_t ephase = 0;  // the same for the barriers that hand a shared buffer back
    bool first = true;
    int b = 0;
    for (; seg < nseg; seg += stride, b ^= 1) {
        const long long next = seg + stride;
        const bool lead_warp = SW == 1 || sub == b;
        bool ok = true;
        if (next < nseg && (SW == 1 || !lead_warp)) {
            // both warps have left the buffer's last segment (none before the first two)
            if (SW > 1 && !first) {
                ok = mbar_wait(&shared_bar[group][b ^ 1], (ephase >> (b ^ 1)) & 1u);
                ephase ^= 1u << (b ^ 1);
            }
            if (SW == 1 || __all_sync(FULL, ok)) issue(b ^ 1, next);
        }
        if constexpr (LSU) {
            // this thread's copies of the current segment (all groups but the newest)
            if (next < nseg) cp_wait<1>();
            else cp_wait<0>();
            __syncwarp();   // and every other lane's
        } else {
            const uint32_t pb = (phase >> b) & 1u;
            if (!BATCH && a1.probe_timeout && first) {
                // test hook: wait on a barrier nothing arrives on, as for a copy that never lands
                ok = mbar_wait(&probe[warp], 0u, PROBE_WAIT);
            } else if (ok) {
                ok = mbar_wait(&st.bar[b], pb);
            }
            phase ^= 1u << b;
            first = false;
            if (__any_sync(FULL, !ok)) {
                // a copy did not land (or the stage's other warp has left): report, let the
                // stage's copies in flight land (both buffers, bounded), leave
                if (lane == 0) atomicOr(BATCH ? dargs[0].err : a1.err, 0x20u);   // LBDEM_DEVERR_TIMEOUT
                mbar_wait(&st.bar[b], pb);
                if (next < nseg) mbar_wait(&st.bar[b ^ 1], (phase >> (b ^ 1)) & 1u);
                return;
            }
        }
        const int sx = st.geo[b][0], sy = st.geo[b][1], z0 = st.geo[b][2], len = st.geo[b][3];
        const CollideArgs<T>& a = BATCH ? dargs[st.geo[b][4]] : a1;
        const Geom& g = a.g;
        const size_t N = g.N;
        const T* Fin = a.f;   // input populations
        const size_t own = ((size_t)sx * g.ny + sy) * g.nz;
        const unsigned long long lead = MIS ? st.lead[b] : 0ull;
        // Odd phase with walls along z, aligned rows: the halo element of an edge
        // cell is its own slot i (half-way bounce-back).
        const uint32_t srcrow = ODD && !PER ? (uint32_t)st.geo[b][5] : 0u;   // bit i: direction i's source row is inside
        if (sizeof(T) == 4 && ODD && !PER && !g.per[2] && (z0 == 0 || z0 + len == g.nz)) {
            if (lane < 10) {
                const int i = zdir(lane);
                if ((srcrow >> i) & 1u) {
                    if (cz(i) > 0 && z0 == 0) st.f[b][i][V - 1] = Fin[(size_t)i * N + own];
                    if (cz(i) < 0 && z0 + len == g.nz) st.f[b][i][V + len] = Fin[(size_t)i * N + own + g.nz - 1];
                }
            }
            __syncwarp();
        }
        if constexpr (sizeof(T) == 4) {
            static_assert(LSU, "FP32: aligned rows of a single lattice (others: k_collide_direct)");
            collide_segment_pairs<ODD, FORCE, PER, STAGE_UP>(a, st, b, sx, sy, z0, len, srcrow, tb);
        } else {
            // FP64 form: one cell per lane at a time; force and torque per cell with
            // double atomics.  The segment's solid cells are taken first (pass 0
            // holds as many of them as fit): a pass whose warp holds a solid cell
            // runs the solid terms for every lane, so gathering them leaves more
            // passes on the fluid path.  A cell's result does not depend on
            // its pass.
            static_assert(SEGW == 64 && SW == 2, "two passes of 32 cells per segment, one for each warp");
            const int vlead = st.geo[b][6];
            const uint32_t wl0 = lane < len ? st.vox[b][vlead + lane] : 0u;
            const uint32_t wl1 = lane + 32 < len ? st.vox[b][vlead + lane + 32] : 0u;
            const unsigned sol0 = __ballot_sync(FULL, (wl0 & VOX_NMASK) != 0u);
            const unsigned sol1 = __ballot_sync(FULL, (wl1 & VOX_NMASK) != 0u);
            const unsigned flu0 = __ballot_sync(FULL, lane < len) & ~sol0;
            const unsigned flu1 = __ballot_sync(FULL, lane + 32 < len) & ~sol1;
            const int ns0 = __popc(sol0), ns = ns0 + __popc(sol1);
            const int nf0 = __popc(flu0), nf = nf0 + __popc(flu1);
            const int p = lead_warp ? 0 : 1;
            const int slot = 32 * p + lane;
            int j = -1;   // the cell this lane takes in pass p
            if (slot < ns) j = slot < ns0 ? nth_bit(sol0, slot) : 32 + nth_bit(sol1, slot - ns0);
            else if (slot - ns < nf) j = slot - ns < nf0 ? nth_bit(flu0, slot - ns) : 32 + nth_bit(flu1, slot - ns - nf0);
            const bool any_solid = ns > 32 * p;   // warp-uniform
            if (j >= 0) {
                const uint32_t w = st.vox[b][vlead + j];
                T Fc[3];
                collide_cell_staged<ODD, FORCE, PER, MIS, STAGE_UP>(a, st, b, j, z0, lead, w, any_solid, Fc);
                // (the segment's data are read again: kept over the update they would spill)
                if (a.cf) {
                    const size_t c = (size_t)st.row[b][row_slot(0, 0)] + st.geo[b][2] + j;
                    a.cf[c] = Fc[0]; a.cf[N + c] = Fc[1]; a.cf[2 * N + c] = Fc[2];
                }
                if (any_solid) {
                    T v[6] = {T(0), T(0), T(0), T(0), T(0), T(0)};
                    const int key = cell_force_terms(a, st.vox[b][vlead + j], st.geo[b][0], st.geo[b][1], st.geo[b][2] + j, Fc[0],
                                                     Fc[1], Fc[2], v);
                    if (key >= 0) add_cell_force(a, key, v);
                }
            }
        }
        // buffer b is free for the segment after next; writes into it (halo elements,
        // populations in units) come before the copies that reuse it
        if constexpr (!LSU) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (SW > 1 && lane == 0) mbar_arrive(&shared_bar[group][b]);
    }
}

// A persistent grid of a kernel: as many blocks as fit the device (or blocks_per_sm of
// them per SM), at most one per `per_block` segments.  `shape` is the kernel's own cache,
// per device: (resident blocks per SM << 16) | SM count, 0 until first use there.
template <typename Kernel>
cudaError_t persistent_grid(Kernel kernel, int threads, size_t smem, std::atomic<int>* shape, long long nseg,
                            int per_block, int blocks_per_sm, unsigned* grid) {
    if (nseg >= (1LL << 31)) return cudaErrorInvalidValue;   // segment indices are split in 32 bits
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= LBDEM_MAX_DEVICES) return cudaErrorInvalidDevice;
    int packed = shape[dev].load(std::memory_order_relaxed);
    if (packed == 0) {
        int sms = 0, per_sm = 0;
        e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem);
        if (e != cudaSuccess) return e;
        if (per_sm < 1) per_sm = 1;
        packed = (per_sm << 16) | (sms & 0xffff);
        shape[dev].store(packed, std::memory_order_relaxed);
    }
    const int per_sm = packed >> 16, sms = packed & 0xffff;
    const int use = (blocks_per_sm > 0 && blocks_per_sm < per_sm) ? blocks_per_sm : per_sm;
    const long long want = (long long)sms * use;
    const long long blocks = (nseg + per_block - 1) / per_block;
    *grid = (unsigned)(blocks < want ? blocks : want);
    return cudaSuccess;
}

template <typename T, bool ODD, bool FORCE, bool PER, bool MIS, bool BATCH>
cudaError_t launch_staged(const CollideArgs<T>& a, long long nseg, const CollideArgs<T>* dargs,
                          const int* seg0, int ndom, int blocks_per_sm, cudaStream_t s) {
    constexpr int GROUPS = WARPS / stage_warps<T>();   // stages (segments in work) per block
    constexpr size_t smem =
        GROUPS * sizeof(WarpStage<T, stage_up<T, BATCH>()>) + (sizeof(T) == 4 ? TAGMAP_BYTES : 0) +
        (BATCH ? SEG0_BYTES : 0);
    static std::atomic<int> shape[LBDEM_MAX_DEVICES];
    unsigned grid = 0;
    const cudaError_t e = persistent_grid(k_collide_staged<T, ODD, FORCE, PER, MIS, BATCH>, COLLIDE_BLOCK, smem, shape,
                                          nseg, GROUPS, blocks_per_sm, &grid);
    if (e != cudaSuccess || grid == 0) return e;
    k_collide_staged<T, ODD, FORCE, PER, MIS, BATCH><<<grid, COLLIDE_BLOCK, smem, s>>>(a, nseg, dargs, seg0, ndom);
    return cudaGetLastError();
}

template <bool ODD, bool FORCE, bool BATCH>
cudaError_t launch_direct(const CollideArgs<float>& a, long long nseg, const CollideArgs<float>* dargs, const int* seg0,
                        int ndom, int blocks_per_sm, cudaStream_t s) {
    constexpr size_t smem = BATCH ? SEG0_BYTES : TAGMAP_BYTES;
    static std::atomic<int> shape[LBDEM_MAX_DEVICES];
    unsigned grid = 0;
    const cudaError_t e = persistent_grid(k_collide_direct<ODD, FORCE, BATCH>, DIRECT_BLOCK, smem, shape, nseg,
                                          DIRECT_BLOCK / 32, blocks_per_sm, &grid);
    if (e != cudaSuccess || grid == 0) return e;
    k_collide_direct<ODD, FORCE, BATCH><<<grid, DIRECT_BLOCK, smem, s>>>(a, nseg, dargs, seg0, ndom);
    return cudaGetLastError();
}

template <typename T, bool ODD, bool FORCE>
cudaError_t launch_one(const CollideArgs<T>& args, cudaStream_t s) {
    CollideArgs<T> a = args;
    // Aligned rows: every population row's start and length 16-byte aligned (nz *
    // sizeof(T)), and 16-byte aligned arrays (device allocations are; a caller's
    // out-of-place target that is not takes the other path).  The FP64 form copies
    // voxel words from the boundary below the row, so an even nz is enough; rows of
    // 2 (mod 4) cells go 6 / 20 % faster this way (160x48x50 channel, even / odd phase
    // 72 / 95 us as unaligned rows, 68 / 74 us).
    const bool arrays_aligned = (((uintptr_t)a.f | (uintptr_t)a.fo | (uintptr_t)a.vox | (uintptr_t)a.up) & 15u) == 0;
    const bool aligned = a.g.nz % (sizeof(T) == 8 ? 2 : 4) == 0 && arrays_aligned;
    const int nzseg = (a.g.nz + SEGW - 1) / SEGW;
    a.dz = div_magic((unsigned)nzseg);
    a.dy = div_magic((unsigned)a.g.ny);
    const long long nseg = (long long)a.g.nx * a.g.ny * nzseg;
    if (aligned) {
        if (a.g.per[0] && a.g.per[1] && a.g.per[2])
            return launch_staged<T, ODD, FORCE, true, false, false>(a, nseg, nullptr, nullptr, 0, 0, s);
        return launch_staged<T, ODD, FORCE, false, false, false>(a, nseg, nullptr, nullptr, 0, 0, s);
    }
    if constexpr (sizeof(T) == 8) return launch_staged<T, ODD, FORCE, false, true, false>(a, nseg, nullptr, nullptr, 0, 0, s);
    else return launch_direct<ODD, FORCE, false>(a, nseg, nullptr, nullptr, 0, 0, s);
}

template <typename T, bool ODD, bool FORCE>
cudaError_t launch_batch(const CollideArgs<T>* dargs, const int* seg0, int ndom, long long nseg, short reach,
                         int blocks_per_sm, cudaStream_t s) {
    CollideArgs<T> none{};
    none.reach = reach;
    if constexpr (sizeof(T) == 4) return launch_direct<ODD, FORCE, true>(none, nseg, dargs, seg0, ndom, blocks_per_sm, s);
    else return launch_staged<T, ODD, FORCE, false, true, true>(none, nseg, dargs, seg0, ndom, blocks_per_sm, s);
}

}  // namespace

template <typename T>
cudaError_t launch_collide_stream(const CollideArgs<T>& a, bool odd, bool force, cudaStream_t s) {
    if (odd) return force ? launch_one<T, true, true>(a, s) : launch_one<T, true, false>(a, s);
    return force ? launch_one<T, false, true>(a, s) : launch_one<T, false, false>(a, s);
}

template <typename T>
cudaError_t launch_collide_batch(const CollideArgs<T>* dargs, const int* seg0, int ndom, long long nseg, short reach,
                                 bool odd, bool force, int blocks_per_sm, cudaStream_t s) {
    if (odd)
        return force ? launch_batch<T, true, true>(dargs, seg0, ndom, nseg, reach, blocks_per_sm, s)
                     : launch_batch<T, true, false>(dargs, seg0, ndom, nseg, reach, blocks_per_sm, s);
    return force ? launch_batch<T, false, true>(dargs, seg0, ndom, nseg, reach, blocks_per_sm, s)
                 : launch_batch<T, false, false>(dargs, seg0, ndom, nseg, reach, blocks_per_sm, s);
}

template cudaError_t launch_collide_stream<float>(const CollideArgs<float>&, bool, bool, cudaStream_t);
template cudaError_t launch_collide_stream<double>(const CollideArgs<double>&, bool, bool, cudaStream_t);
template cudaError_t launch_collide_batch<float>(const CollideArgs<float>*, const int*, int, long long, short, bool, bool,
                                                 int, cudaStream_t);
template cudaError_t launch_collide_batch<double>(const CollideArgs<double>*, const int*, int, long long, short, bool, bool,
                                                  int, cudaStream_t);

}  // namespace lbdem
