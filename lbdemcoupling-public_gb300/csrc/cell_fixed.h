// The FP64 form's collision of one cell on the integer pipe.
//
// GB300 executes double arithmetic at two lanes per clock per SM and integer
// arithmetic at 64 and more, so the update of a cell in double (about 150
// operations for a fluid cell, 270 for a solid one) is bound by the FP64 pipe at
// an eighth of the memory rate.  Here a cell's doubles are
// read as 64-bit fixed-point numbers of one common unit, the update is evaluated
// in those, and every result is rounded once to the nearest double.  A 128^3 suspension
// (solid fraction 0.26) steps in 0.32 / 0.36 ms (even / odd phase) against 0.93 ms in double.
//
// Unit.  With 2^E above every |f_i| of the cell (E from the largest exponent
// field emax, E = emax - 1022) the unit is 2^(E - 57) = 2^(emax - 1079): a
// population is below 2^57 units, the sums of 19 populations are exact and below
// 2^62, and the largest population's last mantissa bit is 16 units.  Products
// are rounded to the unit (mul<S>: error at most 2^(62 - S) units for the low x low
// partial product that is left out, and half a unit: 1.5 units for S = 62, 2.5 for 61), and a
// result then once to double.  Double arithmetic rounds at every one of its operations; both
// errors are measured against 113-bit arithmetic in tests/test_cell_fixed_cpu.py (a result is
// off by a third of what the double update is).
//
// Range.  2^E <= 2^-5 (|f_i| < 1/32, hence |rhoBar| < 0.6; a fluid at rest reaches it at
// |rhoBar| = 0.094, where f_0 = rhoBar / 3 does) and surface velocities and body forces
// below 2^(E + 3) (they raise E if need be: below 1/4); non-zero cells below
// 2^-958 are left out too.  A cell outside the range, or with a NaN or infinity,
// takes the double routine: fits() tells, from the cell's own values alone.
//
// The update (src/ibCompositeDynamics3D.hh:130-203 with the Guo force in the base BGK) is
// regrouped, with g = f - feq(J), J = j + rho g/2 (g the body force), S = feq + source,
// j* = j + rho g below full coverage (else j) and P = rho uPart, as
//   out_k = S_k + A g_k + B (f_i - feq_i(j*) + feq_k(P) - S_k),  A = (1 - omega)(1 - B),
//   out_0 = S_0 + A g_0 + B (f_0 + feq_0(j*) - feq_0(P) - S_0),
//   F = B (2 j - j* - P)
// (the pair terms of the momentum exchange summed over c_k).  S is an equilibrium too: the
// source's even part is that of the tensor M = pre (u g + g u), its odd part that of the
// vector pre g, pre = (1 - omega/2) rho.  Without a body force S = feq, J = j* = j, and
// with Dl = feq - feq(P) the same reads (6 % faster than through S)
//   out_k = feq_k + A g_k + B (g_i - Dl_k),  out_0 = feq_0 + (A + B) g_0 + B Dl_0,
//   F = B (j - P).
#pragma once

#include <cstdint>
#include <cstring>

#ifdef __CUDACC__
#define LBDEM_HD __host__ __device__ __forceinline__
#else
#define LBDEM_HD inline
#endif

namespace lbdem {
namespace fixed {

typedef long long i64;
typedef unsigned long long u64;

LBDEM_HD u64 bits_of(double x) {
#ifdef __CUDA_ARCH__
    return (u64)__double_as_longlong(x);
#else
    u64 b;
    std::memcpy(&b, &x, 8);
    return b;
#endif
}
LBDEM_HD double double_of(u64 b) {
#ifdef __CUDA_ARCH__
    return __longlong_as_double((i64)b);
#else
    double x;
    std::memcpy(&x, &b, 8);
    return x;
#endif
}
LBDEM_HD int exponent_field(u64 b) { return (int)((uint32_t)(b >> 32) >> 20) & 0x7ff; }
LBDEM_HD int imax(int a, int b) { return a > b ? a : b; }
LBDEM_HD int imin(int a, int b) { return a < b ? a : b; }
LBDEM_HD i64 shl(i64 x, int s) { return (i64)((u64)x << s); }

constexpr int EMAX_HI = 1017;   // 2^E <= 2^-5
constexpr int EMAX_LO = 65;     // smallest emax whose results stay normal doubles
constexpr int UP_BITS = 3;      // a surface velocity is below 2^(E + UP_BITS)

// The exponent that fixes the cell's unit: the largest exponent field of its
// populations (0: every one is zero or subnormal), raised for its surface velocity.
LBDEM_HD int cell_exponent(const double (&f)[19]) {
    int e = 0;
#pragma unroll
    for (int i = 0; i < 19; ++i) e = imax(e, exponent_field(bits_of(f[i])));
    return e;
}
LBDEM_HD int cell_exponent_up(int e, double up0, double up1, double up2) {
    e = imax(e, exponent_field(bits_of(up0)) - UP_BITS);
    e = imax(e, exponent_field(bits_of(up1)) - UP_BITS);
    return imax(e, exponent_field(bits_of(up2)) - UP_BITS);
}
LBDEM_HD bool fits(int emax) { return emax <= EMAX_HI && (emax == 0 || emax >= EMAX_LO); }

// x in units of 2^(emax - 1079), |x| < 2^(emax - 1022 + L - 4), truncated.
template <int L>
LBDEM_HD i64 to_fixed(double x, int emax) {
    const u64 b = bits_of(x);
    const int sh = imin(emax + (L - 4) - exponent_field(b), 63);   // zero and subnormal: 63, all bits out
    const u64 m = ((b & 0x000fffffffffffffull) | 0x0010000000000000ull) << L;
    const u64 v = m >> sh;
    const i64 s = (i64)b >> 63;
    return (i64)(v ^ (u64)s) - s;
}
// v units as a double, rounded to nearest: two double additions on words put together
// by hand, the first of them exact (an integer normalisation takes thirty operations).
LBDEM_HD double to_double(i64 v, int emax) {
    const u64 a = ((u64)(uint32_t)(emax - 4) << 52) | (u64)(uint32_t)(u64)v;
    const u64 b = ((u64)(uint32_t)(emax + 28) << 52) | (u64)((uint32_t)((u64)v >> 32) ^ 0x80000000u);
    const u64 k = ((u64)(uint32_t)(emax + 28) << 52) | 0x80100000ull;
    return (double_of(b) - double_of(k)) + double_of(a);
}

// x = h 2^32 + l with -2^31 <= l < 2^31.
struct Split {
    int h, l;
};
LBDEM_HD Split split(i64 x) {
    Split s;
    s.l = (int)(uint32_t)(u64)x;
    s.h = (int)(x >> 32) - (s.l >> 31);
    return s;
}
// a b / 2^S rounded, without the low x low partial product (at most 2^(62 - S)).
template <int S>
LBDEM_HD i64 mul(const Split& a, const Split& b) {
    static_assert(S >= 60 && S <= 64, "shift of a product");
    const i64 t = (i64)a.h * b.l + ((i64)a.l * b.h + ((i64)1 << (S - 33)));
    return shl((i64)a.h * b.h, 64 - S) + (t >> (S - 32));
}

// omega's part of a launch: 1 - omega and 1 - omega/2 in Q62 (omega in (0, 2)).
struct Relax {
    Split om1, hom;
};
LBDEM_HD i64 to_q62(double x) {   // |x| <= 1, exact to 2^-62
    const u64 b = bits_of(x);
    const u64 m = (((b & 0x000fffffffffffffull) | 0x0010000000000000ull) << 10) >> imin(1023 - exponent_field(b), 63);
    const i64 s = (i64)b >> 63;
    return (i64)(m ^ (u64)s) - s;
}
LBDEM_HD Relax relax_of(double omega) { return Relax{split(to_q62(1.0 - omega)), split(to_q62(1.0 - 0.5 * omega))}; }

// Symmetric second-order tensor in units: the diagonal (xx, yy, zz) and the mixed
// entries (xy, yz, zx), each of them one place on when the axes are cycled.
struct Tensor {
    i64 d[3], m[3];
};
// v_a w_b for two vectors in units: product / 2^61, then the rest of the shift.
LBDEM_HD Tensor tensor_of(const Split (&v)[3], const Split (&w)[3], int sh, i64 half) {
    Tensor q;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        q.d[a] = (mul<61>(v[a], w[a]) + half) >> sh;
        q.m[a] = (mul<61>(v[a], w[(a + 1) % 3]) + half) >> sh;
    }
    return q;
}
// An equilibrium's parts: even C_k = t_k (base + 4.5 c_k c_k : q) from t base and q,
// odd L_k = 3 t_k c_k.v from v / 12.
struct Parts {
    i64 b36, b3;   // base / 36, base / 3
    Tensor q;
    i64 o[3];
};
LBDEM_HD Parts parts_of(i64 rb, const Tensor& q, i64 vx, i64 vy, i64 vz) {
    constexpr u64 c36 = 0x071c71c71c71c71cull, c3 = 0x5555555555555555ull;   // 2^64 / 36, 2^64 / 3
    constexpr u64 c12 = 0x1555555555555555ull;                               // 2^64 / 12
    Parts e;
    e.q = q;
    const i64 s = q.d[0] + q.d[1] + q.d[2];
    const Split base = split(rb - (s + (s >> 1)));
    e.b36 = mul<64>(base, split((i64)c36));
    e.b3 = mul<64>(base, split((i64)c3));
    const Split c = split((i64)c12);
    e.o[0] = mul<64>(split(vx), c);
    e.o[1] = mul<64>(split(vy), c);
    e.o[2] = mul<64>(split(vz), c);
    return e;
}
// The parts for c = e_0, e_0 + e_1 and e_0 - e_1 (last cycle: e_1 - e_0) of the
// current cycle of the axes.
struct Three {
    i64 C[3], L[3];
};
LBDEM_HD Three three_of(const Parts& e, bool last) {
    Three r;
    const i64 h = e.b36 + ((e.q.d[0] + e.q.d[1] + 4) >> 3), m = (e.q.m[0] + 2) >> 2;
    r.C[0] = e.b36 + e.b36 + ((e.q.d[0] + 2) >> 2);
    r.C[1] = h + m;
    r.C[2] = h - m;
    r.L[0] = e.o[0] + e.o[0];
    r.L[1] = e.o[0] + e.o[1];
    r.L[2] = last ? e.o[1] - e.o[0] : e.o[0] - e.o[1];
    return r;
}
LBDEM_HD void cycle3(i64 (&v)[3]) {
    const i64 t = v[0];
    v[0] = v[1];
    v[1] = v[2];
    v[2] = t;
}
LBDEM_HD void cycle(Parts& e) {
    cycle3(e.q.d);
    cycle3(e.q.m);
    cycle3(e.o);
}

// 1 / rho in Q61 from rho in Q62 (0.4 < rho < 1.6): a float reciprocal r, its
// error e = 1 - rho r in Q59, and r (1 + e + e^2) (the next term is below 2^-66).
LBDEM_HD i64 reciprocal_q61(i64 rho) {
    const Split s = split(rho);
    const float x = (float)s.h * (1.0f / 1073741824.0f);
#ifdef __CUDA_ARCH__
    const int r = __float2int_rn(__fdividef(536870912.0f, x));
#else
    const int r = (int)(536870912.0f / x);
#endif
    const i64 e = ((i64)1 << 59) - ((i64)s.h * r + (((i64)s.l * r) >> 32));
    const int eh = (int)(e >> 7);
    const Split c = split(e + (((i64)eh * eh) >> 45));
    return shl(r, 32) + shl((i64)c.h * r, 5) + (((i64)c.l * r) >> 27);
}

// Directions of the three cycles of the axes: pairs (k, i), c_k = -c_i, with
// c_k = e_a, e_a + e_b and +-(e_a - e_b), b the axis after a; the sign is minus in the
// last cycle (a = z, b = x), so that the directions are 10 + a, 1 + a and 13, 4, 14, 5
// plus 0, 4, 2.
LBDEM_HD constexpr int diag_of(int a) { return a == 0 ? 0 : (a == 1 ? 4 : 2); }
LBDEM_HD constexpr int dir_of(int a, int q) {   // q = 0..5: k, i of the three pairs
    return q == 0 ? 10 + a : q == 1 ? 1 + a : (q == 2 ? 13 : q == 3 ? 4 : q == 4 ? 14 : 5) + diag_of(a);
}
struct Sums {
    i64 rb, j[3];
};
// Adds the six populations of a cycle and cycles the axes of j.
LBDEM_HD void add_three(Sums& s, const i64 (&x)[6], bool last) {
    const i64 d4 = last ? x[5] - x[4] : x[4] - x[5];
    s.rb += ((x[0] + x[1]) + (x[2] + x[3])) + (x[4] + x[5]);
    s.j[0] += (x[0] - x[1]) + ((x[2] - x[3]) + d4);
    s.j[1] += (x[2] - x[3]) - d4;
    cycle3(s.j);
}

// What the update of a cell needs besides its populations.
struct Cell {
    Parts eq;       // feq(J)
    Parts fs;       // S (with a body force; else eq is taken)
    Parts df;       // solid; with a body force feq(P) - feq(j*), odd parts added; else Dl
    Split A, A0, B; // A0 = A + B (without a body force)
};

// From the sums of the cell's populations; returns the force in F (solid).
// emax: cell_exponent() of the cell, at least EMAX_LO.  gx, gy, gz: body force (FORCE);
// full: n = 125.
template <bool FORCE>
LBDEM_HD Cell cell_setup(bool solid, const Sums& m, int emax, const Relax& rx, double gx, double gy, double gz,
                         bool full, double Bd, double up0, double up1, double up2, double (&F)[3]) {
    Cell c;
    // rho = 1 + rhoBar in Q62: a unit is 2^(emax - 1079)
    const i64 rbq = m.rb >> imin(1017 - emax, 63);
    const Split rq = split(rbq);
    const int sh = imin(1018 - emax, 62);        // >= 1
    const i64 half = (i64)1 << (sh - 1);
    const Split inv = split(reciprocal_q61(((i64)1 << 62) + rbq));
    i64 js[3] = {m.j[0], m.j[1], m.j[2]};        // j*
    Tensor qs;                                   // j* j* / rho
    if (FORCE) {
        // rho g, J = j + rho g / 2 and pre g
        const i64 g[3] = {to_fixed<4 + UP_BITS>(gx, emax), to_fixed<4 + UP_BITS>(gy, emax),
                          to_fixed<4 + UP_BITS>(gz, emax)};
        i64 J[3], pg[3];
        Split JS[3], U[3], W[3];
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const i64 rg = g[a] + mul<62>(split(g[a]), rq);
            J[a] = m.j[a] + ((rg + 1) >> 1);
            pg[a] = mul<62>(split(rg), rx.hom);
            JS[a] = split(J[a]);
            U[a] = split(mul<61>(JS[a], inv));
            W[a] = split(pg[a]);
            if (!full) js[a] += rg;
        }
        const Tensor q = tensor_of(JS, U, sh, half);
        c.eq = parts_of(m.rb, q, J[0], J[1], J[2]);
        Tensor s;
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const int b = (a + 1) % 3;
            s.d[a] = q.d[a] + ((mul<61>(U[a], W[a]) + (half >> 1)) >> (sh - 1));   // 2 u_a pre g_a
            s.m[a] = q.m[a] + ((mul<61>(U[a], W[b]) + mul<61>(U[b], W[a]) + half) >> sh);
        }
        c.fs = parts_of(m.rb, s, J[0] + pg[0], J[1] + pg[1], J[2] + pg[2]);
        if (solid) {
            const Split S[3] = {split(js[0]), split(js[1]), split(js[2])};
            const Split V[3] = {split(mul<61>(S[0], inv)), split(mul<61>(S[1], inv)), split(mul<61>(S[2], inv))};
            qs = tensor_of(S, V, sh, half);
        }
    } else {
        const Split J[3] = {split(m.j[0]), split(m.j[1]), split(m.j[2])};
        const Split U[3] = {split(mul<61>(J[0], inv)), split(mul<61>(J[1], inv)), split(mul<61>(J[2], inv))};
        qs = tensor_of(J, U, sh, half);
        c.eq = parts_of(m.rb, qs, m.j[0], m.j[1], m.j[2]);
    }
    c.A = c.A0 = rx.om1;
    c.B = Split{0, 0};
    c.df = Parts{};
    F[0] = F[1] = F[2] = 0.0;
    if (solid) {
        const i64 Bq = to_q62(Bd);
        c.B = split(Bq);
        const i64 Aq = (shl(rx.om1.h, 32) + rx.om1.l) - mul<62>(rx.om1, c.B);
        c.A = split(Aq);
        if (!FORCE) c.A0 = split(Aq + Bq);
        const i64 u[3] = {to_fixed<4 + UP_BITS>(up0, emax), to_fixed<4 + UP_BITS>(up1, emax),
                          to_fixed<4 + UP_BITS>(up2, emax)};
        const Split U[3] = {split(u[0]), split(u[1]), split(u[2])};
        const i64 P[3] = {u[0] + mul<62>(U[0], rq), u[1] + mul<62>(U[1], rq), u[2] + mul<62>(U[2], rq)};
        const Split PS[3] = {split(P[0]), split(P[1]), split(P[2])};
        Tensor d = tensor_of(PS, U, sh, half);   // P P / rho, P = rho u_p
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            d.d[a] = FORCE ? d.d[a] - qs.d[a] : qs.d[a] - d.d[a];
            d.m[a] = FORCE ? d.m[a] - qs.m[a] : qs.m[a] - d.m[a];
        }
        const i64 v[3] = {m.j[0] - P[0], m.j[1] - P[1], m.j[2] - P[2]};
        if (FORCE) c.df = parts_of(0, d, js[0] + P[0], js[1] + P[1], js[2] + P[2]);
        else c.df = parts_of(0, d, v[0], v[1], v[2]);
#pragma unroll
        for (int a = 0; a < 3; ++a)
            F[a] = to_double(mul<62>(split(FORCE ? v[a] - (js[a] - m.j[a]) : v[a]), c.B), emax);
    }
    return c;
}

// s + a g + b h, both products rounded together.
LBDEM_HD double relaxed(bool solid, i64 s0, i64 g, const Split& a, i64 h, const Split& b, int emax) {
    const Split gs = split(g);
    i64 t = (i64)gs.h * a.l + ((i64)gs.l * a.h + ((i64)1 << 29));
    i64 s = (i64)gs.h * a.h;
    if (solid) {
        const Split hs = split(h);
        t = (i64)hs.h * b.l + ((i64)hs.l * b.h + t);
        s = (i64)hs.h * b.h + s;
    }
    return to_double(s0 + shl(s, 2) + (t >> 30), emax);
}
template <bool FORCE>
LBDEM_HD double update_rest(bool solid, const Cell& c, i64 X0, int emax) {
    if (FORCE) return relaxed(solid, c.fs.b3, X0 - c.eq.b3, c.A, X0 - c.df.b3 - c.fs.b3, c.B, emax);
    return relaxed(solid, c.eq.b3, X0 - c.eq.b3, c.A0, c.df.b3, c.B, emax);
}
// One pair (k, i): populations in units in, doubles out; feq = C +- L, S = Cs +- Ls (with a
// body force), the solid parts Cd +- Ld.
template <bool FORCE>
LBDEM_HD void update_pair(bool solid, const Cell& c, i64 C, i64 L, i64 Cs, i64 Ls, i64 Cd, i64 Ld, i64 Xk, i64 Xi,
                          int emax, double& fk, double& fi) {
    if (!FORCE) {
        const i64 ek = C + L, ei = C - L;
        const i64 gk = Xk - ek, gi = Xi - ei;
        fk = relaxed(solid, ek, gk, c.A, gi - (Cd + Ld), c.B, emax);
        fi = relaxed(solid, ei, gi, c.A, gk - (Cd - Ld), c.B, emax);
        return;
    }
    const i64 sk = Cs + Ls, si = Cs - Ls;
    fk = relaxed(solid, sk, Xk - (C + L), c.A, (Xi - sk) + (Cd + Ld), c.B, emax);
    fi = relaxed(solid, si, Xi - (C - L), c.A, (Xk - si) + (Cd - Ld), c.B, emax);
}

// The three pairs of the current cycle: X(q) is a population in units, put(q, f) takes
// the result, q = 0..5 as in dir_of.  Every result is converted with two double
// additions: the FP64 pipe is otherwise idle, and 38 additions cost it less time than
// integer conversions take (128^3 cycle 586, 567, 550, 543 us with none, one, two and
// all three pairs converted this way).
template <bool FORCE, typename In, typename Out>
LBDEM_HD void update_three(bool solid, Cell& c, bool last, const In& X, int emax, const Out& put) {
    const Three e = three_of(c.eq, last);
    Three s = e, d{};
    if (FORCE) s = three_of(c.fs, last);
    if (solid) d = three_of(c.df, last);
    double fk, fi;
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        update_pair<FORCE>(solid, c, e.C[q], e.L[q], s.C[q], s.L[q], d.C[q], d.L[q], X(2 * q), X(2 * q + 1), emax, fk, fi);
        put(2 * q, fk);
        put(2 * q + 1, fi);
    }
    cycle(c.eq);
    if (FORCE) cycle(c.fs);
    if (solid) cycle(c.df);
}

// One cell with its populations in an array (the kernel runs the same loops over its
// stage).  solid adds the solid correction with the weight B and the surface velocity
// (up0, up1, up2); a fluid cell (B = 0, up = 0) gets the same bits either way.
// emax: cell_exponent() of the same values, fits(emax).
template <bool FORCE>
LBDEM_HD void collide(bool solid, double (&f)[19], int emax, const Relax& rx, double gx, double gy, double gz,
                      bool full, double B, double up0, double up1, double up2, double (&F)[3]) {
    emax = imax(emax, EMAX_LO);
    i64 X[19];
#pragma unroll
    for (int i = 0; i < 19; ++i) X[i] = to_fixed<4>(f[i], emax);
    Sums s{X[0], {0, 0, 0}};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const i64 x[6] = {X[dir_of(a, 0)], X[dir_of(a, 1)], X[dir_of(a, 2)],
                          X[dir_of(a, 3)], X[dir_of(a, 4)], X[dir_of(a, 5)]};
        add_three(s, x, a == 2);
    }
    Cell c = cell_setup<FORCE>(solid, s, emax, rx, gx, gy, gz, full, B, up0, up1, up2, F);
    f[0] = update_rest<FORCE>(solid, c, X[0], emax);
#pragma unroll
    for (int a = 0; a < 3; ++a)
        update_three<FORCE>(solid, c, a == 2, [&](int q) { return X[dir_of(a, q)]; }, emax,
                            [&](int q, double v) { f[dir_of(a, q)] = v; });
}

}  // namespace fixed
}  // namespace lbdem
