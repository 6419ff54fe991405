// K2: sphere voxelization, bit-exact with SetSingleSphere3D.
//
// Replaces setSpheresOnLattice -> SetSingleSphere3D::process for every sphere
// (src/ibDataExchangeWrappers3D.hh:33-146, src/ibProcessors3D.hh:53-184).
//
// Order.  The reference applies spheres one after another, and a cell's new
// state depends on its previous state and on the order of the spheres whose
// bounding box covers it (decFlag, src/ibProcessors3D.hh:85-105).  The GPU
// keeps that order per cell: every sphere is binned to the 8^3-cell tiles its
// box overlaps, each tile's bin is sorted by sphere index in shared memory, and
// every cell folds the sorted list through the same state machine.  Cells are
// independent, so the result equals the sequential sweep.  A bin holds
// TILE_BIN spheres; a tile overlapped by more re-collects its spheres by
// testing every box (slow but exact).
//
// Exactness of the sub-cell count.  The reference decides, in IEEE double,
//   dist = (dx^2 + dy^2) + dz^2  against (r + sqrt(3.1)/2)^2 and (r - sqrt(3.1)/2)^2,
//   (xs_i + ys_j) + zs_k < r^2   for the 125 sub-cell centres of shell cells.
// GB300 executes double arithmetic at two lanes per clock per SM, so each
// comparison is first made in float with a margin M = 2^-19 (r + 4)^2.  For a
// cell inside the box (|dx| < r + 3, centre split x = xh + xl with |x| < 2^24)
// the float value differs from the double one by at most 27 u (r + 3.5)^2,
// u = 2^-24 (sample sums), resp. 22 u (r + 3.2)^2 (dist), so a float result
// farther than M from the threshold decides the comparison as the double
// computation does.  Only comparisons inside the band are evaluated with the
// reference's double sequence (__dadd_rn/__dmul_rn: no fused multiply-add).
// Counts n and owner tags are identical to the sequential CPU result; the
// FP64 form also reproduces the particle surface velocity bit for bit.
#include "lbdem_internal.h"

#include <climits>

namespace lbdem {
namespace {

constexpr unsigned FULL_MASK = 0xffffffffu;

constexpr double SQRT3HALF = 0.8803408430829505;  // sqrt(3.1)/2, src/ibProcessors3D.hh:128-130
// -0.5 + (i + 0.5) * (1./5.), src/ibProcessors3D.hh:141-147, evaluated in double:
__device__ __forceinline__ double sub_delta(int i) {
    return i == 0 ? -0.4 : i == 1 ? -0.19999999999999996 : i == 2 ? 0.0 : i == 3 ? 0.20000000000000007 : 0.4;
}
__device__ __forceinline__ float sub_delta_f(int i) {
    return i == 0 ? -0.4f : i == 1 ? -0.2f : i == 2 ? 0.0f : i == 3 ? 0.2f : 0.4f;
}

// Single operations with round-to-nearest and no contraction into fused
// multiply-adds (results independent of how the compiler schedules a kernel).
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double add_rn(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double sub_rn(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float add_rn(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float sub_rn(float a, float b) { return __fsub_rn(a, b); }

// Region of a cell against the early-out thresholds in the reference's double
// arithmetic: 0 outside (dist > rp2), 1 inside (dist < rm2), 2 shell.
__device__ __noinline__ int region_exact(int X, int Y, int Z, const SphereDev& s) {
    const double dx = __dsub_rn((double)X, s.x[0]);
    const double dy = __dsub_rn((double)Y, s.x[1]);
    const double dz = __dsub_rn((double)Z, s.x[2]);
    const double dist = __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
    if (dist > s.rp2) return 0;
    if (dist < s.rm2) return 1;
    return 2;
}

__device__ __forceinline__ int tiles_along(int n) { return (n + TILE - 1) / TILE; }

// Where the prepare launches put a sphere list, and what they clear beside it.
struct SphereTables {
    SphereDev* sph;
    SphereFast* fast;
    float* xpf;
    int* tag2slot;
    unsigned* err;
    double* ft_zero;      // (may be null) 6 n force/torque sums of the coming step, zeroed
    double* rec_copy;     // (may be null, never overlapping the source) a copy of the records
};

// Per sphere: bounding box (double -> integer truncation toward zero,
// src/ibProcessors3D.h:43-45) intersected with the lattice
// (src/ibDataExchangeWrappers3D.hh:127-133), thresholds, the float split of
// the centre, and the tag -> lowest list index map (LAMMPS atom->map keeps the
// owned atom, which precedes its ghost images).
// L lanes (8 or 32) share a sphere: they read its record as one piece, and lanes 0-2
// take one axis each (GB300's two double lanes per clock make an instruction cost the
// same for one lane as for 32, so a warp's spheres and axes go through it together).
// Returns, in lane d < 3 of the sphere, the cell range along axis d that its tiles are
// binned by, lo > hi in all of them when the sphere reaches no cell.  `on`: the lanes
// that hold a sphere.  Must be reached by all 32 lanes.
template <int L>
__device__ __forceinline__ void prepare_sphere(const double* __restrict__ p, bool on, int i, int il, int n,
                                               const Geom& g, int max_tag, double max_radius, const SphereTables& t,
                                               int& blo, int& bhi) {
    const int lane = threadIdx.x & 31, sub = lane % L, base = lane - sub;
    double ra = 0.0, rb = 0.0;   // record words sub and (L < 12) L + sub
    if (on && sub < REC_STRIDE) ra = p[sub];
    if (L < REC_STRIDE && on && sub < REC_STRIDE - L) rb = p[L + sub];
    if (on && t.rec_copy) {
        double* c = t.rec_copy + (size_t)i * REC_STRIDE;
        if (sub < REC_STRIDE) c[sub] = ra;
        if (L < REC_STRIDE && sub < REC_STRIDE - L) c[L + sub] = rb;
    }
    if (on && t.ft_zero && sub < 6) t.ft_zero[(size_t)sub * n + i] = 0.0;
    auto word = [&](int k) -> double {
        const double a = __shfl_sync(FULL_MASK, ra, base + (k % L));
        if (L >= REC_STRIDE) return a;
        const double b = __shfl_sync(FULL_MASK, rb, base + (k % L));
        return k < L ? a : b;
    };
    const int d = min(sub, 2);
    const double x = word(d), v = word(3 + d), w = word(6 + d), r = word(9), tagd = word(10);
    const int dim = d == 0 ? g.nx : (d == 1 ? g.ny : g.nz);
    const bool tag_ok = tagd >= 1.0 && tagd <= (double)max_tag;
    const bool r_ok = r > 0.0 && r <= max_radius;
    // |x| < 2^24 keeps the integer conversions defined and the float split
    // accurate; a sphere farther out cannot reach the lattice.
    const bool x_ok = x > -16777216.0 && x < 16777216.0;
    float xh = 0.f, xl = 0.f;
    int lo = 1, hi = 0;
    if (x_ok) {
        xh = (float)x;
        xl = (float)(x - (double)xh);
        long long l = (long long)(__dsub_rn(__dsub_rn(x, r), 2.0));
        long long h = (long long)(__dadd_rn(__dadd_rn(x, r), 2.0));
        if (l < 0) l = 0;
        if (h > dim - 1) h = dim - 1;
        lo = (int)(l < (long long)dim ? l : dim);
        hi = (int)(h > -1 ? h : -1);
    }
    const unsigned good = __ballot_sync(FULL_MASK, x_ok && lo <= hi);
    const bool valid = tag_ok && r_ok && ((good >> base) & 7u) == 7u;
    blo = on && valid ? lo : 1;
    bhi = on && valid ? hi : 0;
    if (!on) return;
    const int tag = tag_ok ? (int)tagd : 0;
    SphereDev& s = t.sph[i];
    SphereFast& q = t.fast[i];
    float* xp = t.xpf + (size_t)i * XPF_STRIDE;
    const float vf = (float)v, wf = (float)w;
    if (sub < 3) {
        s.x[sub] = x; s.v[sub] = v; s.w[sub] = w;
        s.lo[sub] = lo; s.hi[sub] = hi;
        q.xh[sub] = xh; q.xl[sub] = xl;
        q.lo[sub] = blo; q.hi[sub] = bhi;
        q.v[sub] = vf; q.w[sub] = wf;
        xp[sub] = xh; xp[3 + sub] = xl; xp[6 + sub] = vf; xp[9 + sub] = wf; xp[12 + sub] = 0.f;
    }
    const double rp = __dadd_rn(r, SQRT3HALF), rm = __dsub_rn(r, SQRT3HALF);
    const double rp2 = __dmul_rn(rp, rp), rm2 = __dmul_rn(rm, rm), rsq = __dmul_rn(r, r);
    const float r4 = (float)r + 4.0f;
    if (sub == 3) {
        s.r = r; s.rp2 = rp2; s.rm2 = rm2; s.rsq = rsq;
        s.tag = tag; s.valid = valid ? 1 : 0;
        q.rp2 = (float)rp2; q.rm2 = (float)rm2; q.rsq = (float)rsq;
        q.margin = ldexpf(r4 * r4, -19);
        q.tag = tag; q.pad = 0;
        xp[15] = 0.f;
        if (!tag_ok) atomicOr(t.err, 0x4u);  // LBDEM_DEVERR_TAG_RANGE
        if (!r_ok) atomicOr(t.err, 0x10u);   // LBDEM_DEVERR_RADIUS
        if (tag >= 1) atomicMin(t.tag2slot + tag, il);
    }
}

// A warp prepares 32 / L spheres, then its lanes stride over the tiles that each
// sphere's box overlaps and append the sphere to each
// tile's bin (entries past TILE_BIN are dropped; the voxelization of such a
// tile re-collects its spheres; a tile's bin is rank-sorted there, so the
// append order does not matter).  The first sphere of a tile also appends the
// tile to the work list.
// BATCH: slot i belongs to the domain d with soff[d] <= i; slots past the
// domain's particle count are skipped; the map stores domain-local slots.
// old: a list whose entries in its own tag map are cleared by the way (map null: none).
// L = 32, one sphere per warp, is the shorter chain for short lists; L = 8 shares the
// double instructions of four spheres (PREPARE_WIDE).
struct OldList {
    int* map;
    const double* rec;
    int n, max_tag;
};
template <bool BATCH, int L>
__global__ void k_prepare_bin(const double* __restrict__ rec, int n, SphereTables t, Geom g, int max_tag,
                              double max_radius, const DomView* __restrict__ doms, const int* __restrict__ soff,
                              int ndom, const int* __restrict__ ncur, int* __restrict__ tile_cnt,
                              int* __restrict__ bins, int* __restrict__ work, int* __restrict__ work_n, OldList old) {
    const int lane = threadIdx.x & 31;
    const int i = (blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * (32 / L) + lane / L;
    if (old.map)
        for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < old.n; k += gridDim.x * blockDim.x) {
            const double tagd = old.rec[(size_t)k * REC_STRIDE + 10];
            if (tagd >= 1.0 && tagd <= (double)old.max_tag) old.map[(int)tagd] = NO_SLOT;
        }
    bool on = i < n;
    int il = i, t0 = 0;
    if (BATCH) {
        if (on) {
            const int d = find_domain(soff, ndom, i);
            il = i - __ldg(soff + d);
            const DomView& D = doms[d];
            g = D.g;
            t.tag2slot += D.tag0;
            t0 = D.t0;
            if (t.ft_zero && lane % L < 6) t.ft_zero[(size_t)(lane % L) * n + i] = 0.0;   // unused slots too
            on = il < __ldg(ncur + d);
        }
    }
    int blo, bhi;
    prepare_sphere<L>(rec + (size_t)(on ? i : 0) * REC_STRIDE, on, i, il, n, g, max_tag, max_radius, t, blo, bhi);
    const int my_tny = tiles_along(g.ny), my_tnz = tiles_along(g.nz);
#pragma unroll
    for (int q = 0; q < 32; q += L) {
        const int x0 = __shfl_sync(FULL_MASK, blo, q), x1 = __shfl_sync(FULL_MASK, bhi, q);
        const int y0 = __shfl_sync(FULL_MASK, blo, q + 1), y1 = __shfl_sync(FULL_MASK, bhi, q + 1);
        const int z0 = __shfl_sync(FULL_MASK, blo, q + 2), z1 = __shfl_sync(FULL_MASK, bhi, q + 2);
        const int ql = __shfl_sync(FULL_MASK, il, q), qt0 = __shfl_sync(FULL_MASK, t0, q);
        const int tny = BATCH ? __shfl_sync(FULL_MASK, my_tny, q) : my_tny;
        const int tnz = BATCH ? __shfl_sync(FULL_MASK, my_tnz, q) : my_tnz;
        if (x0 > x1) continue;   // warp-uniform: no sphere, or one that reaches no cell
        const int tx0 = x0 / TILE, ty0 = y0 / TILE, tz0 = z0 / TILE;
        const int ex = x1 / TILE - tx0 + 1, ey = y1 / TILE - ty0 + 1, ez = z1 / TILE - tz0 + 1;
        const int total = ex * ey * ez;
        for (int k = lane; k < total; k += 32) {
            const int kz = k % ez, kr = k / ez;
            const int ky = kr % ey, kx = kr / ey;
            const size_t tile = (size_t)qt0 + ((size_t)(tx0 + kx) * tny + (ty0 + ky)) * tnz + (tz0 + kz);
            const int pos = atomicAdd(tile_cnt + tile, 1);
            if (pos == 0) work[atomicAdd(work_n, 1)] = (int)tile;
            if (pos < TILE_BIN) bins[tile * TILE_BIN + pos] = ql;
        }
    }
}

// The tables without the bins.
__global__ void k_prepare(const double* __restrict__ rec, int n, SphereTables t, Geom g, int max_tag,
                          double max_radius) {
    const int i = (blockIdx.x * blockDim.x + threadIdx.x) / 8;
    int blo, bhi;
    prepare_sphere<8>(rec + (size_t)(i < n ? i : 0) * REC_STRIDE, i < n, i, i, n, g, max_tag, max_radius, t, blo, bhi);
}

// Location of population i of cell c in the AA layout (phase = completed steps mod 2).
template <typename T>
__device__ __forceinline__ T* pop_slot(T* f, int i, int x, int y, int z, int phase, const Geom& g) {
    if (phase == 0 || i == 0) return f + (size_t)i * g.N + ((size_t)x * g.ny + y) * g.nz + z;
    // odd layout: f_i(x) sits in slot (opp i, x - c_i), or (i, x) when x - c_i is beyond a wall
    int X = x - cx(i), Y = y - cy(i), Z = z - cz(i);
    bool out = false;
    if (X < 0 || X >= g.nx) { if (g.per[0]) X = (X + g.nx) % g.nx; else out = true; }
    if (Y < 0 || Y >= g.ny) { if (g.per[1]) Y = (Y + g.ny) % g.ny; else out = true; }
    if (Z < 0 || Z >= g.nz) { if (g.per[2]) Z = (Z + g.nz) % g.nz; else out = true; }
    if (out) return f + (size_t)i * g.N + ((size_t)x * g.ny + y) * g.nz + z;
    return f + (size_t)opp(i) * g.N + ((size_t)X * g.ny + Y) * g.nz + Z;
}

// setValues, src/ibProcessors3D.hh:163-174 (com == x for single spheres):
// u = v + omega x (cell - com), in the reference's double operation order.
__device__ __forceinline__ void surface_velocity(const SphereDev& s, int X, int Y, int Z, double& u0, double& u1,
                                                 double& u2) {
    const double dx = __dsub_rn((double)X, s.x[0]);
    const double dy = __dsub_rn((double)Y, s.x[1]);
    const double dz = __dsub_rn((double)Z, s.x[2]);
    u0 = __dadd_rn(s.v[0], __dsub_rn(__dmul_rn(s.w[1], dz), __dmul_rn(s.w[2], dy)));
    u1 = __dadd_rn(s.v[1], __dadd_rn(__dmul_rn(-s.w[0], dz), __dmul_rn(s.w[2], dx)));
    u2 = __dadd_rn(s.v[2], __dsub_rn(__dmul_rn(s.w[0], dy), __dmul_rn(s.w[1], dx)));
}

// Packed pairs of floats for the sample sums.
__device__ __forceinline__ unsigned long long pk2(float a, float b) {
    unsigned long long v;
    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(a), "f"(b));
    return v;
}
__device__ __forceinline__ unsigned long long add2(unsigned long long a, unsigned long long b) {
    unsigned long long d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ unsigned long long sub2(unsigned long long a, unsigned long long b) {
    unsigned long long d;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
// Sub-cell count of one x-slice (i fixed: 25 of the 125 samples) of a shell
// cell in float, every operation rounded on its own (the error bound of the
// header holds for this form): the sums t = (xs + ys_j) + zs_k are formed two
// at a time in packed f32x2 arithmetic, d = t - r^2 (exact near r^2), and a
// sample is inside when the sign bit of d is set.  *unsure is set when some
// |d| <= M (a sample inside the decision band).
__device__ __forceinline__ int slice_count_fast(float dxf, float dyf, float dzf, int i, float rsq, float M,
                                                bool* unsure) {
    const float ax = __fadd_rn(dxf, sub_delta_f(i));
    const float xs = __fmul_rn(ax, ax);
    float ys[5], zs[5];
#pragma unroll
    for (int j = 0; j < 5; ++j) {
        const float d = sub_delta_f(j);
        const float ay = __fadd_rn(dyf, d); ys[j] = __fmul_rn(ay, ay);
        const float az = __fadd_rn(dzf, d); zs[j] = __fmul_rn(az, az);
    }
    const unsigned long long z01 = pk2(zs[0], zs[1]), z23 = pk2(zs[2], zs[3]), r2 = pk2(rsq, rsq);
    unsigned neg = 0u;
    float mind = 3.0e38f;
#pragma unroll
    for (int j = 0; j < 5; ++j) {
        const float a = __fadd_rn(xs, ys[j]);
        const unsigned long long a2 = pk2(a, a);
        const unsigned long long d01 = sub2(add2(a2, z01), r2), d23 = sub2(add2(a2, z23), r2);
        const float d4 = __fsub_rn(__fadd_rn(a, zs[4]), rsq);
        const unsigned u0 = (unsigned)d01, u1 = (unsigned)(d01 >> 32), u2 = (unsigned)d23, u3 = (unsigned)(d23 >> 32);
        neg += (u0 >> 31) + (u1 >> 31) + (u2 >> 31) + (u3 >> 31) + (__float_as_uint(d4) >> 31);
        mind = fminf(mind, fminf(fminf(fabsf(__uint_as_float(u0)), fabsf(__uint_as_float(u1))),
                                 fminf(fminf(fabsf(__uint_as_float(u2)), fabsf(__uint_as_float(u3))), fabsf(d4))));
    }
    *unsure = !(mind > M);
    return (int)neg;
}

// The same slice with the samples inside the band decided by the reference's
// double sequence ((xs_i + ys_j) + zs_k < r^2, src/ibProcessors3D.hh:141-155).
// Inlined into the count loop (a call there cost its register saves and restores on
// every pass, 0.235 against 0.227 ms; the cell-distance routine region_exact stays out
// of line, inlining it measured slower).
__device__ __forceinline__ int slice_count_resolve(float dxf, float dyf, float dzf, int i, float rsq, float M, int X,
                                                int Y, int Z, const SphereDev& s) {
    const double dx = __dsub_rn((double)X, s.x[0]);
    const double dy = __dsub_rn((double)Y, s.x[1]);
    const double dz = __dsub_rn((double)Z, s.x[2]);
    const double axd = __dadd_rn(dx, sub_delta(i));
    const double xsd = __dmul_rn(axd, axd);
    const float ax = dxf + sub_delta_f(i);
    const float xs = ax * ax;
    const float lo = rsq - M, hi = rsq + M;
    int n = 0;
    for (int j = 0; j < 5; ++j) {
        const float ay = dyf + sub_delta_f(j);
        const float a = xs + ay * ay;
        double ad = 0.0;
        bool have_ad = false;
        for (int k = 0; k < 5; ++k) {
            const float az = dzf + sub_delta_f(k);
            const float t = a + az * az;
            if (t < lo) {
                ++n;
            } else if (t < hi) {
                if (!have_ad) {
                    const double ayd = __dadd_rn(dy, sub_delta(j));
                    ad = __dadd_rn(xsd, __dmul_rn(ayd, ayd));
                    have_ad = true;
                }
                const double azd = __dadd_rn(dz, sub_delta(k));
                n += (__dadd_rn(ad, __dmul_rn(azd, azd)) < s.rsq) ? 1 : 0;
            }
        }
    }
    return n;
}

// ---------------------------------------------------------------------------
// Voxelization, one warp per 8^3 tile.
//
// The tile's cell state (voxel words, and per cell the list index of the
// sphere that last set or cleared it) lives in per-warp shared memory while
// the tile's spheres are applied in list order.  Lane `lane` handles cells
// l = lane + 32 j (j = 0..15): the half x-plane j holds x = j >> 1,
// y = (lane >> 3) + 4 (j & 1), z = lane & 7.  Per sphere (apply_sphere):
//  1  the half-planes that meet the sphere's box are classified in float
//     (outside: n = 0, inside: n = 125, shell); comparisons within the float
//     error band are decided in the reference's double arithmetic; outside and
//     inside cells are folded through decFlag at once, shell cells queued;
//  2  all lanes take the queued cells' sub-cell counts, five x-slices (25
//     samples) per cell, added into per-cell bytes with shared-memory atomics;
//  3  the queued cells are folded through decFlag.
// No block-wide barrier is involved, so the warps of a block work on
// unrelated tiles.  The spheres of a tile come from its bin (at most
// TILE_BIN, put in ascending list order by repeated warp minima), or, for a
// tile whose bin overflowed, from a scan of every sphere's box in list order.
constexpr int VOX_WARPS = 8;                        // warps per block
constexpr int VOX_THREADS = 32 * VOX_WARPS;
constexpr int VOX_STAGE = 32;                       // sphere records staged at a time
constexpr int VOX_SLAB_ROUNDS = 2;
// A tile's sphere count and, above it, the arrivals of its warps (at most 8).
constexpr int TILE_CNT_BITS = 28;
constexpr unsigned TILE_CNT_MASK = (1u << TILE_CNT_BITS) - 1u;
constexpr int TOFF_SMEM = 512;                      // batch: domains whose first tiles a CTA keeps
constexpr uint32_t SETTER_ZERO = 0xffffffffu;       // the cell was set to zero (setToZero)
constexpr uint32_t SETTER_KEEP = 0xfffffffeu;       // the cell keeps its state (and velocity)

// Per-warp shared memory.  setter: the list index of the sphere that last set
// the cell in this pass (or SETTER_ZERO / SETTER_KEEP); defv (INIT_VEL): the
// setter code at the cell's last full coverage (defineVelocity), SETTER_ZERO
// + SETTER_KEEP markers as for setter, DEFV_NONE without full coverage.
constexpr uint32_t DEFV_NONE = 0xfffffffdu;
template <bool INIT_VEL>
struct alignas(16) WarpVox {
    SphereFast q[VOX_STAGE];                        // staged sphere records
    int list[TILE_BIN];                             // the tile's spheres in list order
    uint32_t w[TILE_CELLS];                         // voxel words (n | tag << 7)
    uint32_t setter[TILE_CELLS];
    uint32_t defv[INIT_VEL ? TILE_CELLS : 1];
    uint32_t cnt4[TILE_CELLS / 4];                  // shell sub-cell counts, one byte per cell
    uint16_t queue[TILE_CELLS];                     // shell cells of the current sphere
    uint16_t items[5 * 32];                         // x-slices left to count: tile cell << 3 | slice
};

// decFlag, src/ibProcessors3D.hh:85-105 (sf > 0.001 <=> n > 0; sf > sf_old <=>
// n > n_old), for cell l with the sub-cell count n of sphere m.
template <bool INIT_VEL>
__device__ __forceinline__ void fold_cell(WarpVox<INIT_VEL>& S, int l, uint32_t n, uint32_t tag, int m) {
    const uint32_t w = S.w[l];
    const uint32_t nold = w & VOX_NMASK, idold = w >> VOX_NBITS;
    const int dec = (n > 0u ? 1 : 0) + (nold > 0u ? 2 : 0);
    if (dec == 2 && idold == tag) {
        S.w[l] = 0u;
        S.setter[l] = SETTER_ZERO;
    } else if (dec == 1 || (dec == 3 && ((n > nold) || (idold == tag)))) {
        S.w[l] = n | (tag << VOX_NBITS);
        S.setter[l] = (uint32_t)m;
    }
    // dec == 0 is setToZero on a cell that is already empty
    // the velocity the cell holds right after this sphere (src/ibProcessors3D.hh:107-108)
    if (INIT_VEL && n == 125u) S.defv[l] = S.setter[l];
}

// Steps 1-3 above for sphere m (float record q in shared memory) on the x-planes
// xa..xb of the tile at (X0, Y0, Z0).  Inlined at both sphere sources (an out-of-line routine measured
// 5 % slower: the call's register saves and restores).
template <bool INIT_VEL>
__device__ __forceinline__ void apply_sphere(WarpVox<INIT_VEL>& S, const SphereFast& q, int m,
                                          const SphereDev* __restrict__ sph, int X0, int Y0, int Z0, int xa, int xb) {
    const int lane = threadIdx.x & 31;
    const int bx0 = max(q.lo[0] - X0, xa), bx1 = min(q.hi[0] - X0, xb);
    const int by0 = max(q.lo[1] - Y0, 0), by1 = min(q.hi[1] - Y0, TILE - 1);
    const int bz0 = max(q.lo[2] - Z0, 0), bz1 = min(q.hi[2] - Z0, TILE - 1);
    if (bx0 > bx1 || by0 > by1 || bz0 > bz1) return;
    const float M = q.margin, rp2 = q.rp2, rm2 = q.rm2;
    const uint32_t tag = (uint32_t)q.tag;
    const int z = lane & 7, yl = lane >> 3;
    const bool zin = z >= bz0 && z <= bz1;
    const float dzf = ((float)(Z0 + z) - q.xh[2]) - q.xl[2];
    uint8_t* cnt8 = reinterpret_cast<uint8_t*>(S.cnt4);
    const unsigned below = (1u << lane) - 1u;
    int qn = 0;
    // 1: the box's cells of the tile, x-plane by x-plane in the half-planes h
    // (rows y = yl + 4 h) that meet the box's y range.  The squared distance is
    // formed as dx^2 + (dy^2 + dz^2), every rounding explicit, the x-free part
    // once per lane and half-plane.
    const float dz2 = __fmul_rn(dzf, dzf);
    float sh[2];
    bool inh[2], meet[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int y = yl + 4 * h;
        const float dyf = ((float)(Y0 + y) - q.xh[1]) - q.xl[1];
        sh[h] = __fmaf_rn(dyf, dyf, dz2);
        inh[h] = zin && y >= by0 && y <= by1;
        meet[h] = !(4 * h > by1 || 4 * h + 3 < by0);   // warp-uniform
    }
    // A sphere whose shell stays clear of the box's cells in this tile (about half
    // of the (tile, sphere) pairs at r = 8) only clears the cells that hold its tag
    // (decFlag 2, setToZero): the box's squared distance from the centre, formed
    // like a cell's, is more than 2 M beyond (r + sqrt(3.1)/2)^2, so every cell of the
    // box is outside in the reference's double arithmetic too.
    {
        auto gap = [](float lo, float hi) { return fmaxf(0.f, fmaxf(lo, -hi)); };
        const float ex = gap(((float)(X0 + bx0) - q.xh[0]) - q.xl[0], ((float)(X0 + bx1) - q.xh[0]) - q.xl[0]);
        const float ey = gap(((float)(Y0 + by0) - q.xh[1]) - q.xl[1], ((float)(Y0 + by1) - q.xh[1]) - q.xl[1]);
        const float ez = gap(((float)(Z0 + bz0) - q.xh[2]) - q.xl[2], ((float)(Z0 + bz1) - q.xh[2]) - q.xl[2]);
        const float d2 = __fmaf_rn(ex, ex, __fmaf_rn(ey, ey, __fmul_rn(ez, ez)));
        if (d2 > rp2 + 2.f * M) {   // warp-uniform
            for (int x = bx0; x <= bx1; ++x) {
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    if (!meet[h] || !inh[h]) continue;
                    const int l = lane + 64 * x + 32 * h;
                    const uint32_t w = S.w[l];
                    if ((w & VOX_NMASK) != 0u && (w >> VOX_NBITS) == tag) {
                        S.w[l] = 0u;
                        S.setter[l] = SETTER_ZERO;
                    }
                }
            }
            return;
        }
    }
    for (int x = bx0; x <= bx1; ++x) {
        const float dxf = ((float)(X0 + x) - q.xh[0]) - q.xl[0];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            if (!meet[h]) continue;
            int region = -1;
            if (inh[h]) {
                const float distf = __fmaf_rn(dxf, dxf, sh[h]);
                if (fabsf(distf - rp2) <= M || fabsf(distf - rm2) <= M)
                    region = region_exact(X0 + x, Y0 + yl + 4 * h, Z0 + z, sph[m]);
                else
                    region = distf > rp2 ? 0 : (distf < rm2 ? 1 : 2);
            }
            const int l = lane + 64 * x + 32 * h;
            const unsigned bal = __ballot_sync(FULL_MASK, region == 2);
            if (region == 2) {
                S.queue[qn + __popc(bal & below)] = (uint16_t)l;
            } else if (region >= 0) {
                fold_cell(S, l, region == 1 ? 125u : 0u, tag, m);
            }
            qn += __popc(bal);
        }
    }
    if (qn == 0) return;
    __syncwarp();
    // 2: counts of the queued cells, 32 at a time.  Lane `lane` takes queued
    // cell c0 + lane and decides each x-slice from its largest and smallest
    // sample sums, (xs_i + max ys) + max zs and (xs_i + min ys) + min zs: these
    // are samples of the slice, and the rounded sums are monotone in every term,
    // so a bound farther than M from r^2 decides all 25 samples as the
    // per-sample rule would (25 inside, or none).  The slices left are queued
    // and counted sample by sample, one slice per lane.
    for (int c0 = 0; c0 < qn; c0 += 32) {
        uint32_t mixed = 0u;
        int l = 0;
        if (c0 + lane < qn) {
            l = S.queue[c0 + lane];
            const int X = X0 + (l >> 6), Y = Y0 + ((l >> 3) & 7), Z = Z0 + (l & 7);
            const float dxf = ((float)X - q.xh[0]) - q.xl[0];
            const float dyf = ((float)Y - q.xh[1]) - q.xl[1];
            const float dzq = ((float)Z - q.xh[2]) - q.xl[2];
            float ymin = 3.0e38f, ymax = 0.f, zmin = 3.0e38f, zmax = 0.f;
#pragma unroll
            for (int j = 0; j < 5; ++j) {
                const float d = sub_delta_f(j);
                const float ay = __fadd_rn(dyf, d), az = __fadd_rn(dzq, d);
                const float ys = __fmul_rn(ay, ay), zs = __fmul_rn(az, az);
                ymin = fminf(ymin, ys); ymax = fmaxf(ymax, ys);
                zmin = fminf(zmin, zs); zmax = fmaxf(zmax, zs);
            }
            int inside = 0;
#pragma unroll
            for (int i = 0; i < 5; ++i) {
                const float ax = __fadd_rn(dxf, sub_delta_f(i));
                const float xs = __fmul_rn(ax, ax);
                const float hi = __fsub_rn(__fadd_rn(__fadd_rn(xs, ymax), zmax), q.rsq);
                const float lo = __fsub_rn(__fadd_rn(__fadd_rn(xs, ymin), zmin), q.rsq);
                if (hi < -M) inside += 25;
                else if (!(lo > M)) mixed |= 1u << i;
            }
            cnt8[l] = (uint8_t)inside;
        }
        const int k = __popc(mixed);
        int incl = k;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int o = __shfl_up_sync(FULL_MASK, incl, d);
            if (lane >= d) incl += o;
        }
        const int total = __shfl_sync(FULL_MASK, incl, 31);
        for (int pos = incl - k; mixed; mixed &= mixed - 1u) S.items[pos++] = (uint16_t)((l << 3) | (__ffs(mixed) - 1));
        __syncwarp();
        for (int u = lane; u < total; u += 32) {
            const int it = S.items[u];
            const int l = it >> 3, i = it & 7;
            const int X = X0 + (l >> 6), Y = Y0 + ((l >> 3) & 7), Z = Z0 + (l & 7);
            const float dxf = ((float)X - q.xh[0]) - q.xl[0];
            const float dyf = ((float)Y - q.xh[1]) - q.xl[1];
            const float dzq = ((float)Z - q.xh[2]) - q.xl[2];
            bool unsure;
            int cs = slice_count_fast(dxf, dyf, dzq, i, q.rsq, M, &unsure);
            if (unsure) cs = slice_count_resolve(dxf, dyf, dzq, i, q.rsq, M, X, Y, Z, sph[m]);
            if (cs) atomicAdd(&S.cnt4[l >> 2], (uint32_t)cs << (8 * (l & 3)));
        }
        __syncwarp();
    }
    // 3
    for (int e = lane; e < qn; e += 32) {
        const int l = S.queue[e];
        fold_cell(S, l, (uint32_t)cnt8[l], tag, m);
    }
    __syncwarp();
}

// Surface velocity of a cell set by sphere `code` (SETTER_ZERO: zero).
template <typename T>
__device__ __forceinline__ void setter_velocity(uint32_t code, const SphereDev* __restrict__ sph,
                                                const SphereFast* __restrict__ fast, int X, int Y, int Z, T& u0,
                                                T& u1, T& u2) {
    if (code == SETTER_ZERO) {
        u0 = u1 = u2 = T(0);
    } else if (sizeof(T) == 8) {
        // setValues, src/ibProcessors3D.hh:163-174 (com == x for single spheres)
        double a0, a1, a2;
        surface_velocity(sph[code], X, Y, Z, a0, a1, a2);
        u0 = T(a0); u1 = T(a1); u2 = T(a2);
    } else {
        const SphereFast& q = fast[code];
        const float dxf = ((float)X - q.xh[0]) - q.xl[0];
        const float dyf = ((float)Y - q.xh[1]) - q.xl[1];
        const float dzf = ((float)Z - q.xh[2]) - q.xl[2];
        u0 = T(add_rn(q.v[0], sub_rn(mul_rn(q.w[1], dzf), mul_rn(q.w[2], dyf))));
        u1 = T(add_rn(q.v[1], add_rn(mul_rn(-q.w[0], dzf), mul_rn(q.w[2], dxf))));
        u2 = T(add_rn(q.v[2], sub_rn(mul_rn(q.w[0], dyf), mul_rn(q.w[1], dxf))));
    }
}

// The x-planes xa..xb of one tile by one warp (parts warps take the tile's slabs).
// up == nullptr: no surface-velocity field is kept.
// INIT_VEL: defineVelocity (src/ibCompositeDynamics3D.hh:118-127) with the
// velocity a fully covered cell holds right after the last sphere covering it.
template <typename T, bool INIT_VEL>
__device__ __forceinline__ void voxelize_tile(WarpVox<INIT_VEL>& S, int t, const SphereDev* __restrict__ sph,
                                              const SphereFast* __restrict__ fast, int nsph,
                                              int* __restrict__ tile_cnt, const int* __restrict__ bins,
                                              uint32_t* __restrict__ vox, T* __restrict__ up, T* __restrict__ f,
                                              int phase, const Geom& g, const OwnerTable& ot, int xa, int xb,
                                              unsigned parts) {
    const int lane = threadIdx.x & 31;
    const int tny = tiles_along(g.ny), tnz = tiles_along(g.nz);
    const int tx = t / (tny * tnz);
    const int rem = t - tx * tny * tnz;
    const int ty = rem / tnz;
    const int tz = rem - ty * tnz;
    const int X0 = tx * TILE, Y0 = ty * TILE, Z0 = tz * TILE;
    // The tile's count, both bin slots of the lane (read whatever the count; the
    // slots past it are ignored) and its 16 voxel words are independent loads,
    // issued together so that the tile waits for one memory latency, not four.
    const int cnt = (int)((unsigned)tile_cnt[t] & TILE_CNT_MASK);
    const int a0 = bins[(size_t)t * TILE_BIN + lane];
    const int b0 = bins[(size_t)t * TILE_BIN + lane + 32];
    // cell state; a lane's cells share z and, per plane half, the row
    const int z = lane & 7, Z = Z0 + z;
    const bool zok = Z < g.nz;
    uint32_t wv[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) {
        const int X = X0 + (j >> 1), Y = Y0 + (lane >> 3) + 4 * (j & 1);
        wv[j] = (zok && X < g.nx && Y < g.ny && (j >> 1) >= xa && (j >> 1) <= xb) ? vox[((size_t)X * g.ny + Y) * g.nz + Z] : 0u;
    }
#pragma unroll
    for (int j = 0; j < 16; ++j) {
        const int l = lane + 32 * j;
        S.w[l] = wv[j];
        S.setter[l] = SETTER_KEEP;
        if (INIT_VEL) S.defv[l] = DEFV_NONE;
    }
    // the lane's bin entries (list indices)
    int a = (cnt <= TILE_BIN && lane < cnt) ? a0 : INT_MAX;
    int b = (cnt <= TILE_BIN && lane + 32 < cnt) ? b0 : INT_MAX;
    if (cnt <= 0) return;   // (a listed tile has a sphere)
    // the bins are reused by the next voxelization: the count is zeroed by the last of
    // the tile's warps to have read it (arrivals in the bits above TILE_CNT_MASK; a warp
    // arrives when every lane of it has)
    __syncwarp();
    if (lane == 0) {
        if (parts == 1 || atomicAdd((unsigned*)(tile_cnt + t), TILE_CNT_MASK + 1u) >> TILE_CNT_BITS == parts - 1u)
            tile_cnt[t] = 0;
    }
    constexpr int W4 = (int)(sizeof(SphereFast) / 16);
    const uint4* src = reinterpret_cast<const uint4*>(fast);
    uint4* dst = reinterpret_cast<uint4*>(S.q);
    if (cnt <= TILE_BIN) {
        for (int k = 0; k < cnt; ++k) {
            const int m = __reduce_min_sync(FULL_MASK, min(a, b));
            if (a == m) a = INT_MAX;
            if (b == m) b = INT_MAX;
            if (lane == 0) S.list[k] = m;
        }
        for (int base = 0; base < cnt; base += VOX_STAGE) {
            const int nst = min(VOX_STAGE, cnt - base);
            __syncwarp();
            for (int i = lane; i < W4 * nst; i += 32) {
                const int e = i / W4;
                dst[i] = __ldg(src + (size_t)S.list[base + e] * W4 + (i - W4 * e));
            }
            __syncwarp();
            for (int k = 0; k < nst; ++k) apply_sphere(S, S.q[k], S.list[base + k], sph, X0, Y0, Z0, xa, xb);
        }
    } else {
        // bin overflow: every sphere whose box reaches the tile, in list order
        for (int base = 0; base < nsph; base += 32) {
            const int i = base + lane;
            bool hit = false;
            if (i < nsph) {
                const SphereFast& q = fast[i];
                hit = q.lo[0] <= q.hi[0] && q.lo[1] <= q.hi[1] && q.lo[2] <= q.hi[2] && q.lo[0] <= X0 + TILE - 1 &&
                      q.hi[0] >= X0 && q.lo[1] <= Y0 + TILE - 1 && q.hi[1] >= Y0 && q.lo[2] <= Z0 + TILE - 1 &&
                      q.hi[2] >= Z0;
            }
            unsigned bal = __ballot_sync(FULL_MASK, hit);
            while (bal) {
                const int m = base + __ffs(bal) - 1;
                bal &= bal - 1u;
                __syncwarp();
                if (lane < W4) dst[lane] = __ldg(src + (size_t)m * W4 + lane);
                __syncwarp();
                apply_sphere(S, S.q[0], m, sph, X0, Y0, Z0, xa, xb);
            }
        }
    }
    __syncwarp();

    // defineVelocity first: it may need the surface velocity a cell held before this pass
    if (INIT_VEL) {
#pragma unroll 1
        for (int j = 0; j < 16; ++j) {
            const int l = lane + 32 * j;
            const uint32_t code = S.defv[l];
            if (code == DEFV_NONE) continue;
            const int X = X0 + (j >> 1), Y = Y0 + (lane >> 3) + 4 * (j & 1);
            const size_t c = ((size_t)X * g.ny + Y) * g.nz + Z;
            T d0, d1, d2;
            if (code == SETTER_KEEP && up != nullptr) {
                d0 = up[c]; d1 = up[g.N + c]; d2 = up[2 * g.N + c];
            } else if (code == SETTER_KEEP) {
                // no velocity field (float form): the velocity of the cell's
                // unchanged owner, recomputed as the collision does
                d0 = d1 = d2 = T(0);
                if constexpr (sizeof(T) == 4) {
                    const int slot = owner_slot(vox[c], ot.tag2slot, ot.max_tag, nsph);
                    if (slot >= 0) table_velocity(ot.xpf + (size_t)slot * XPF_STRIDE, X, Y, Z, g, d0, d1, d2);
                }
            } else {
                setter_velocity<T>(code, sph, fast, X, Y, Z, d0, d1, d2);
            }
            // f̄_i = feq_i(rhoBar = 0, invRho = 1, j = u), rounded operation by operation
            // (no contraction), so that every kernel variant writes the same bits
            const T uSqr = add_rn(add_rn(mul_rn(d0, d0), mul_rn(d1, d1)), mul_rn(d2, d2));
#pragma unroll
            for (int i = 0; i < Q; ++i) {
                const T cu = add_rn(add_rn(mul_rn(T(cx(i)), d0), mul_rn(T(cy(i)), d1)), mul_rn(T(cz(i)), d2));
                const T e = mul_rn(T(wt(i)), add_rn(mul_rn(T(3), cu),
                                                    sub_rn(mul_rn(mul_rn(T(4.5), cu), cu), mul_rn(T(1.5), uSqr))));
                *pop_slot(f, i, X, Y, Z, phase, g) = e;
            }
        }
    }
    // write back the changed cells
#pragma unroll 2
    for (int j = 0; j < 16; ++j) {
        const int l = lane + 32 * j;
        const uint32_t code = S.setter[l];
        if (code == SETTER_KEEP) continue;
        const int X = X0 + (j >> 1), Y = Y0 + (lane >> 3) + 4 * (j & 1);
        const size_t c = ((size_t)X * g.ny + Y) * g.nz + Z;
        vox[c] = S.w[l];
        if (up != nullptr) {
            T u0, u1, u2;
            setter_velocity<T>(code, sph, fast, X, Y, Z, u0, u1, u2);
            up[c] = u0; up[g.N + c] = u1; up[2 * g.N + c] = u2;
        }
    }
}

// Persistent voxelization: warps claim items of the work list one at a time
// (work_n[0] tiles listed, work_n[1] claim counter, work_n[2] finished blocks; the last
// block to finish zeroes all three for the next voxelization).
// An item is a tile, or, when the tiles are few for the grid's warps, an x-slab of one
// (cells are independent): a tile is a serial chain of up to 15 us per sphere shell for
// one warp, and a short list, or the last round of a longer one, waits for that chain.
// slab_bits() takes the number of slabs per tile that makes rounds x chain least, with
// the part of the chain that every slab repeats (tile setup, list, records) a 16th of a
// tile's: fitted to the cycle times of a 128^3 suspension, 4096 tiles on 3648 warps,
// 535, 502, 492 us with 1, 2, 4 slabs, and a 96^3 one, 1728 tiles, 65, 60, 67, 73 us
// with 1, 2, 4, 8.  SLABS false: whole tiles only, for lattices of more than
// VOX_SLAB_ROUNDS tiles per warp (their lists are long enough as a rule, and the slab
// bounds cost the kernel 4 % on a 256^3 suspension).
// A warp's first item is its own number, counted across the blocks first: a short list
// spreads over the SMs and starts without a claim.
// BATCH: a listed tile belongs to the domain d with toff[d] <= tile.
__device__ __forceinline__ int slab_bits(int nwork, int warps) {
    int best = 0, cost = INT_MAX;
#pragma unroll
    for (int lp = 0; lp <= 3; ++lp) {
        const int rounds = min(((nwork << lp) + warps - 1) / warps, 1 << 24);
        const int c = rounds * (1 + (16 >> lp));
        if (c < cost) {
            cost = c;
            best = lp;
        }
    }
    return nwork < (1 << 24) ? best : 0;   // (longer lists: no slabs, and no overflow above)
}

template <typename T, bool INIT_VEL, bool BATCH, bool SLABS>
__global__ void __launch_bounds__(VOX_THREADS, INIT_VEL ? 2 : 3)
k_voxelize(const SphereDev* __restrict__ sph, const SphereFast* __restrict__ fast, int nsph,
           int* __restrict__ tile_cnt, const int* __restrict__ bins, const int* __restrict__ work,
           int* __restrict__ work_n, uint32_t* __restrict__ vox, T* __restrict__ up, T* __restrict__ f, int phase,
           Geom g, const DomView* __restrict__ doms, const int* __restrict__ toff, int ndom,
           const int* __restrict__ ncur, OwnerTable ot) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    WarpVox<INIT_VEL>& S = reinterpret_cast<WarpVox<INIT_VEL>*>(smem_raw)[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    // batch: the CTA's copy of the domains' first tiles (ndom <= TOFF_SMEM), for the
    // per-tile domain search
    const int* stoff = nullptr;
    if constexpr (BATCH) {
        int* m = reinterpret_cast<int*>(smem_raw + sizeof(WarpVox<INIT_VEL>) * VOX_WARPS);
        if (ndom <= TOFF_SMEM) {
            for (int k = threadIdx.x; k < ndom; k += blockDim.x) m[k] = __ldg(toff + k);
            stoff = m;
        }
        __syncthreads();   // every thread of the CTA reaches it (before any leaves)
    }
    const int nwork = *(volatile int*)work_n;
    const int warps = (int)gridDim.x * VOX_WARPS;
    const int lp = SLABS ? slab_bits(nwork, warps) : 0;
    const int nitems = nwork << lp;
    int part = 0;
    // the next item is claimed and its tile read while the current one is worked on
    auto item = [&](int w) -> int {
        part = w & ((1 << lp) - 1);
        return w < nitems ? work[w >> lp] : -1;
    };
    int next = item((int)(blockIdx.x + gridDim.x * (threadIdx.x >> 5)));
    while (next >= 0) {
        const int tg = next;
        const int xa = part << (3 - lp), xb = xa + (TILE >> lp) - 1;
        int w = 0;
        if (lane == 0) w = atomicAdd(work_n + 1, 1) + warps;
        next = item(__shfl_sync(FULL_MASK, w, 0));
        if (BATCH) {
            int d;
            if (stoff) {
                int lo = 0, hi = ndom - 1;
                while (lo < hi) {
                    const int mid = (lo + hi + 1) >> 1;
                    if (stoff[mid] <= tg) lo = mid;
                    else hi = mid - 1;
                }
                d = lo;
            } else {
                d = find_domain(toff, ndom, tg);
            }
            const DomView& D = doms[d];
            const OwnerTable od{ot.xpf + (size_t)XPF_STRIDE * D.s0, ot.tag2slot + D.tag0, ot.max_tag};
            voxelize_tile<T, INIT_VEL>(S, tg - D.t0, sph + D.s0, fast + D.s0, __ldg(ncur + d), tile_cnt + D.t0,
                                       bins + (size_t)D.t0 * TILE_BIN, vox + D.cell0, up ? up + D.up0 : up,
                                       f ? f + D.f0 : f, phase, D.g, od, xa, xb, 1u << lp);
        } else {
            voxelize_tile<T, INIT_VEL>(S, tg, sph, fast, nsph, tile_cnt, bins, vox, up, f, phase, g, ot, xa, xb,
                                       1u << lp);
        }
        __syncwarp();
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(work_n + 2, 1) == (int)gridDim.x - 1) {
            work_n[0] = 0;
            work_n[1] = 0;
            work_n[2] = 0;
        }
    }
}

}  // namespace

namespace {

// Spheres per warp: one up to PREPARE_WIDE spheres (the launch is then a chain of
// latencies), four beyond it.  5, 498, 2902, 9535 spheres: 5.8, 7.3, 12.7, 25.4 us with
// one, 7.6, 10.2, 13.2, 17.1 us with four (6.6, 8.8, 16.5, 40.7 us with one lane
// preparing a sphere).
constexpr int PREPARE_WIDE = 4096;
template <bool BATCH>
cudaError_t launch_prepare_any(const double* rec, int n, const SphereTables& t, const Geom& g, int max_tag,
                               double max_radius, const DomView* doms, const int* soff, int ndom, const int* ncur,
                               int* tile_cnt, int* bins, int* work, int* work_n, const OldList& old, cudaStream_t s) {
    if (n <= PREPARE_WIDE)
        k_prepare_bin<BATCH, 32><<<(n + 3) / 4, 128, 0, s>>>(rec, n, t, g, max_tag, max_radius, doms, soff, ndom, ncur,
                                                             tile_cnt, bins, work, work_n, old);
    else
        k_prepare_bin<BATCH, 8><<<(n + 15) / 16, 128, 0, s>>>(rec, n, t, g, max_tag, max_radius, doms, soff, ndom,
                                                              ncur, tile_cnt, bins, work, work_n, old);
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_prepare_bin(const double* rec, int n, SphereDev* sph, SphereFast* fast, float* xpf,
                               int* tag2slot, unsigned* err, Geom g, int max_tag, double max_radius,
                               double* ft_zero, double* rec_copy, int* tile_cnt, int* bins, int* work, int* work_n,
                               int* old_map, const double* old_rec, int old_n, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    return launch_prepare_any<false>(rec, n, SphereTables{sph, fast, xpf, tag2slot, err, ft_zero, rec_copy}, g, max_tag,
                                     max_radius, nullptr, nullptr, 0, nullptr, tile_cnt, bins, work, work_n,
                                     OldList{old_map, old_rec, old_n, max_tag}, s);
}

cudaError_t launch_prepare(const double* rec, int n, SphereDev* sph, SphereFast* fast, float* xpf, int* tag2slot,
                           unsigned* err, Geom g, int max_tag, double max_radius, double* ft_zero, double* rec_copy,
                           cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    k_prepare<<<(n + 7) / 8, 64, 0, s>>>(rec, n, SphereTables{sph, fast, xpf, tag2slot, err, ft_zero, rec_copy}, g,
                                         max_tag, max_radius);
    return cudaGetLastError();
}

cudaError_t launch_prepare_bin_batch(const double* rec, int nslots, SphereDev* sph, SphereFast* fast, float* xpf,
                                     int* tag2slot, unsigned* err, int max_tag, double max_radius,
                                     const DomView* doms, const int* soff, int ndom, const int* ncur,
                                     double* ft_zero, int* tile_cnt, int* bins, int* work, int* work_n,
                                     cudaStream_t s) {
    if (nslots <= 0) return cudaSuccess;
    return launch_prepare_any<true>(rec, nslots, SphereTables{sph, fast, xpf, tag2slot, err, ft_zero, nullptr}, Geom{},
                                    max_tag, max_radius, doms, soff, ndom, ncur, tile_cnt, bins, work, work_n,
                                    OldList{nullptr, nullptr, 0, 0}, s);
}

namespace {

template <typename T, bool INIT_VEL, bool BATCH>
cudaError_t launch_vox(const SphereDev* sph, const SphereFast* fast, int n, int* tile_cnt, const int* bins,
                       const int* work, int* work_n, int ntiles, uint32_t* vox, T* up, T* f, int phase, Geom g,
                       const DomView* doms, const int* toff, int ndom, const int* ncur, const OwnerTable& ot,
                       cudaStream_t s) {
    constexpr size_t smem = sizeof(WarpVox<INIT_VEL>) * VOX_WARPS + (BATCH ? sizeof(int) * TOFF_SMEM : 0);
    static std::atomic<int> cached[LBDEM_MAX_DEVICES];   // per device: persistent grid size
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= LBDEM_MAX_DEVICES) return cudaErrorInvalidDevice;
    int blocks = cached[dev].load(std::memory_order_relaxed);
    if (blocks == 0) {
        int sms = 0, per_sm = 0, per_sm_slabs = 0;
        e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(k_voxelize<T, INIT_VEL, BATCH, false>,
                                     cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(k_voxelize<T, INIT_VEL, BATCH, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)smem);
        if (e == cudaSuccess)
            e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_voxelize<T, INIT_VEL, BATCH, false>,
                                                              VOX_THREADS, smem);
        if (e == cudaSuccess)
            e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm_slabs, k_voxelize<T, INIT_VEL, BATCH, true>,
                                                              VOX_THREADS, smem);
        if (e != cudaSuccess) return e;
        if (per_sm_slabs < per_sm) per_sm = per_sm_slabs;
        blocks = sms * (per_sm > 0 ? per_sm : 1);
        cached[dev].store(blocks, std::memory_order_relaxed);
    }
    const int grid = ntiles < blocks ? ntiles : blocks;   // up to TILE slabs per tile, one per warp
    if (ntiles <= VOX_SLAB_ROUNDS * blocks * VOX_WARPS)
        k_voxelize<T, INIT_VEL, BATCH, true><<<grid, VOX_THREADS, smem, s>>>(sph, fast, n, tile_cnt, bins, work, work_n,
                                                                             vox, up, f, phase, g, doms, toff, ndom,
                                                                             ncur, ot);
    else
        k_voxelize<T, INIT_VEL, BATCH, false><<<grid, VOX_THREADS, smem, s>>>(sph, fast, n, tile_cnt, bins, work,
                                                                              work_n, vox, up, f, phase, g, doms, toff,
                                                                              ndom, ncur, ot);
    return cudaGetLastError();
}

}  // namespace

template <typename T>
cudaError_t launch_voxelize(const SphereDev* sph, const SphereFast* fast, int n, int* tile_cnt, const int* bins,
                            const int* work, int* work_n, int ntiles, uint32_t* vox, T* up, T* f, int init_vel,
                            int odd_phase, Geom g, const OwnerTable& ot, cudaStream_t s) {
    if (ntiles <= 0) return cudaSuccess;
    if (init_vel)
        return launch_vox<T, true, false>(sph, fast, n, tile_cnt, bins, work, work_n, ntiles, vox, up, f, odd_phase, g,
                                          nullptr, nullptr, 0, nullptr, ot, s);
    return launch_vox<T, false, false>(sph, fast, n, tile_cnt, bins, work, work_n, ntiles, vox, up, f, odd_phase, g,
                                       nullptr, nullptr, 0, nullptr, ot, s);
}

template <typename T>
cudaError_t launch_voxelize_batch(const SphereDev* sph, const SphereFast* fast, int* tile_cnt, const int* bins,
                                  const int* work, int* work_n, int ntiles, uint32_t* vox, T* up, T* f, int init_vel,
                                  int odd_phase, const DomView* doms, const int* toff, int ndom, const int* ncur,
                                  const OwnerTable& ot, cudaStream_t s) {
    if (ntiles <= 0) return cudaSuccess;
    if (init_vel)
        return launch_vox<T, true, true>(sph, fast, 0, tile_cnt, bins, work, work_n, ntiles, vox, up, f, odd_phase,
                                         Geom{}, doms, toff, ndom, ncur, ot, s);
    return launch_vox<T, false, true>(sph, fast, 0, tile_cnt, bins, work, work_n, ntiles, vox, up, f, odd_phase,
                                      Geom{}, doms, toff, ndom, ncur, ot, s);
}

#define INST(T)                                                                                                    \
    template cudaError_t launch_voxelize<T>(const SphereDev*, const SphereFast*, int, int*, const int*, const int*, \
                                            int*, int, uint32_t*, T*, T*, int, int, Geom, const OwnerTable&,       \
                                            cudaStream_t);                                                         \
    template cudaError_t launch_voxelize_batch<T>(const SphereDev*, const SphereFast*, int*, const int*,          \
                                                  const int*, int*, int, uint32_t*, T*, T*, int, int,              \
                                                  const DomView*, const int*, int, const int*, const OwnerTable&,  \
                                                  cudaStream_t);
INST(float)
INST(double)
#undef INST

}  // namespace lbdem
