// relaxdf.cu — the double-float relaxation (precision MAFM_DF).
//
// Every quantity of the relaxation is a dfloat (dfloat.cuh): the tip–atom
// terms, their sums, the tip–dummy terms, positions, velocities, the FIRE
// time step and mixing factor, energies.  The minimiser's and integrators'
// operations are those of the FP64 kernel (fire_t / sd_t, relax_tpl.cuh),
// stage by stage, so the relaxation takes the same steps as FP64 unless one
// of FIRE's discrete decisions — the convergence test, the sign of P = v.F —
// falls within the double-float error (about 1e-13 of the largest term) of
// its threshold.  Such near-ties are recognised with a margin far above that
// error (TieMargins): the column is given up at its first one, goes on the
// list of the FP64 re-relaxation, and is relaxed again from its top height by
// one warp in FP64 with the plain FP64 kernel's bits (its points from that
// height on carry MAFM_PT_NEAR_TIE, all of them MAFM_PT_FP64) — inside this
// kernel by warps that have run out of columns, the rest by repair64_kernel
// after it.
//
// Why not FP32 with a near-tie repair: with FP32 pair terms (about 1e-6 of a
// term) FIRE's decisions come within FP32 error of their thresholds in
// nearly every pixel column of a scan, and the FP32 trajectory itself drifts
// from FP64's by about 1e-7 A, so no decision margin separates the columns
// that follow FP64 from those that do not.
//
// Every lane relaxes one pixel column at a time (columns from a global
// queue, in each scan's expected-cost order) in a slot machine: one force
// evaluation per lane per iteration, then the lane's own minimiser stage, so
// a warp's lanes stay busy whatever their columns' step counts (one thread
// running a whole column kept only 13 of 32 lanes active on average).  The
// terms are read through the read-only cache, every lane of a warp reading
// the same record (broadcast).
//
// Reference correspondence (src/): LJ / Morse / Coulomb interactions.cpp:15-51,
// tip–dummy terms interactions.cpp:252-266 and simulation.cpp:503-515,
// external field lookup force_grid.cpp:88-275, minimiser and column as in
// relax_tpl.cuh.
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <type_traits>

#define MAFM_PLAIN_DIV64   // see relax64_dev.cuh
#include "mafm_df.h"
#include "relax64_dev.cuh"
#include "relax_tpl.cuh"

namespace mafm {
namespace {

using D = dfloat;
using V3D = V3T<dfloat>;

// One term at the distance squared r2: LJ (interactions.cpp:15-27) or Morse
// (:29-40), plus Coulomb (:42-51) when coul.  1/r comes from a double-float rsqrt;
// the force on the first particle is s times the separation.
__device__ __forceinline__ void pair_df(int kind, D p0, D p1, D p2, bool coul, D qq, D r2, D& s, D& e) {
    const D ir = dfl_rsqrt(r2);
    const D ir2 = ir * ir;
    if (kind == MAFM_PAIR_LJ) {
        const D ir6 = ir2 * ir2 * ir2;
        const D a = p1 * (ir6 * ir6);   // es12 / r^12
        const D b = p0 * ir6;           // es6 / r^6
        e = a - b;
        s = (a * 12.0f - b * 6.0f) * ir2;
    } else {
        const D r = r2 * ir;
        const D q = dfl_exp(-(p1 * (r - p2)));
        const D q2 = q * q;
        e = p0 * ((q2 - q * 2.0f) + D(1.0f, 0.0f));
        s = ((p0 * p1) * 2.0f) * (q2 - q) * ir;
    }
    if (coul) {
        const D ec = qq * ir;
        e = e + ec;
        s = s + ec * ir2;
    }
}

using D2 = dfloat2;

// Sum of many double-floats, two at a time: the high parts through two_sum,
// every rounding error and low part into one FP32 word per element (a few
// ulps of the high part after hundreds of terms, far below the double-float
// error of a term).
struct LazySum2 {
    float2 h = {0.0f, 0.0f}, l = {0.0f, 0.0f};
    __device__ __forceinline__ void add(D2 x) {
        const D2 s = dfl2_two_sum(h, x.h);
        h = s.h;
        l = p_add(l, p_add(s.l, x.l));
    }
    // both elements' sums, added
    __device__ __forceinline__ D value() const {
        const D a = dfl_two_sum(h.x, l.x), b = dfl_two_sum(h.y, l.y);
        return a + b;
    }
};

__device__ __forceinline__ float2 f2(float4 v, int hi) {
    return hi ? make_float2(v.z, v.w) : make_float2(v.x, v.y);
}

// x^2: the square of the high part exactly (product and FMA residue), the
// cross term 2 h l into the low part (l^2 is below 2^-46 of the square).
__device__ __forceinline__ D2 sq_u(D2 x) {
    const float2 p = p_mul(x.h, x.h);
    return {p, p_fma(p_add(x.h, x.h), x.l, p_fma(x.h, x.h, p_neg(p)))};
}

// 1 / sqrt(a) as dfl2_rsqrt, for an operand that need not be normalised
__device__ __forceinline__ D2 rsqrt_u(D2 a) {
    const float2 y = make_float2(dfl_rsqrt_approx(a.h.x), dfl_rsqrt_approx(a.h.y));
    const D2 t = dfl2_mulf_u(dfl2_mulf_u(a, y), y);
    const float2 e = p_sub(p_sub(p_bcast(1.0f), t.h), t.l);
    return dfl2_fast_two_sum(y, p_mul(p_mul(y, e), p_bcast(0.5f)));
}

// The two terms of a TermPairDF record (element .x the first, .y the second).
struct PairDF2 {
    D2 x, y, z, qq, p0, p1, p2;
    int coul;
};

template <int KIND>
__device__ __forceinline__ PairDF2 load_pair(const TermPairDF* rec) {
    const float4* q = reinterpret_cast<const float4*>(rec);
    const float4 a = __ldg(q), b = __ldg(q + 1), c = __ldg(q + 2), g = __ldg(q + 3);
    const float4 h = __ldg(q + 4), m = __ldg(q + 5);
    PairDF2 t;
    t.x = {f2(a, 0), f2(a, 1)};
    t.y = {f2(b, 0), f2(b, 1)};
    t.z = {f2(c, 0), f2(c, 1)};
    t.qq = {f2(g, 0), f2(g, 1)};
    t.p0 = {f2(h, 0), f2(h, 1)};
    t.p1 = {f2(m, 0), f2(m, 1)};
    if (KIND == MAFM_PAIR_MORSE) {
        const float4 n = __ldg(q + 6);
        t.p2 = {f2(n, 0), f2(n, 1)};
    } else {
        t.p2 = {p_bcast(0.0f), p_bcast(0.0f)};
    }
    t.coul = __float_as_int(__ldg(reinterpret_cast<const float*>(q + 7)));
    return t;
}

// LJ (interactions.cpp:15-27) or Morse (:29-40), plus Coulomb (:42-51) when
// the record has one, for the separation d = tip - atom with r2 = |d|^2; the
// force on the tip and the energy go into the lazy sums.  1/r comes from a
// double-float rsqrt.
template <int KIND>
__device__ __forceinline__ void pair_df2_at(const PairDF2& t, D2 dx, D2 dy, D2 dz, D2 r2, LazySum2& fx,
                                            LazySum2& fy, LazySum2& fz, LazySum2& ee) {
    const D2 ir = rsqrt_u(r2);
    const D2 ir2 = dfl2_mul_u(ir, ir);
    D2 e, s;
    if (KIND == MAFM_PAIR_LJ) {
        // A = es12 / r^6, u = A - es6: E = u / r^6 = es12 / r^12 - es6 / r^6 and
        // (12 es12 / r^12 - 6 es6 / r^6) / r^2 = 6 (A + u) / r^6 / r^2; the
        // Coulomb term's qq / r^3 = (qq / r) / r^2 joins before the last / r^2
        const D2 ir6 = dfl2_norm(dfl2_mul_u(dfl2_mul_u(ir2, ir2), ir2));
        const D2 A = dfl2_mul_u(t.p1, ir6);
        const D2 u = dfl2_sub_u(A, t.p0);
        e = dfl2_mul_u(ir6, u);
        D2 sr = dfl2_mulf_u(dfl2_mul_u(dfl2_add_u(A, u), ir6), p_bcast(6.0f));
        if (t.coul) {
            const D2 ec = dfl2_mul_u(t.qq, ir);
            e = dfl2_add_u(e, ec);
            sr = dfl2_add_u(sr, ec);
        }
        s = dfl2_mul_u(sr, ir2);
    } else {
        const D2 r = dfl2_mul_u(r2, ir);
        const D2 qe = dfl2_exp(-dfl2_mul_u(t.p1, dfl2_sub_u(r, t.p2)));
        const D2 qe2 = dfl2_mul_u(qe, qe);
        // De (q^2 - 2 q + 1), 2 De a (q^2 - q) / r
        e = dfl2_mul_u(t.p0, dfl2_add_u(dfl2_sub_u(qe2, dfl2_mulf_u(qe, p_bcast(2.0f))),
                                        D2{p_bcast(1.0f), p_bcast(0.0f)}));
        s = dfl2_mul_u(dfl2_mul_u(dfl2_mulf_u(dfl2_mul_u(t.p0, t.p1), p_bcast(2.0f)),
                                  dfl2_sub_u(qe2, qe)), ir);
    }
    if (KIND == MAFM_PAIR_MORSE && t.coul) {
        const D2 ec = dfl2_mul_u(t.qq, ir);
        e = dfl2_add_u(e, ec);
        s = dfl2_add_u(s, dfl2_mul_u(ec, ir2));
    }
    fx.add(dfl2_mul_u(s, dx));
    fy.add(dfl2_mul_u(s, dy));
    fz.add(dfl2_mul_u(s, dz));
    ee.add(e);
}

// The two terms of a record at the tip (tx, ty, tz).
template <int KIND>
__device__ __forceinline__ void pair_df2(const TermPairDF* rec, D2 tx, D2 ty, D2 tz, LazySum2& fx,
                                         LazySum2& fy, LazySum2& fz, LazySum2& ee) {
    const PairDF2 t = load_pair<KIND>(rec);
    const D2 dx = dfl2_sub_u(tx, t.x), dy = dfl2_sub_u(ty, t.y), dz = dfl2_sub_u(tz, t.z);
    const D2 r2 = dfl2_add_u(dfl2_add_u(sq_u(dx), sq_u(dy)), sq_u(dz));
    pair_df2_at<KIND>(t, dx, dy, dz, r2, fx, fy, fz, ee);
}

// ForceGrid::interpolate (force_grid.cpp:88-155) on the double-float copy of
// a periodic grid (the external field).
__device__ void interp_df(const GridViewDF& g, V3D pos, V3D& f, D& e) {
    const V3D q = {pos.x - g.origin[0], pos.y - g.origin[1], pos.z - g.origin[2]};
    V3D pb;
    if (g.orthogonal) {
        pb.x = q.x / g.basis[0];
        pb.y = q.y / g.basis[4];
        pb.z = q.z / g.basis[8];
    } else {
        pb.x = g.inv[0] * q.x + g.inv[1] * q.y + g.inv[2] * q.z;
        pb.y = g.inv[3] * q.x + g.inv[4] * q.y + g.inv[5] * q.z;
        pb.z = g.inv[6] * q.x + g.inv[7] * q.y + g.inv[8] * q.z;
    }
    const D fl[3] = {dfl_floor(pb.x), dfl_floor(pb.y), dfl_floor(pb.z)};
    int gp[3];
    for (int a = 0; a < 3; ++a) gp[a] = (int)fl[a].h + (int)fl[a].l;
    int lo[3], hi[3];
    for (int a = 0; a < 3; ++a) {
        int x0 = gp[a] % g.n[a];
        if (x0 < 0) x0 += g.n[a];
        lo[a] = x0;
        hi[a] = x0 + 1 == g.n[a] ? 0 : x0 + 1;
    }
    const D dx = pb.x - fl[0], dy = pb.y - fl[1], dz = pb.z - fl[2];
    const D one(1.0f, 0.0f);
    const long long n12 = (long long)g.n[1] * g.n[2];
    NodeDF s[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) {
        const int x = (c >> 2) ? hi[0] : lo[0];
        const int y = ((c >> 1) & 1) ? hi[1] : lo[1];
        const int z = (c & 1) ? hi[2] : lo[2];
        const float4* p = reinterpret_cast<const float4*>(g.g + (long long)x * n12 +
                                                          (long long)y * g.n[2] + z);
        const float4 u = __ldg(p), v = __ldg(p + 1);
        s[c].x = D(u.x, u.y); s[c].y = D(u.z, u.w); s[c].z = D(v.x, v.y); s[c].w = D(v.z, v.w);
    }
    D out[4];
#pragma unroll
    for (int m = 0; m < 4; ++m) {
        auto comp = [m](const NodeDF& n) { return m == 0 ? n.x : m == 1 ? n.y : m == 2 ? n.z : n.w; };
        const D v00 = comp(s[0]) * (one - dx) + comp(s[4]) * dx;
        const D v01 = comp(s[1]) * (one - dx) + comp(s[5]) * dx;
        const D v10 = comp(s[2]) * (one - dx) + comp(s[6]) * dx;
        const D v11 = comp(s[3]) * (one - dx) + comp(s[7]) * dx;
        const D v0 = v00 * (one - dy) + v10 * dy;
        const D v1 = v01 * (one - dy) + v11 * dy;
        out[m] = v0 * (one - dz) + v1 * dz;
    }
    f = {out[0], out[1], out[2]};
    e = out[3];
}

// The sum of v over a group of G lanes (G a power of two, the group aligned
// in the warp), added in the same order on every lane of the group, so all
// of them hold the same bits.
template <int G>
__device__ __forceinline__ D group_sum(D v, int sub, unsigned gmask) {
#pragma unroll
    for (int m = 1; m < G; m <<= 1) {
        const D o(__shfl_xor_sync(gmask, v.h, m), __shfl_xor_sync(gmask, v.l, m));
        v = (sub & m) ? o + v : v + o;
    }
    return v;
}

// ForceGrid::interpolate (force_grid.cpp:88-275) on the double-float rigid
// grid, with interp64's handling of its border: a base node outside the grid
// is clamped and marks the point MAFM_PT_OUTSIDE (the reference's warning), a
// corner outside sets ERR_GRID_INDEX (the reference stops) and is clamped so
// that no read leaves the grid.
__device__ void interp_df_grid(const GridViewDF& g, V3D pos, V3D& f, D& e, int& outside,
                               unsigned& err) {
    const V3D q = {pos.x - g.origin[0], pos.y - g.origin[1], pos.z - g.origin[2]};
    const V3D pb = {q.x / g.basis[0], q.y / g.basis[4], q.z / g.basis[8]};
    const D fl[3] = {dfl_floor(pb.x), dfl_floor(pb.y), dfl_floor(pb.z)};
    int gp[3];
    for (int a = 0; a < 3; ++a) {
        gp[a] = (int)fl[a].h + (int)fl[a].l;
        if (gp[a] < 0) { gp[a] = 0; outside = 1; }
        else if (gp[a] >= g.n[a]) { gp[a] = g.n[a] - 1; outside = 1; }
    }
    int lo[3], hi[3];
    for (int a = 0; a < 3; ++a) {
        lo[a] = gp[a];
        hi[a] = gp[a] + 1;
        if (hi[a] >= g.n[a]) {
            err |= ERR_GRID_INDEX;
            hi[a] = g.n[a] - 1;
        }
    }
    const D dx = pb.x - D(gp[0]), dy = pb.y - D(gp[1]), dz = pb.z - D(gp[2]);
    const D one(1.0f, 0.0f);
    const long long n12 = (long long)g.n[1] * g.n[2];
    NodeDF s[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) {
        const int x = (c >> 2) ? hi[0] : lo[0];
        const int y = ((c >> 1) & 1) ? hi[1] : lo[1];
        const int z = (c & 1) ? hi[2] : lo[2];
        const float4* p = reinterpret_cast<const float4*>(g.g + (long long)x * n12 +
                                                          (long long)y * g.n[2] + z);
        const float4 u = __ldg(p), v = __ldg(p + 1);
        s[c].x = D(u.x, u.y); s[c].y = D(u.z, u.w); s[c].z = D(v.x, v.y); s[c].w = D(v.z, v.w);
    }
    D out[4];
#pragma unroll
    for (int m = 0; m < 4; ++m) {
        auto comp = [m](const NodeDF& n) { return m == 0 ? n.x : m == 1 ? n.y : m == 2 ? n.z : n.w; };
        const D v00 = comp(s[0]) * (one - dx) + comp(s[4]) * dx;
        const D v01 = comp(s[1]) * (one - dx) + comp(s[5]) * dx;
        const D v10 = comp(s[2]) * (one - dx) + comp(s[6]) * dx;
        const D v11 = comp(s[3]) * (one - dx) + comp(s[7]) * dx;
        const D v0 = v00 * (one - dy) + v10 * dy;
        const D v1 = v01 * (one - dy) + v11 * dy;
        out[m] = v0 * (one - dz) + v1 * dz;
    }
    f = {out[0], out[1], out[2]};
    e = out[3];
}

// Vectors of a column's state.  With G >= 4 lanes per column lane c of every quad
// holds component c (x, y, z; lane 3 goes along with z, and holds E where forces
// are summed), so that the vector arithmetic of the minimiser, which every lane of
// the group would otherwise repeat, costs a third; with fewer lanes every lane
// holds all three.  The operations of a component are the same: the same bits.
// 40 x 40 x 21 graphene (G = 8) 11.8 -> 10.8 ms; at G = 4 the runs differ by as much.
struct QuadDF {
    D c;
};
template <int G>
using VecDF = std::conditional_t<(G >= 4), QuadDF, V3D>;

// Component m of a quad, on all of its lanes.
__device__ __forceinline__ D quad_get(D v, int m, unsigned gmask) {
    const int src = ((int)threadIdx.x & 28) | m;
    return D(__shfl_sync(gmask, v.h, src), __shfl_sync(gmask, v.l, src));
}
template <int G>
__device__ __forceinline__ V3D whole(VecDF<G> v, unsigned gmask) {
    if constexpr (G >= 4) return {quad_get(v.c, 0, gmask), quad_get(v.c, 1, gmask), quad_get(v.c, 2, gmask)};
    else return v;
}
template <int G>
__device__ __forceinline__ VecDF<G> own(V3D v) {
    if constexpr (G >= 4) {
        const int c = threadIdx.x & 3;
        return {c == 0 ? v.x : c == 1 ? v.y : v.z};
    } else {
        return v;
    }
}
// f of the components of a, b
template <class F>
__device__ __forceinline__ QuadDF vmap(QuadDF a, QuadDF b, F f) { return {f(a.c, b.c)}; }
template <class F>
__device__ __forceinline__ V3D vmap(V3D a, V3D b, F f) { return {f(a.x, b.x), f(a.y, b.y), f(a.z, b.z)}; }
// a . b, the products added in the order x, y, z
template <int G>
__device__ __forceinline__ D vdot(VecDF<G> a, VecDF<G> b, unsigned gmask) {
    if constexpr (G >= 4) {
        const D s = a.c * b.c;
        return quad_get(s, 0, gmask) + quad_get(s, 1, gmask) + quad_get(s, 2, gmask);
    } else {
        return a.x * b.x + a.y * b.y + a.z * b.z;
    }
}

// The sums over the G >= 4 lanes of a group of fx, fy, fz and e, one on each lane
// of a quad, each added as group_sum adds it.
template <int G>
__device__ __forceinline__ D quad_sum(D fx, D fy, D fz, D e, int sub, unsigned gmask) {
    auto other = [&](D v, int m) {
        return D(__shfl_xor_sync(gmask, v.h, m), __shfl_xor_sync(gmask, v.l, m));
    };
    const bool odd = sub & 1, up = sub & 2;
    const D a = (odd ? fy : fx) + other(odd ? fx : fy, 1);
    const D b = (odd ? e : fz) + other(odd ? fz : e, 1);
    D v = (up ? b : a) + other(up ? a : b, 2);
#pragma unroll
    for (int m = 4; m < G; m <<= 1) v = v + other(v, m);
    return v;
}

// System::evalTipSurfaceForces (system.cpp:41-51): the tip–surface force and
// energy at tip, by the G lanes of a group (lane sub of the group takes the
// term pairs sub, sub + G, ...; the external field on lane 0).  The loop over
// terms is the same for every group of a scan.
template <int G>
__device__ __forceinline__ void ts_df(const ScanParamsDF& p, VecDF<G> at, int sub, unsigned gmask,
                                      VecDF<G>& F, D& E, int& outside, unsigned& err) {
    const V3D tip = whole<G>(at, gmask);
    if (p.ts_mode == 2) {
        // the rigid grid alone; every lane of the group looks it up
        V3D f;
        interp_df_grid(p.grid, tip, f, E, outside, err);
        F = own<G>(f);
        return;
    }
    LazySum2 fx, fy, fz, ee;
    const D2 tx = dfl2(tip.x), ty = dfl2(tip.y), tz = dfl2(tip.z);
    const int n_lj = p.n_lj_pairs, n_all = p.n_lj_pairs + p.n_morse_pairs;
    for (int i = sub; i < n_lj; i += G)
        pair_df2<MAFM_PAIR_LJ>(p.pairs + i, tx, ty, tz, fx, fy, fz, ee);
    for (int i = n_lj + sub; i < n_all; i += G)
        pair_df2<MAFM_PAIR_MORSE>(p.pairs + i, tx, ty, tz, fx, fy, fz, ee);
    if (p.ts_mode == 1 && sub == 0) {
        V3D f;
        D e;
        interp_df(p.es, tip, f, e);
        fx.add(D2{make_float2(f.x.h, 0.0f), make_float2(f.x.l, 0.0f)});
        fy.add(D2{make_float2(f.y.h, 0.0f), make_float2(f.y.l, 0.0f)});
        fz.add(D2{make_float2(f.z.h, 0.0f), make_float2(f.z.l, 0.0f)});
        ee.add(D2{make_float2(e.h, 0.0f), make_float2(e.l, 0.0f)});
    }
    if constexpr (G >= 4) {
        const D v = quad_sum<G>(fx.value(), fy.value(), fz.value(), ee.value(), sub, gmask);
        F = {v};
        E = quad_get(v, 3, gmask);
    } else {
        F = {group_sum<G>(fx.value(), sub, gmask), group_sum<G>(fy.value(), sub, gmask),
             group_sum<G>(fz.value(), sub, gmask)};
        E = group_sum<G>(ee.value(), sub, gmask);
    }
}

// The tip–dummy terms and the XY spring, added in Eval64::all's order
// (simulation.cpp:503-515, interactions.cpp:252-266).
template <int G>
__device__ __forceinline__ void tip_dummy_df(const ScanParamsDF& p, VecDF<G> tip, VecDF<G> dum, unsigned gmask,
                                             VecDF<G>& F, D& E) {
    const VecDF<G> r = vmap(dum, tip, [](D d, D x) { return d - x; });
    D xx, yy, r2;
    if constexpr (G >= 4) {
        const D q = r.c * r.c;
        xx = quad_get(q, 0, gmask);
        yy = quad_get(q, 1, gmask);
        r2 = xx + yy + quad_get(q, 2, gmask);
    } else {
        xx = r.x * r.x;
        yy = r.y * r.y;
        r2 = xx + yy + r.z * r.z;
    }
    D s, e;
    pair_df(p.td_kind, p.td_p[0], p.td_p[1], p.td_p[2], p.td_coul != 0, p.td_qq, r2, s, e);
    F = vmap(F, r, [&](D f, D x) { return f - s * x; });
    E = E + e;
    const D rr = dfl_sqrt(xx + yy);
    const D dr = rr - p.harm_r0;
    E = E + p.harm_k * dr * dr;
    if (rr > D(1e-10)) {
        const D h = -(p.harm_k * 2.0f) * dr / rr;
        if constexpr (G >= 4) {
            const D f = F.c - h * r.c;
            if ((threadIdx.x & 3) < 2) F.c = f;
        } else {
            F.x = F.x - h * r.x;
            F.y = F.y - h * r.y;
        }
    }
}

enum : int { DF_EVAL0 = 0, DF_EVAL1 = 1, DF_EVAL2 = 2, DF_EVAL3 = 3, DF_OUT = 4 };

// Steps of a height up to which its lane does not wait for the warp's stage.  300 x
// 300 cluster x 15 heights that converge in energy after a few steps: rk4 4.33 ms,
// with waiting 5.21, midpoint 2.46 / 2.68; force and energy, hundreds of steps: the
// same either way (rk4 126 ms, never waiting 131-137; 101 x 101 graphene 103, never
// waiting 113-115).  4 and 16 measure the same as 8.
constexpr int kAlignSteps = 8;

// One lane's column: the state fire_t / sd_t keep in locals, held across
// slots.  u is the midpoint v2 / the RK4 v_k; vs, fs, es the RK4 sums.
template <int G>
struct LaneDF {
    int col, scan, k, n, nnn, phase, tie, outside;
    bool aligned;   // waits for the warp's stage
    VecDF<G> tip, vel, dum, ex, u, vs, fs;
    D energy, es, alpha, dt;
};

// An unwritten entry of the near-tie list (the host fills the list with it
// before each launch); real entries are scan << 32 | column.
constexpr unsigned long long kNoEntry = ~0ull;

// Claim the next near-tie list slot that a producer has already reserved
// (never past the count pushed so far, nor past the list); kNoEntry when
// there is none now.  Each failed compare-and-swap means another warp took a
// slot, so the loop ends; its bound is a safeguard.
__device__ unsigned long long claim_repair(RunCounters* ctr, unsigned cap) {
    unsigned long long cur = *reinterpret_cast<volatile unsigned long long*>(&ctr->repair_next);
    for (int i = 0; i < (1 << 20); ++i) {
        const unsigned n = min(*reinterpret_cast<volatile unsigned*>(&ctr->n_tie), cap);
        if (cur >= n) return kNoEntry;
        const unsigned long long prev = atomicCAS(&ctr->repair_next, cur, cur + 1);
        if (prev == cur) return cur;
        cur = prev;
    }
    return kNoEntry;
}

// The entry of a claimed slot: its producer reserved the slot and writes it
// right after, so the wait is short; it is bounded all the same (about half
// a second), after which ERR_REPAIR_WAIT is set and kNoEntry returned.
__device__ unsigned long long wait_entry(const unsigned long long* slot, unsigned& err) {
    for (int i = 0; i < (1 << 22); ++i) {
        const unsigned long long v = *reinterpret_cast<const volatile unsigned long long*>(slot);
        if (v != kNoEntry) return v;
        __nanosleep(100);
    }
    err |= ERR_REPAIR_WAIT;
    return kNoEntry;
}

__device__ __forceinline__ unsigned long long df_global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// The double-float relaxation as a slot machine: every group of G lanes of a
// warp holds one pixel column, and each loop iteration performs one force
// evaluation for every group that has one (the costly, uniform part; the
// group's lanes split the terms), then advances each group's minimiser by
// that evaluation: the integrator's stages (euler 1, midpoint 2, rk4 4
// evaluations per step), the convergence test and FIRE's mixing and time-step
// control, exactly in the order of fire_t / sd_t (relax_tpl.cuh), and the
// output evaluation of each height.  Every lane of a group holds the same
// state (the group sums are formed in one order on all of them) and runs the
// same minimiser code; lane 0 of the group writes.  A group whose column is
// done takes the next one from the global queue, so groups never wait for
// the slowest column of their warp.  G > 1 shortens each column's
// evaluations, which pays when a scan's longest columns, not the total work,
// set the launch's duration.
//
// Near-ties: at its first near-tie decision a column is given up.  Its
// unwritten heights get placeholder records (no steps, MAFM_PT_NEAR_TIE),
// and after a fence the column goes on repair_list.  A warp whose groups
// find the queue empty then re-relaxes listed columns in FP64, one warp per
// column (EvalWarp64 and relax_column_t<double>, the bits of repair64_kernel
// and relax64_kernel), while other warps still relax their last columns;
// repair64_kernel, launched after this kernel, takes the entries left.
template <int G>
__global__ void __launch_bounds__(128) relaxdf_kernel(const BatchDF* __restrict__ scans,
                                                      const BatchScan* __restrict__ scans64,
                                                      int n_scans, long long n_cols,
                                                      RunCounters* ctr,
                                                      unsigned long long* __restrict__ repair_list,
                                                      unsigned repair_cap,
                                                      unsigned long long watchdog_ns) {
    extern __shared__ __align__(32) unsigned char df_smem[];
    constexpr unsigned kFull = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int sub = lane & (G - 1);
    const int leader = lane & ~(G - 1);
    const unsigned gmask = G == 32 ? kFull : ((1u << G) - 1u) << leader;
    unsigned long long steps = 0, evals = 0, pairs = 0;
    unsigned status_or = 0, err = 0;
    const unsigned long long t0 = df_global_ns();
    unsigned ticks = 0;

    LaneDF<G> s;
    s.col = -1;
    s.scan = 0;
    s.tie = 0;
    bool done = false;
    const BatchDF* B = scans;

    // the column's first near-tie: placeholders for its unwritten heights, a
    // fence (the re-relaxation's records must land after these), then the
    // list; the group drops the column
    auto give_up = [&]() {
        const ScanParamsDF& P = B->p;
        if (sub == 0) {
            mafm_point* o = B->out + (size_t)(s.col - B->col_begin) * P.nz;
            mafm_point r{};
            r.status = MAFM_PT_NEAR_TIE;
            for (int kk = s.k; kk < P.nz; ++kk) o[kk] = r;
            __threadfence();
            const unsigned slot = atomicAdd(&ctr->n_tie, 1u);
            if (slot < repair_cap)
                repair_list[slot] = ((unsigned long long)s.scan << 32) | (unsigned)s.col;
        }
        s.col = -1;
    };

    auto start_level = [&]() {
        s.outside = 0;
        s.alpha = D(0.1);
        s.dt = B->p.dt;
        s.nnn = 0;
        s.n = 1;
        s.phase = s.n >= B->p.maxsteps ? DF_OUT : DF_EVAL0;
        s.ex = s.tip;
    };

    for (;;) {
        // groups without a column take the next queue entries (one atomic per
        // warp; a group is counted by its first lane)
        const unsigned idle = __ballot_sync(kFull, sub == 0 && s.col < 0 && !done);
        if (idle) {
            unsigned long long base = 0;
            if (lane == 0) base = atomicAdd(&ctr->next_work, (unsigned long long)__popc(idle));
            base = __shfl_sync(kFull, base, 0);
            if (s.col < 0 && !done) {
                const long long g = (long long)base + __popc(idle & ((1u << leader) - 1u));
                if (g >= n_cols) {
                    done = true;
                } else {
                    int lo = 0, hi = n_scans - 1;
                    while (lo < hi) {
                        const int mid = (lo + hi + 1) >> 1;
                        if (scans[mid].col_first <= g) lo = mid;
                        else hi = mid - 1;
                    }
                    s.scan = lo;
                    B = scans + lo;
                    const long long a = g - B->col_first;
                    s.col = B->order ? __ldg(B->order + a) : B->col_begin + (int)a;
                    // a new column (Simulation::run, simulation.cpp:93-99)
                    const ScanParamsDF& P = B->p;
                    const bool wrap = P.tip_pbc && P.ts_mode != 2;
                    const int i = s.col / P.ny, j = s.col % P.ny;
                    D x, y;
                    dummy_xy_t(P, wrap, D(i) * P.dx, D(j) * P.dy, x, y);
                    s.dum = own<G>(V3D{x, y, P.zhigh});
                    s.tip = own<G>(V3D{x, y, P.zhigh - P.tip_dummy_d});
                    s.vel = own<G>(V3D{D(0), D(0), D(0)});
                    s.energy = D(0);
                    s.k = 0;
                    s.tie = 0;
                    s.aligned = true;
                    start_level();
                }
            }
        }
        if (__all_sync(kFull, done)) break;
        if ((++ticks & 255u) == 0 && __any_sync(kFull, df_global_ns() - t0 > watchdog_ns)) {
            err |= ERR_WATCHDOG;
            break;
        }
        if (s.col < 0) continue;
        const ScanParamsDF& P = B->p;
        // A step starts, and a height's record is made, only in every second
        // iteration (midpoint; rk4: every fourth), so that the lanes of a warp
        // are in the same stage: without it they drift apart by one evaluation
        // at every record, and the warp runs every stage's code in every
        // iteration.  A lane waits for at most one (three) evaluations of a
        // height, so heights of few steps are not worth it: a lane whose last
        // height took kAlignSteps or fewer does not wait.
        if (s.aligned && (s.phase == DF_EVAL0 || s.phase == DF_OUT) && (ticks & P.stage_mask)) continue;

        // ---- one evaluation per lane ----
        VecDF<G> F;
        D E;
        ts_df<G>(P, s.ex, sub, gmask, F, E, s.outside, err);
        if (sub == 0) {
            evals += 1;
            pairs += (unsigned long long)B->n_pairs_per_eval;
        }
        if (s.phase == DF_OUT) {
            // System::getOutput (system.cpp:28-51)
            int st = (s.n >= P.maxsteps ? MAFM_PT_MAXSTEPS : 0) | (s.tie ? MAFM_PT_NEAR_TIE : 0) |
                     (s.outside ? MAFM_PT_OUTSIDE : 0);
            const V3D f = whole<G>(F, gmask), tip = whole<G>(s.tip, gmask);
            if (!dfl_isfinite(f.x) || !dfl_isfinite(f.y) || !dfl_isfinite(f.z) || !dfl_isfinite(E))
                st |= MAFM_PT_NONFINITE;
            mafm_point r;
            r.tip[0] = to_double(tip.x); r.tip[1] = to_double(tip.y); r.tip[2] = to_double(tip.z);
            r.force[0] = to_double(f.x); r.force[1] = to_double(f.y); r.force[2] = to_double(f.z);
            r.energy = to_double(E);
            r.steps = s.n;
            r.status = st;
            if (sub == 0) {
                B->out[(size_t)(s.col - B->col_begin) * P.nz + s.k] = r;
                steps += (unsigned long long)s.n;
                status_or |= (unsigned)st;
            }
            // System::lowerTip (system.hpp:51-54)
            if constexpr (G >= 4) {
                if ((lane & 3) >= 2) {
                    s.dum.c = s.dum.c - P.dz;
                    s.tip.c = s.tip.c - P.dz;
                }
            } else {
                s.dum.z = s.dum.z - P.dz;
                s.tip.z = s.tip.z - P.dz;
            }
            s.aligned = s.n > kAlignSteps;
            if (++s.k < P.nz) {
                start_level();
            } else {
                s.col = -1;
            }
            continue;
        }
        tip_dummy_df<G>(P, s.ex, s.dum, gmask, F, E);

        // ---- the integrator stage this evaluation belongs to (integrators.cpp:8-111) ----
        bool step_done = false;
        VecDF<G> SF = F;
        D SE = E;
        const D dt = s.dt;
        // x + w y of every component
        auto step = [](VecDF<G> x, D w, VecDF<G> y) { return vmap(x, y, [&](D a, D b) { return a + w * b; }); };
        if (P.minimiser == MAFM_MIN_SD) {
            step_done = true;
        } else if (P.integrator == MAFM_INT_EULER) {
            s.tip = step(s.tip, dt, s.vel);
            s.vel = step(s.vel, dt, F);
            step_done = true;
        } else if (P.integrator == MAFM_INT_MIDPOINT) {
            const D h(__fmul_rn(dt.h, 0.5f), __fmul_rn(dt.l, 0.5f));   // dt / 2, exactly
            if (s.phase == DF_EVAL0) {
                s.ex = step(s.tip, h, s.vel);
                s.u = step(s.vel, h, F);
                s.phase = DF_EVAL1;
            } else {
                s.tip = step(s.tip, dt, s.u);
                s.vel = step(s.vel, dt, F);
                step_done = true;
            }
        } else {   // RK4
            const D h(__fmul_rn(dt.h, 0.5f), __fmul_rn(dt.l, 0.5f));   // dt / 2, exactly
            auto sum = [](VecDF<G> x, VecDF<G> y) { return vmap(x, y, [](D a, D b) { return a + b; }); };
            if (s.phase == DF_EVAL0) {
                s.fs = F; s.es = E; s.vs = s.vel;
                s.ex = step(s.tip, h, s.vel);
                s.u = step(s.vel, h, F);
                s.phase = DF_EVAL1;
            } else if (s.phase == DF_EVAL1 || s.phase == DF_EVAL2) {
                const D two(2);
                s.fs = step(s.fs, two, F);
                s.es = s.es + two * E;
                s.vs = step(s.vs, two, s.u);
                const D w = s.phase == DF_EVAL1 ? h : dt;
                s.ex = step(s.tip, w, s.u);
                s.u = step(s.vel, w, F);
                s.phase = s.phase + 1;
            } else {
                s.fs = sum(s.fs, F);
                s.es = s.es + E;
                s.vs = sum(s.vs, s.u);
                const D s6 = dt / D(6);
                const D sixth = D(1.0 / 6.0);
                s.tip = step(s.tip, s6, s.vs);
                s.vel = step(s.vel, s6, s.fs);
                SF = vmap(s.fs, s.fs, [&](D a, D) { return a * sixth; });
                SE = s.es * sixth;
                step_done = true;
            }
        }
        if (!step_done) continue;

        // ---- end of a minimiser step: FIREMinimisation / SDMinimisation
        //      (minimiser.cpp:39-129) ----
        const D prev = s.energy;
        s.energy = SE;
        const D ediff = SE - prev;
        const D fl = dfl_sqrt(vdot<G>(SF, SF, gmask));
        bool conv;
        {
            // checkConvergence (minimiser.cpp:15-37), and its near-ties
            const bool e_ok = dfl_fabs(ediff) < P.etol, f_ok = fl < P.ftol;
            conv = P.minterm == MAFM_TERM_E ? e_ok : P.minterm == MAFM_TERM_F ? f_ok : (e_ok && f_ok);
            const D ea = dfl_fabs(ediff) - P.etol, fa = fl - P.ftol;
            const bool e_tie = dfl_fabs(ea) < P.tie.conv_e, f_tie = dfl_fabs(fa) < P.tie.conv_f;
            bool near;
            if (P.minterm == MAFM_TERM_E) near = e_tie;
            else if (P.minterm == MAFM_TERM_F) near = f_tie;
            else near = (e_tie && !(fa > P.tie.conv_f)) || (f_tie && !(ea > P.tie.conv_e));
            s.tie |= near;
        }
        if (s.tie && repair_list) {
            give_up();
            continue;
        }
        if (conv) {
            s.phase = DF_OUT;
            s.ex = s.tip;
            continue;
        }
        if (P.minimiser == MAFM_MIN_SD) {
            s.tip = vmap(s.tip, SF, [&](D x, D f) { return x + P.dt * f; });
        } else {
            const VecDF<G> w = s.vel;
            const D pw = vdot<G>(w, SF, gmask);
            VecDF<G> fh = own<G>(V3D{D(0), D(0), D(0)});
            if (fl > D(1e-10)) {
                const D ifl = dfl_rcp(fl);
                fh = vmap(SF, SF, [&](D f, D) { return f * ifl; });
            }
            const D vl = dfl_sqrt(vdot<G>(w, w, gmask));
            s.tie |= dfl_fabs(pw) < vl * (P.tie.p_f + P.tie.p_v * fl);
            if (s.tie && repair_list) {
                give_up();
                continue;
            }
            const D one_a = D(1) - s.alpha;
            s.vel = vmap(w, fh, [&](D x, D f) { return one_a * x + s.alpha * f * vl; });
            if (pw < D(0)) {
                s.vel = own<G>(V3D{D(0), D(0), D(0)});
                s.nnn = 0;
                s.dt = s.dt * D(0.5);
                s.alpha = D(0.1);
            } else {
                if (s.nnn > 5) {
                    const D g = s.dt * D(1.1);
                    const D dt_max = D(10) * P.dt;
                    s.dt = dt_max < g ? dt_max : g;
                    s.alpha = s.alpha * D(0.99);
                }
                s.nnn++;
            }
        }
        s.n++;
        s.phase = s.n >= P.maxsteps ? DF_OUT : DF_EVAL0;
        s.ex = s.tip;
    }

    // ---- the warp's columns are done: FP64 re-relaxation of listed columns ----
    if (repair_list && !(err & ERR_WATCHDOG)) {
        Node64* buf = reinterpret_cast<Node64*>(df_smem) + (size_t)(threadIdx.x >> 5) * 2 * kWarpChunk;
        long long rsteps = 0;
        unsigned long long revals = 0, rpairs = 0;
        unsigned rstatus = 0;
        for (;;) {
            unsigned long long slot = kNoEntry;
            if (lane == 0) slot = claim_repair(ctr, repair_cap);
            slot = __shfl_sync(kFull, slot, 0);
            if (slot == kNoEntry) break;
            unsigned long long e = kNoEntry;
            if (lane == 0) e = wait_entry(repair_list + slot, err);
            e = __shfl_sync(kFull, e, 0);
            if (e == kNoEntry) break;
            const BatchScan& R = scans64[(int)(e >> 32)];
            const long long c = (long long)(unsigned)(e & 0xffffffffull);
            EvalWarp64 ev{R.p, R.p.atoms64, R.p.n_terms_direct, R.p.ts_mode, lane, buf,
                          R.n_pairs_per_eval, 0u, 0ull};
            relax_column_t<double>(ev, R.p, c, R.out + (size_t)(c - R.col_begin) * R.p.nz, lane == 0,
                                   true, rsteps, revals, rstatus);
            rpairs += ev.pairs;
            err |= ev.err;
            __syncwarp();
        }
        if (lane == 0) {
            steps += (unsigned long long)rsteps;   // modular: a replacement subtracts
            evals += revals;
            pairs += rpairs;
            status_or |= rstatus;
        }
    }
    for (int off = 16; off > 0; off >>= 1) {
        steps += __shfl_xor_sync(kFull, steps, off);
        evals += __shfl_xor_sync(kFull, evals, off);
        pairs += __shfl_xor_sync(kFull, pairs, off);
        status_or |= __shfl_xor_sync(kFull, status_or, off);
        err |= __shfl_xor_sync(kFull, err, off);
    }
    if (lane == 0) {
        atomicAdd(&ctr->total_steps, steps);
        atomicAdd(&ctr->force_evals, evals);
        atomicAdd(&ctr->pair_evals, pairs);
        if (status_or | err) atomicOr(&ctr->error_word, status_or | err);
    }
}

__global__ void nodes_to_df_kernel(const Node64* in, NodeDF* out, long long n) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x) {
        const Node64 v = in[i];
        out[i] = NodeDF{D(v.x), D(v.y), D(v.z), D(v.w)};
    }
}

// The sums of the NB tips of a strip (the same x and y).
template <int NB>
struct StripSums {
    LazySum2 fx[NB], fy[NB], fz[NB], ee[NB];
};

// One record for a strip: the x and y separations and their squares once for all
// of its tips.
template <int NB>
__device__ __forceinline__ void strip_record(const ScanParamsDF& p, int r, D2 tx, D2 ty, const D2 (&tz)[NB],
                                             StripSums<NB>& sm) {
    const bool lj = r < p.n_lj_pairs;
    const PairDF2 t = lj ? load_pair<MAFM_PAIR_LJ>(p.pairs + r) : load_pair<MAFM_PAIR_MORSE>(p.pairs + r);
    const D2 dx = dfl2_sub_u(tx, t.x), dy = dfl2_sub_u(ty, t.y);
    const D2 dxy2 = dfl2_add_u(sq_u(dx), sq_u(dy));
#pragma unroll
    for (int m = 0; m < NB; ++m) {
        const D2 dz = dfl2_sub_u(tz[m], t.z);
        const D2 r2 = dfl2_add_u(dxy2, sq_u(dz));
        if (lj) pair_df2_at<MAFM_PAIR_LJ>(t, dx, dy, dz, r2, sm.fx[m], sm.fy[m], sm.fz[m], sm.ee[m]);
        else pair_df2_at<MAFM_PAIR_MORSE>(t, dx, dy, dz, r2, sm.fx[m], sm.fy[m], sm.fz[m], sm.ee[m]);
    }
}

// Simulation::buildTipGridInteractions (simulation.cpp:420-501) in
// double-float.  One thread per strip of NB consecutive nodes of a grid
// column (z fastest, so a warp's strips share x and y and read the same term
// records): the tip on each node (the node's x and y wrapped into the cell
// under tip_pbc, as temp_system does, :462-464), every tip–surface term of p
// (ts_mode 1: with the external field).  The x and y separations of a record
// and their squares are formed once for the strip.
template <int NB>
__global__ void __launch_bounds__(128) grid_builddf_kernel(const ScanParamsDF p, NodeDF* out) {
    const GridViewDF& g = p.grid;
    const int nzs = (g.n[2] + NB - 1) / NB;
    const long long total = (long long)g.n[0] * g.n[1] * nzs;
    const int n_all = p.n_lj_pairs + p.n_morse_pairs;
    for (long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
         idx += (long long)gridDim.x * blockDim.x) {
        const int k0 = (int)(idx % nzs) * NB;
        const long long ij = idx / nzs;
        const int j = (int)(ij % g.n[1]), i = (int)(ij / g.n[1]);
        D x, y;
        dummy_xy_t(p, p.tip_pbc != 0, D(i) * g.basis[0] + g.origin[0], D(j) * g.basis[4] + g.origin[1],
                   x, y);
        const D2 tx = dfl2(x), ty = dfl2(y);
        D2 tz[NB];
#pragma unroll
        for (int m = 0; m < NB; ++m) tz[m] = dfl2(D(k0 + m) * g.basis[8] + g.origin[2]);
        StripSums<NB> sm;
#pragma unroll 1
        for (int r = 0; r < n_all; ++r) strip_record<NB>(p, r, tx, ty, tz, sm);
#pragma unroll
        for (int m = 0; m < NB; ++m) {
            if (k0 + m >= g.n[2]) break;
            V3D F = {sm.fx[m].value(), sm.fy[m].value(), sm.fz[m].value()};
            D E = sm.ee[m].value();
            if (p.ts_mode == 1) {
                V3D f;
                D e;
                interp_df(p.es, V3D{x, y, D(k0 + m) * g.basis[8] + g.origin[2]}, f, e);
                F = {F.x + f.x, F.y + f.y, F.z + f.z};
                E = E + e;
            }
            out[ij * g.n[2] + k0 + m] = NodeDF{F.x, F.y, F.z, E};
        }
    }
}

// Each double-float node as FP64: h + l (exact, both parts fit 53 bits).
__global__ void nodes_df_to_64_kernel(const NodeDF* in, Node64* out, long long n) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x) {
        const NodeDF v = in[i];
        out[i] = Node64{to_double(v.x), to_double(v.y), to_double(v.z), to_double(v.w)};
    }
}

// ---- grid build with interpolated far terms -------------------------------------
//
// Far from an atom its force is smooth, so within a block of nodes the sum over
// the far records is evaluated at 16 x 16 x 16 Chebyshev points and interpolated
// to the block's nodes, and only the records near the block are evaluated at every
// node.  A record is far from a block when, on every axis, the ellipse around the
// block's interval (scaled to [-1, 1]) on which the term has its nearest
// singularity has a half axis of at least kFarAxis.  At that distance a force
// r^-7 is interpolated to 4.2e-16 of itself at worst, the Coulomb force and an
// energy r^-6 better, and a force r^-13 to 3.1e-13 beside a block much longer than
// wide, 6e-14 beside a block about as long as wide (evaluated in extended
// precision; 1.3e-14 from 12 on, 1e-15 from 14 on).  That part is at most 2 (sigma /
// r)^6 of a term's force, with r >= 7.2 A for the shortest blocks (1.6 A) and 14.4 A
// for 3.2 A ones, so that for sigma = 3.2 A a term is good to 5e-15 and 5e-16 of itself.  What a
// double-float term itself rounds is larger: nodes above slabs and molecules
// differ from the FP64 build by 4e-14 to 1e-13 rms with either build, also where the
// pairs have no attraction at all (up to 7e-13 at single nodes).  Morse records are always near:
// exp(-2 a r) over an interval of half length h converges with a h, whatever the
// distance, and a term with a = 2 A^-1 over 3.2 A would be good to 1e-7 of itself
// only, which counts where every term is weak.  Blocks, Chebyshev points and the
// interpolation weights are laid out once (plan_far_df); every build classifies
// the records and evaluates all of it.
//
// Slab of 9,216 records: 64 x 64 px (157 x 157 x 141 nodes) 270 -> 46 ms, 256 x 256
// px (541 x 541 x 141) 3198 -> 481 ms; and fewer roundings per node: the nodes'
// error against FP64 falls from 1.2e-11 to 5.9e-14 rms (40 x 40 px).

constexpr int kFarP = kFarPoints;

// Half axis of the ellipse through a singularity at distance off along the axis
// from the interval's centre and gap beside it.
__host__ __device__ __forceinline__ float far_axis(float off, float gap, float half) {
    const float u = off / half, v = gap / half;
    return 0.5f * (sqrtf((u - 1) * (u - 1) + v * v) + sqrtf((u + 1) * (u + 1) + v * v));
}

// Whether the point a is near the box of centre c and half sizes h.
__host__ __device__ __forceinline__ bool near_box(const float a[3], const float c[3], const float h[3]) {
    float d[3], gap[3];
    for (int m = 0; m < 3; ++m) {
        d[m] = fabsf(a[m] - c[m]);
        gap[m] = fmaxf(d[m] - h[m], 0.f);
    }
    for (int m = 0; m < 3; ++m) {
        const float ga = gap[(m + 1) % 3], gb = gap[(m + 2) % 3];
        if (far_axis(d[m], sqrtf(ga * ga + gb * gb), h[m]) < kFarAxis) return true;
    }
    return false;
}

struct FarBlock {
    int b[3];        // block index per axis
};

// Block at of a launch.
__device__ __forceinline__ FarBlock far_block(const FarViewDF& f, int at) {
    const int id = f.first + at;
    FarBlock q;
    q.b[2] = id % f.nb[2];
    q.b[1] = id / f.nb[2] % f.nb[1];
    q.b[0] = id / f.nb[2] / f.nb[1];
    return q;
}

// One bit per record and block: set when the record is a Morse one (past the first
// n_lj) or either of its terms is near.
__global__ void far_classify_kernel(const FarViewDF f, const TermPairDF* pairs, int n_lj, int n_rec) {
    const FarBlock q = far_block(f, blockIdx.x);
    float c[3], h[3];
    for (int a = 0; a < 3; ++a) {
        c[a] = f.box[a][q.b[a]].x;
        h[a] = f.box[a][q.b[a]].y;
    }
    for (int w = threadIdx.x; w < f.words; w += blockDim.x) {
        unsigned bits = 0;
        for (int k = 0; k < 32 && 32 * w + k < n_rec; ++k) {
            const TermPairDF& t = pairs[32 * w + k];
            const float a0[3] = {t.xh.x, t.yh.x, t.zh.x}, a1[3] = {t.xh.y, t.yh.y, t.zh.y};
            if (32 * w + k >= n_lj || near_box(a0, c, h) || near_box(a1, c, h)) bits |= 1u << k;
        }
        f.mask[(size_t)blockIdx.x * f.words + w] = bits;
    }
}

// The near (or the far) records of a block for a strip, and the strip's values.
// The words are the same for all threads of the block: no divergence.
template <int NB>
__device__ __forceinline__ void strip_masked(const ScanParamsDF& p, const unsigned* mask, int words, bool far,
                                             D x, D y, const D (&z)[NB], NodeDF (&val)[NB]) {
    const D2 tx = dfl2(x), ty = dfl2(y);
    D2 tz[NB];
#pragma unroll
    for (int m = 0; m < NB; ++m) tz[m] = dfl2(z[m]);
    StripSums<NB> sm;
    const int n_rec = p.n_lj_pairs + p.n_morse_pairs;
    for (int w = 0; w < words; ++w) {
        unsigned bits = __ldg(mask + w);
        if (far) bits = ~bits & (n_rec - 32 * w >= 32 ? 0xffffffffu : (1u << (n_rec - 32 * w)) - 1u);
#pragma unroll 1
        while (bits) {
            const int r = 32 * w + __ffs(bits) - 1;
            bits &= bits - 1;
            strip_record<NB>(p, r, tx, ty, tz, sm);
        }
    }
#pragma unroll
    for (int m = 0; m < NB; ++m)
        val[m] = NodeDF{sm.fx[m].value(), sm.fy[m].value(), sm.fz[m].value(), sm.ee[m].value()};
}

// The far sums at a block's Chebyshev points: blockIdx.y the block, a thread NB
// points along z.
template <int NB>
__global__ void __launch_bounds__(128) far_coef_kernel(const ScanParamsDF p, const FarViewDF f) {
    const FarBlock q = far_block(f, blockIdx.y);
    const int t = blockIdx.x * 128 + threadIdx.x;   // < kFarP * kFarP * kFarP / NB
    const int k0 = t % (kFarP / NB) * NB, j = t / (kFarP / NB) % kFarP, i = t / (kFarP / NB) / kFarP;
    D z[NB];
#pragma unroll
    for (int m = 0; m < NB; ++m) z[m] = f.cheb[2][q.b[2] * kFarP + k0 + m];
    NodeDF val[NB];
    strip_masked<NB>(p, f.mask + (size_t)blockIdx.y * f.words, f.words, true,
                                f.cheb[0][q.b[0] * kFarP + i], f.cheb[1][q.b[1] * kFarP + j], z, val);
    NodeDF* o = f.coef + ((size_t)blockIdx.y * kFarP * kFarP + i * kFarP + j) * kFarP + k0;
#pragma unroll
    for (int m = 0; m < NB; ++m) o[m] = val[m];
}

// The near sums at a block's nodes, a thread four nodes along z.
__global__ void __launch_bounds__(128) far_near_kernel(const ScanParamsDF p, const FarViewDF f, NodeDF* out) {
    const FarBlock q = far_block(f, blockIdx.y);
    int lo[3], n[3];
    for (int a = 0; a < 3; ++a) {
        lo[a] = f.begin[a][q.b[a]];
        n[a] = f.begin[a][q.b[a] + 1] - lo[a];
    }
    const int nzs = (n[2] + 3) / 4;
    const int t = blockIdx.x * 128 + threadIdx.x;
    if (t >= n[0] * n[1] * nzs) return;
    const int k0 = lo[2] + t % nzs * 4, j = lo[1] + t / nzs % n[1], i = lo[0] + t / nzs / n[1];
    const int k1 = lo[2] + n[2];
    D z[4];
#pragma unroll
    for (int m = 0; m < 4; ++m) z[m] = f.pos[2][min(k0 + m, k1 - 1)];
    NodeDF val[4];
    strip_masked<4>(p, f.mask + (size_t)blockIdx.y * f.words, f.words, false, f.pos[0][i], f.pos[1][j],
                                z, val);
    NodeDF* o = out + ((long long)i * p.grid.n[1] + j) * p.grid.n[2];
#pragma unroll
    for (int m = 0; m < 4; ++m)
        if (k0 + m < k1) o[k0 + m] = val[m];
}

// sum_m l[m] c[m stride] of the nodes' four values, two per packed operation.
__device__ __forceinline__ NodeDF far_dot(const D* l, const NodeDF* c, int stride) {
    D2 f0 = {p_bcast(0.f), p_bcast(0.f)}, f1 = f0;
#pragma unroll 4
    for (int m = 0; m < kFarP; ++m) {
        const float4* v = reinterpret_cast<const float4*>(c + m * stride);
        const float4 a = v[0], b = v[1];
        const D2 w = dfl2(l[m]);
        f0 = dfl2_add_u(f0, dfl2_mul_u(D2{make_float2(a.x, a.z), make_float2(a.y, a.w)}, w));
        f1 = dfl2_add_u(f1, dfl2_mul_u(D2{make_float2(b.x, b.z), make_float2(b.y, b.w)}, w));
    }
    f0 = dfl2_norm(f0);
    f1 = dfl2_norm(f1);
    return NodeDF{dfl2_x(f0), dfl2_y(f0), dfl2_x(f1), dfl2_y(f1)};
}

// The far sums interpolated to a plane of a block's nodes (blockIdx.x: the plane
// along x, blockIdx.y: the block), added to the near sums in out, with the
// external field (ts_mode 1); and the nodes' FP64 copy.
__global__ void __launch_bounds__(256) far_interp_kernel(const ScanParamsDF p, const FarViewDF f, NodeDF* out,
                                                         Node64* out64) {
    __shared__ NodeDF plane[kFarP * kFarP];              // at the node's x
    __shared__ NodeDF rows[kFarMaxNodes * kFarP];        // at the nodes' x, y
    const FarBlock q = far_block(f, blockIdx.y);
    const int i = f.begin[0][q.b[0]] + blockIdx.x;
    if (i >= f.begin[0][q.b[0] + 1]) return;
    const int j0 = f.begin[1][q.b[1]], ny = f.begin[1][q.b[1] + 1] - j0;
    const int k0 = f.begin[2][q.b[2]], nz = f.begin[2][q.b[2] + 1] - k0;
    const NodeDF* c = f.coef + (size_t)blockIdx.y * kFarP * kFarP * kFarP;
    for (int t = threadIdx.x; t < kFarP * kFarP; t += 256)
        plane[t] = far_dot(f.lag[0] + i * kFarP, c + t, kFarP * kFarP);
    __syncthreads();
    for (int t = threadIdx.x; t < ny * kFarP; t += 256)
        rows[t] = far_dot(f.lag[1] + (j0 + t / kFarP) * kFarP, plane + t % kFarP, kFarP);
    __syncthreads();
    for (int t = threadIdx.x; t < ny * nz; t += 256) {
        const int j = t / nz, k = t % nz;
        const NodeDF v = far_dot(f.lag[2] + (k0 + k) * kFarP, rows + j * kFarP, 1);
        const long long at = ((long long)i * p.grid.n[1] + j0 + j) * p.grid.n[2] + k0 + k;
        const NodeDF nr = out[at];
        NodeDF s = {nr.x + v.x, nr.y + v.y, nr.z + v.z, nr.w + v.w};
        if (p.ts_mode == 1) {
            V3D fe;
            D e;
            interp_df(p.es, V3D{f.pos[0][i], f.pos[1][j0 + j], f.pos[2][k0 + k]}, fe, e);
            s = {s.x + fe.x, s.y + fe.y, s.z + fe.z, s.w + e};
        }
        out[at] = s;
        out64[at] = Node64{to_double(s.x), to_double(s.y), to_double(s.z), to_double(s.w)};
    }
}

}  // namespace

std::vector<TermPairDF> term_pairs_df(const std::vector<AtomRec64>& terms, int& n_lj_pairs,
                                      int& n_morse_pairs) {
    auto split = [](double v, float2& hi, float2& lo, int e) {
        const float h = (float)v, l = (float)(v - (double)h);
        (e ? hi.y : hi.x) = h;
        (e ? lo.y : lo.x) = l;
    };
    std::vector<TermPairDF> out;
    auto add_run = [&](int kind) {
        std::vector<const AtomRec64*> run;
        for (const AtomRec64& r : terms)
            if (r.kind == kind) run.push_back(&r);
        for (size_t i = 0; i < run.size(); i += 2) {
            TermPairDF q{};
            for (int e = 0; e < 2; ++e) {
                // the second element of an odd run's last record: zero
                // parameters and charge at the first element's position
                const AtomRec64& r = *run[i + e < run.size() ? i + e : i];
                const bool real = i + e < run.size();
                split(r.x, q.xh, q.xl, e);
                split(r.y, q.yh, q.yl, e);
                split(r.z, q.zh, q.zl, e);
                split(real && r.coul ? r.qq : 0.0, q.qqh, q.qql, e);
                split(real ? r.p0 : 0.0, q.p0h, q.p0l, e);
                split(real ? r.p1 : 0.0, q.p1h, q.p1l, e);
                split(real ? r.p2 : 0.0, q.p2h, q.p2l, e);
                if (real && r.coul) q.coul = 1;
            }
            out.push_back(q);
        }
        return (int)((run.size() + 1) / 2);
    };
    n_lj_pairs = add_run(MAFM_PAIR_LJ);
    n_morse_pairs = add_run(MAFM_PAIR_MORSE);
    return out;
}

static GridViewDF grid_view_df(const GridView& g, const NodeDF* nodes) {
    GridViewDF q{};
    q.g = nodes;
    for (int a = 0; a < 3; ++a) {
        q.n[a] = g.n[a];
        q.origin[a] = D(g.origin[a]);
    }
    q.periodic = g.periodic;
    q.orthogonal = g.orthogonal;
    for (int k = 0; k < 9; ++k) {
        q.basis[k] = D(g.basis[k]);
        q.inv[k] = D(g.inv[k]);
    }
    return q;
}

ScanParamsDF params_df(const ScanParams& p, const TermPairDF* pairs, int n_lj_pairs,
                       int n_morse_pairs, const NodeDF* es_nodes, const NodeDF* grid_nodes) {
    ScanParamsDF q{};
    q.n_lj_pairs = n_lj_pairs;
    q.n_morse_pairs = n_morse_pairs;
    q.pairs = pairs;
    q.ts_mode = p.ts_mode;
    q.es = grid_view_df(p.es, es_nodes);
    q.grid = grid_view_df(p.grid, grid_nodes);
    for (int a = 0; a < 3; ++a) {
        q.offset[a] = D(p.offset[a]);
        q.td_p[a] = D(p.td_p[a]);
    }
    for (int k = 0; k < 9; ++k) {
        q.cell[k] = D(p.cell[k]);
        q.cell_inv[k] = D(p.cell_inv[k]);
    }
    q.td_kind = p.td_kind;
    q.td_coul = p.td_coul;
    q.td_qq = D(p.td_qq);
    q.harm_k = D(p.harm_k);
    q.harm_r0 = D(p.harm_r0);
    q.tip_dummy_d = D(p.tip_dummy_d);
    q.nx = p.nx; q.ny = p.ny; q.nz = p.nz;
    q.tip_pbc = p.tip_pbc;
    q.dx = D(p.dx); q.dy = D(p.dy); q.dz = D(p.dz); q.zhigh = D(p.zhigh);
    q.minimiser = p.minimiser;
    q.integrator = p.integrator;
    q.stage_mask = p.minimiser == MAFM_MIN_SD || p.integrator == MAFM_INT_EULER ? 0u
                   : p.integrator == MAFM_INT_MIDPOINT ? 1u : 3u;
    q.minterm = p.minterm;
    q.maxsteps = p.maxsteps;
    q.etol = D(p.etol);
    q.ftol = D(p.ftol);
    q.dt = D(p.dt);
    // Near-tie margins: 1e-8 of the tolerances, 1e-10 of |F| for the sign of
    // P; the double-float error of a force is about 1e-13 of the largest term.
    // MAFM_DF_TIE_SCALE multiplies them (a diagnostic: a huge scale sends
    // every column to the FP64 re-relaxation).
    double k = 1.0;
    if (const char* e = std::getenv("MAFM_DF_TIE_SCALE")) {
        const double v = std::atof(e);
        if (v > 0.0 && v <= 1.0e30) k = v;
    }
    q.tie.conv_e = D(k * 1.0e-8 * p.etol);
    q.tie.conv_f = D(k * 1.0e-8 * p.ftol);
    q.tie.p_f = D(k * 1.0e-8 * p.ftol);
    q.tie.p_v = D(k * 1.0e-10);
    return q;
}

// Shared memory of a block: the FP64 re-relaxation's per-warp buffers.
constexpr size_t kDfSmem = (size_t)(128 / 32) * 2 * kWarpChunk * sizeof(Node64);

// Default: one lane per column while the columns fill the resident lanes;
// fewer columns share out their terms, G = the largest power of two up to 8
// with G x columns <= 1.25 x the resident lanes.  Measured (MAFM_DF_LANES
// overrides), 41 heights, G = 1 / 2 / 4 / 8: 401 x 401 cluster (160,801 columns,
// 58,368 resident lanes) 589 / 721 / 885 / 1396 ms; 128 x 128 cluster at 0.1 A
// (16,384) 288 / 271 / 275 / 357; 101 x 101 graphene (10,201) 142 / 115 / 102 / 133;
// 85 x 85 cluster at 0.2 A (7,225) 160 / 108 / 94 / 103; 60 x 60 graphene 118 / 76 / 52 /
// 53; 40 x 40 cluster at 0.5 A 157 / 103 / 69 / 60.
int df_lanes_per_column(long long n_cols, int requested) {
    if (requested == 1 || requested == 2 || requested == 4 || requested == 8) return requested;
    if (const char* e = std::getenv("MAFM_DF_LANES")) {
        const int v = std::atoi(e);
        if (v == 1 || v == 2 || v == 4 || v == 8) return v;
    }
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, relaxdf_kernel<1>, 128, kDfSmem) != cudaSuccess ||
        per_sm <= 0)
        per_sm = 1;
    const long long lanes = (long long)sm_count() * per_sm * 128;
    int g = 1;
    while (g < 8 && n_cols > 0 && 4 * (2 * g * n_cols) <= 5 * lanes) g *= 2;
    return g;
}

template <int G>
static cudaError_t launch_relaxdf_g(const BatchDF* scans, const BatchScan* scans64, int n_scans,
                                   long long n_cols, RunCounters* ctr,
                                   unsigned long long* repair_list, unsigned repair_cap,
                                   unsigned long long watchdog_ns, cudaStream_t s) {
    constexpr int kThreads = 128;
    int per_sm = 0;
    cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, relaxdf_kernel<G>, kThreads,
                                                                  kDfSmem);
    if (e != cudaSuccess) return e;
    if (per_sm <= 0) per_sm = 1;
    long long blocks = (long long)sm_count() * per_sm;
    const long long need = (n_cols * G + kThreads - 1) / kThreads;
    blocks = std::max(1ll, std::min(blocks, need));
    relaxdf_kernel<G><<<(unsigned)blocks, kThreads, kDfSmem, s>>>(
        scans, scans64, n_scans, n_cols, ctr, repair_list, repair_list ? repair_cap : 0u, watchdog_ns);
    return cudaGetLastError();
}

cudaError_t launch_relaxdf(const BatchDF* scans, const BatchScan* scans64, int n_scans, long long n_cols,
                           RunCounters* ctr, unsigned long long* repair_list, unsigned repair_cap,
                           unsigned long long watchdog_ns, int lanes_per_column, cudaStream_t s) {
    if (n_cols <= 0) return cudaSuccess;
    if (repair_list) {
        // an unwritten entry reads as kNoEntry (all bits set)
        const cudaError_t e = cudaMemsetAsync(repair_list, 0xFF, (size_t)repair_cap * sizeof(*repair_list), s);
        if (e != cudaSuccess) return e;
    }
    switch (df_lanes_per_column(n_cols, lanes_per_column)) {
        case 2: return launch_relaxdf_g<2>(scans, scans64, n_scans, n_cols, ctr, repair_list, repair_cap, watchdog_ns, s);
        case 4: return launch_relaxdf_g<4>(scans, scans64, n_scans, n_cols, ctr, repair_list, repair_cap, watchdog_ns, s);
        case 8: return launch_relaxdf_g<8>(scans, scans64, n_scans, n_cols, ctr, repair_list, repair_cap, watchdog_ns, s);
        default: return launch_relaxdf_g<1>(scans, scans64, n_scans, n_cols, ctr, repair_list, repair_cap, watchdog_ns, s);
    }
}

cudaError_t launch_nodes_to_df(const Node64* in, NodeDF* out, long long n, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    long long blocks = std::min((n + 255) / 256, (long long)sm_count() * 32);
    nodes_to_df_kernel<<<(unsigned)blocks, 256, 0, s>>>(in, out, n);
    return cudaGetLastError();
}

// Lay out the blocks of a rigid grid for the interpolated build, or return false
// where it would not pay: the node positions (x and y wrapped into the cell, on
// the host as the FP64 build wraps them), blocks of about the length that costs
// least by the estimate below, none across a jump of the wrapped positions, and
// for every axis Chebyshev points and the weights of the block's nodes.  xyz: the
// positions of the records' two terms.
bool plan_far_df(const ScanParams& p, const GridView& g, const std::vector<float>& xyz, int n_lj,
                 FarPlanDF& plan) {
    const long long n_rec = (long long)xyz.size() / 6;
    if (n_rec < 64) return false;
    if (p.tip_pbc)
        for (int r = 0; r < 3; ++r)
            for (int c = 0; c < 3; ++c)
                if (r != c && (p.cell[3 * r + c] != 0 || p.cell_inv[3 * r + c] != 0)) return false;
    std::vector<double> pos[3];
    for (int a = 0; a < 3; ++a) {
        pos[a].resize(g.n[a]);
        for (int i = 0; i < g.n[a]; ++i) {
            double x = i * g.basis[4 * a] + g.origin[a];
            if (p.tip_pbc && a < 2) {   // System::setDummyXY for a diagonal cell
                double cn = p.cell_inv[4 * a] * (x - p.offset[a]);
                cn -= std::floor(cn);
                x = p.cell[4 * a] * cn + p.offset[a];
            }
            pos[a][i] = x;
        }
    }
    // blocks of one axis: runs without a jump, cut evenly to at most length len
    auto cut = [&](int a, double len) {
        const double s = g.basis[4 * a];
        const int most = std::min(std::max((int)(len / s + 0.5) + 1, 2), kFarMaxNodes);
        std::vector<int> begin;
        for (int i = 0; i < g.n[a];) {
            int e = i + 1;
            while (e < g.n[a] && std::fabs(pos[a][e] - pos[a][e - 1] - s) < 0.01 * s) ++e;
            const int parts = (e - i + most - 1) / most;
            for (int q = 0; q < parts; ++q) begin.push_back(i + (int)((long long)(e - i) * q / parts));
            i = e;
        }
        begin.push_back(g.n[a]);
        return begin;
    };
    auto box = [&](int a, const std::vector<int>& begin, int b) {
        const double lo = pos[a][begin[b]], hi = pos[a][begin[b + 1] - 1];
        // one node: an interval around it
        return std::make_pair(0.5 * (lo + hi), std::max(0.5 * (hi - lo), 0.5 * g.basis[4 * a]));
    };
    const double nodes = (double)g.n[0] * g.n[1] * g.n[2];
    const double direct = nodes * n_rec;
    const long long step = (n_rec + 1023) / 1024;
    double best = 0.7 * direct;
    std::vector<int> begin[3];
    for (double len : {1.6, 2.4, 3.2, 4.8, 6.4}) {
        std::vector<int> bg[3];
        double blocks = 1;
        for (int a = 0; a < 3; ++a) {
            bg[a] = cut(a, len);
            blocks *= (double)bg[a].size() - 1;
        }
        const double coef = blocks * kFarP * kFarP * kFarP;
        if (blocks > 65535 || coef * n_rec > best) continue;
        // near records, of a few blocks and at most about 1,000 records
        double near = 0;
        long long tried = 0;
        for (int q : {0, 7, 8}) {   // two corners and the middle
            float c[3], h[3];
            for (int a = 0; a < 3; ++a) {
                const int last = (int)bg[a].size() - 2;
                const auto b = box(a, bg[a], q == 8 ? last / 2 : (q >> a & 1) ? last : 0);
                c[a] = (float)b.first;
                h[a] = (float)b.second;
            }
            for (long long r = 0; r < n_rec; r += step, ++tried)
                near += r >= n_lj || near_box(&xyz[6 * r], c, h) || near_box(&xyz[6 * r + 3], c, h);
        }
        near *= (double)n_rec / tried;
        // per node the interpolation costs about four records
        const double cost = coef * (n_rec - near) + nodes * (near + 4);
        if (cost < best) {
            best = cost;
            for (int a = 0; a < 3; ++a) begin[a] = bg[a];
        }
    }
    if (begin[0].empty()) return false;
    const double pi = 3.14159265358979323846;
    for (int a = 0; a < 3; ++a) {
        FarAxisDF& A = plan.axis[a];
        A.begin = begin[a];
        A.pos.clear();
        for (double x : pos[a]) A.pos.push_back(D(x));
        A.lag.assign((size_t)g.n[a] * kFarP, D(0.0f, 0.0f));
        A.cheb.clear();
        A.box.clear();
        for (size_t b = 0; b + 1 < begin[a].size(); ++b) {
            const auto bx = box(a, begin[a], (int)b);
            A.box.push_back(make_float2((float)bx.first, (float)bx.second));
            long double x[kFarP], w[kFarP];
            for (int m = 0; m < kFarP; ++m) {
                const D q(bx.first + bx.second * std::cos((2 * m + 1) * pi / (2 * kFarP)));
                A.cheb.push_back(q);
                x[m] = (long double)q.h + (long double)q.l;   // the point as the kernels have it
            }
            for (int m = 0; m < kFarP; ++m) {
                w[m] = 1;
                for (int k = 0; k < kFarP; ++k)
                    if (k != m) w[m] *= 2 * (x[m] - x[k]) / (long double)bx.second;
                w[m] = 1 / w[m];
            }
            for (int i = begin[a][b]; i < begin[a][b + 1]; ++i) {
                const D q = A.pos[i];
                const long double v = (long double)q.h + (long double)q.l;
                long double sum = 0;
                int hit = -1;
                for (int m = 0; m < kFarP; ++m) {
                    if (v == x[m]) hit = m;
                    else sum += w[m] / (v - x[m]);
                }
                for (int m = 0; m < kFarP; ++m)
                    A.lag[(size_t)i * kFarP + m] =
                        hit >= 0 ? D(hit == m ? 1.0f : 0.0f, 0.0f) : D((double)(w[m] / (v - x[m]) / sum));
            }
        }
    }
    plan.words = (int)((n_rec + 31) / 32);
    return true;
}

static cudaError_t launch_far(const ScanParamsDF& p, NodeDF* out, Node64* out64, const FarViewDF& f, cudaStream_t s) {
    const int blocks = f.nb[0] * f.nb[1] * f.nb[2];
    // Four points a thread share the x and y separations; grids of so few blocks
    // that this would not fill the GPU once take one (slab of 16 px 10.7 -> 7.5
    // ms, 24 px 13.3 -> 10.3 ms; 64 px 46.2 ms either way, 256 px 478 / 528 ms).
    constexpr int kPoints = kFarP * kFarP * kFarP;
    const bool few = kPoints / 4 / 128 * (long long)blocks < 3ll * sm_count();
    for (FarViewDF c = f; c.first < blocks; c.first += kFarChunk) {
        const unsigned n = (unsigned)std::min(kFarChunk, blocks - c.first);
        far_classify_kernel<<<n, 128, 0, s>>>(c, p.pairs, p.n_lj_pairs, p.n_lj_pairs + p.n_morse_pairs);
        if (few) far_coef_kernel<1><<<dim3(kPoints / 128, n), 128, 0, s>>>(p, c);
        else far_coef_kernel<4><<<dim3(kPoints / 4 / 128, n), 128, 0, s>>>(p, c);
        far_near_kernel<<<dim3((unsigned)((f.max_strips + 127) / 128), n), 128, 0, s>>>(p, c, out);
        far_interp_kernel<<<dim3((unsigned)f.max_planes, n), 256, 0, s>>>(p, c, out, out64);
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

cudaError_t launch_grid_builddf(const ScanParamsDF& p, NodeDF* out, Node64* out64, const FarViewDF* far,
                                cudaStream_t s) {
    const long long n = (long long)p.grid.n[0] * p.grid.n[1] * p.grid.n[2];
    if (n <= 0) return cudaSuccess;
    if (far) return launch_far(p, out, out64, *far, s);
    ScanParamsDF q = p;
    q.grid.g = out;
    constexpr int kNB = 4;
    const long long strips = (long long)p.grid.n[0] * p.grid.n[1] * ((p.grid.n[2] + kNB - 1) / kNB);
    int per_sm = 0;
    cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, grid_builddf_kernel<kNB>, 128, 0);
    if (e != cudaSuccess) return e;
    if (per_sm <= 0) per_sm = 1;
    const long long blocks = std::max(1ll, std::min((strips + 127) / 128, (long long)sm_count() * per_sm * 8));
    grid_builddf_kernel<kNB><<<(unsigned)blocks, 128, 0, s>>>(q, out);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    const long long b64 = std::min((n + 255) / 256, (long long)sm_count() * 32);
    nodes_df_to_64_kernel<<<(unsigned)b64, 256, 0, s>>>(out, out64, n);
    return cudaGetLastError();
}

}  // namespace mafm
