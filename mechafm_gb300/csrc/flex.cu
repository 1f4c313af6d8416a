// flex.cu — flexible molecules (`flexible on`) on the GPU, FP64.
//
// With a flexible molecule every surface atom whose xyz "fixed" flag is not 1
// moves with the tip (parse.cpp:559-563), held by bonds, angles, dihedrals,
// non-bonded pairs between bonded fragments, a substrate wall and XY tethers
// (simulation.cpp:516-693, interactions.cpp:268-370).  FIRE / SD and the
// integrators then run over all atoms (minimiser.cpp:39-129,
// integrators.cpp:8-111); convergence looks at the tip only.
//
// Layout: one block per pixel column, the atoms' positions, velocities and
// force accumulators in shared memory.  The reference sums each atom's force
// over its interaction list in list order; here every interaction is computed
// once, into force slots, and every atom has its list of (slot, sign) entries in
// that same order (built on the host), which one thread per component adds, so
// every per-atom sum is formed in the reference's order.  FIRE's P = sum_i v_i .
// F_i is summed by one thread in atom order.  Expressions follow the reference's
// operation order (vectors.hpp:99-125); the transcendental functions (exp,
// acos, sin, atan) are CUDA's, so results agree with the reference to
// rounding, not bit for bit.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "ieee64.cuh"
#include "mafm_internal.h"

struct mafm_flex {
    int device = 0;
    mafm_scan_desc d{};
    mafm::ScanParams P{};   // pixel grid, cell, minimiser, tip–dummy terms
    int n_sys = 0;          // atoms incl. dummy (0) and tip (1)
    int n_ts = 0;
    void* dev_block = nullptr;   // every device array, one allocation
    size_t block_bytes = 0;
    struct Dev {
        const double* pos0;         // [n_sys*3] initial positions
        const int* fixed;           // [n_sys]
        const void* ts;             // FlexTS[n_ts]
        const int* bonds;           // [2 n_bonds] system indices
        const double* bond_par;     // [2 n_bonds]
        const int* angles;          // [3 n_angles]
        const double* angle_par;
        const int* dihedrals;       // [4 n_dihedrals]
        const double* dihedral_par;
        const int* pairs;           // [2 n_pairs]
        const void* pair_par;       // FlexPair[n_pairs]
        const void* coul;           // FlexCoul of the pairs with charges
        const double* xy;           // [3 n_xy] atom (as double), x0, y0
        const int* list_begin;      // [n_sys + 1]
        const int* list;            // per atom, in the reference's order: slot << 1 | negated
        const int* warp_begin;      // [kFlexWarps + 1] chunks of every warp
        const int* chunk_kind;      // [chunks]
        const int* task;            // [32 chunks] interaction indices, -1: none
        int slot_base[12];          // first force slot of every kind
        int n_energies;             // the tip's terms: slots 0 .. n_energies - 1
    } dv{};
    int n_slots = 0;
    mafm::RunCounters* ctr = nullptr;
    mafm::RunCounters* host_ctr = nullptr;
    double sub[6] = {0, 0, 0, 0, 0, 0};   // multiplier, ulj, ushift, z0, rc, sig
    double sub_k = 0;
};

namespace mafm {
namespace {

enum : int {
    FT_TS_VDW = 0, FT_TS_COUL, FT_TD_VDW, FT_TD_COUL, FT_TD_HARM, FT_BOND, FT_ANGLE,
    FT_DIHEDRAL, FT_PAIR_VDW, FT_PAIR_COUL, FT_SUBSTRATE, FT_XY
};

// Force vectors an interaction leaves: one for its first atom (the second gets
// its negative); an angle's for atom 1, atom 2 and their sum; a dihedral's four.
__host__ __device__ constexpr int flex_slots(int kind) {
    return kind == FT_ANGLE ? 3 : kind == FT_DIHEDRAL ? 4 : 1;
}

constexpr int kFlexWarps = 8;

struct FlexTS {          // one tip–surface term: LJ / Morse (+ the image shift), or Coulomb
    int atom;            // system index of the surface atom
    int kind;            // MAFM_PAIR_LJ / MAFM_PAIR_MORSE
    double shift[3];
    double p[3];
    double qq;           // Coulomb term when coul
    int coul;
    int pad;
};

struct FlexPair {        // van der Waals part of a non-bonded pair
    int kind, pad;
    double p[3];
};

struct FlexCoul {        // Coulomb part of one whose charges are not zero
    int i, j;
    double qq;
};

struct V3 {
    double x, y, z;
};

__device__ __forceinline__ V3 v3(const double* p) { return V3{p[0], p[1], p[2]}; }
__device__ __forceinline__ V3 sub3(V3 a, V3 b) { return V3{a.x - b.x, a.y - b.y, a.z - b.z}; }
__device__ __forceinline__ V3 add3(V3 a, V3 b) { return V3{a.x + b.x, a.y + b.y, a.z + b.z}; }
__device__ __forceinline__ V3 scal(double s, V3 a) { return V3{s * a.x, s * a.y, s * a.z}; }
__device__ __forceinline__ V3 mul3(V3 a, double s) { return V3{a.x * s, a.y * s, a.z * s}; }
__device__ __forceinline__ V3 div3(V3 a, double s) { return V3{div64(a.x, s), div64(a.y, s), div64(a.z, s)}; }
__device__ __forceinline__ double dot3(V3 a, V3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ double len3(V3 a) { return sqrt64(a.x * a.x + a.y * a.y + a.z * a.z); }
__device__ __forceinline__ V3 cross3(V3 a, V3 b) {
    return V3{a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x};
}
// LJ (interactions.cpp:15-27) / Morse (:29-40): force on atom 1 of r_vec = x1 - x2.
__device__ __forceinline__ V3 vdw_force(int kind, const double p[3], V3 r, double& e) {
    if (kind == MAFM_PAIR_LJ) {
        const double r_sqr = r.x * r.x + r.y * r.y + r.z * r.z;
        const double r6 = r_sqr * r_sqr * r_sqr;
        const double ta = div64(p[1], r6 * r6);
        const double tb = div64(p[0], r6);
        e = ta - tb;
        return scal(div64(12 * ta - 6 * tb, r_sqr), r);
    }
    const double rl = len3(r);
    const double d = exp(-p[1] * (rl - p[2]));
    e = p[0] * (d * d - 2 * d + 1);
    const double f_abs = 2 * p[0] * p[1] * (d * d - d);
    return scal(div64(f_abs, rl), r);
}

// Coulomb (interactions.cpp:42-51).
__device__ __forceinline__ V3 coul_force(double qq, V3 r, double& e) {
    const double rl = len3(r);
    e = div64(qq, rl);
    return scal(div64(qq, rl * rl * rl), r);
}

struct FlexKernelArgs {
    mafm_flex::Dev dv;
    ScanParams P;
    double sub[6];
    double sub_k;
    int n_sys;
    int n_ts;
    int n_slots;
    int col_begin, col_end;
    mafm_point* out;
    int state_column;
    double* states;
    double* scratch;      // energies and force slots of every block, null: shared memory
    unsigned long long watchdog_ns;
    RunCounters* ctr;
};

__device__ __forceinline__ unsigned long long now_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ void put3(double* res, int slot, V3 v) {
    res[3 * slot] = v.x;
    res[3 * slot + 1] = v.y;
    res[3 * slot + 2] = v.z;
}

// One interaction of kind `kind` (all lanes of a warp the same kind): its force
// vectors into its slots, its energy into e (used for the tip's terms only).
__device__ void eval_task(const FlexKernelArgs& A, const double* pe, int kind, int idx, double* res,
                          double* en) {
    const auto& dv = A.dv;
    const FlexTS* ts = static_cast<const FlexTS*>(dv.ts);
    const FlexPair* pp = static_cast<const FlexPair*>(dv.pair_par);
    const int slot = dv.slot_base[kind] + idx * flex_slots(kind);
    auto P3 = [&](int i) { return v3(pe + 3 * i); };
    double e = 0;
    switch (kind) {
        case FT_TS_VDW: {   // LJInteraction(1, j, shift) / Morse
            const FlexTS& t = ts[idx];
            const V3 sh{t.shift[0], t.shift[1], t.shift[2]};
            put3(res, slot, vdw_force(t.kind, t.p, sub3(P3(1), add3(P3(t.atom), sh)), e));
            en[slot] = e;
            break;
        }
        case FT_TS_COUL: {
            const FlexTS& t = ts[idx];
            put3(res, slot, coul_force(t.qq, sub3(P3(1), P3(t.atom)), e));
            en[slot] = e;
            break;
        }
        case FT_TD_VDW: {   // addVDWInteraction(0, 1)
            put3(res, slot, vdw_force(A.P.td_kind, A.P.td_p, sub3(P3(0), P3(1)), e));
            en[slot] = e;
            break;
        }
        case FT_TD_COUL: {
            put3(res, slot, coul_force(A.P.td_qq, sub3(P3(0), P3(1)), e));
            en[slot] = e;
            break;
        }
        case FT_TD_HARM: {  // TipHarmonicInteraction (interactions.cpp:252-266)
            const V3 r_vec = sub3(P3(0), P3(1));
            const double r = sqrt64(r_vec.x * r_vec.x + r_vec.y * r_vec.y);
            const double dr = r - A.P.harm_r0;
            en[slot] = A.P.harm_k * dr * dr;
            V3 f{0, 0, 0};
            if (r > 1e-10) {
                const double c = div64(-2 * A.P.harm_k * dr, r);
                f = V3{c * r_vec.x, c * r_vec.y, 0};
            }
            put3(res, slot, f);
            break;
        }
        case FT_BOND: {     // HarmonicInteraction (interactions.cpp:298-309)
            const int i = dv.bonds[2 * idx], j = dv.bonds[2 * idx + 1];
            const double k = dv.bond_par[2 * idx], r0 = dv.bond_par[2 * idx + 1];
            const V3 r_vec = sub3(P3(i), P3(j));
            const double r = len3(r_vec);
            const double dr = r - r0;
            put3(res, slot, scal(div64(-2 * k * dr, r), r_vec));
            break;
        }
        case FT_ANGLE: {    // HarmonicAngleInteraction (interactions.cpp:311-338)
            const int sh = dv.angles[3 * idx], i1 = dv.angles[3 * idx + 1], i2 = dv.angles[3 * idx + 2];
            const double k = dv.angle_par[2 * idx], theta0 = dv.angle_par[2 * idx + 1];
            const V3 r1_vec = sub3(P3(i1), P3(sh));
            const V3 r2_vec = sub3(P3(i2), P3(sh));
            const double r1 = len3(r1_vec), r2 = len3(r2_vec);
            double cos_t = div64(dot3(r1_vec, r2_vec), r1 * r2);
            if (cos_t > 1) cos_t = 1;
            else if (cos_t < -1) cos_t = -1;
            const double theta = acos(cos_t);
            const double sin_t = sin(theta);
            const double d_theta = theta - theta0;
            const double f_mul = div64(-2 * k * d_theta, sin_t);
            const V3 f1 = scal(div64(-f_mul, r1), sub3(div3(r2_vec, r2), div3(mul3(r1_vec, cos_t), r1)));
            const V3 f2 = scal(div64(-f_mul, r2), sub3(div3(r1_vec, r1), div3(mul3(r2_vec, cos_t), r2)));
            put3(res, slot, f1);
            put3(res, slot + 1, f2);
            put3(res, slot + 2, add3(f1, f2));
            break;
        }
        case FT_DIHEDRAL: { // HarmonicDihedralInteraction (interactions.cpp:340-370)
            const int* at = dv.dihedrals + 4 * idx;
            const double k = dv.dihedral_par[2 * idx], sigma0 = dv.dihedral_par[2 * idx + 1];
            const V3 r12 = sub3(P3(at[0]), P3(at[1]));
            const V3 r23v = sub3(P3(at[1]), P3(at[2]));
            const V3 r43 = sub3(P3(at[3]), P3(at[2]));
            const double r23 = len3(r23v);
            const V3 m_vec = cross3(r12, r23v);
            const V3 n_vec = cross3(r43, r23v);
            const double m = len3(m_vec), n = len3(n_vec);
            const double tan_s = div64(dot3(n_vec, r12) * r23, dot3(m_vec, n_vec));
            const double sigma = atan(tan_s);
            const double d_sigma = sigma - sigma0;
            const double f_mul = 2 * k * d_sigma;
            put3(res, slot, scal(div64(-f_mul * r23, m * m), m_vec));
            put3(res, slot + 1, scal(-f_mul, sub3(scal(div64(dot3(r43, r23v), n * n * r23), n_vec),
                                                  scal(div64((r23 * r23) + dot3(r12, r23v), m * m * r23), m_vec))));
            put3(res, slot + 2, scal(-f_mul, add3(scal(div64(dot3(r12, r23v), m * m * r23), m_vec),
                                                  scal(div64((r23 * r23) - dot3(r43, r23v), n * n * r23), n_vec))));
            put3(res, slot + 3, scal(div64(f_mul * r23, n * n), n_vec));
            break;
        }
        case FT_PAIR_VDW: {
            const int i = dv.pairs[2 * idx], j = dv.pairs[2 * idx + 1];
            put3(res, slot, vdw_force(pp[idx].kind, pp[idx].p, sub3(P3(i), P3(j)), e));
            break;
        }
        case FT_PAIR_COUL: {
            const FlexCoul& q = static_cast<const FlexCoul*>(dv.coul)[idx];
            put3(res, slot, coul_force(q.qq, sub3(P3(q.i), P3(q.j)), e));
            break;
        }
        case FT_SUBSTRATE: { // SubstrateInteraction (interactions.cpp:280-296); idx: the atom
            const double dz = pe[3 * idx + 2] - A.sub[3];
            const double sig_z = div64(A.sub[5], dz);
            const double sig_z2 = sig_z * sig_z;
            const double sig_z4 = sig_z2 * sig_z2;
            const double sig_z10 = sig_z4 * sig_z4 * sig_z2;
            double fterm = 0.0;
            if (dz <= A.sub[4]) fterm += div64(4 * A.sub[0], dz) * (sig_z10 - sig_z4) + 2 * A.sub[1] * dz;
            // -0: adding it leaves x and y as they are, signed zeros too
            put3(res, slot, V3{-0.0, -0.0, fterm});
            break;
        }
        case FT_XY: {       // XYHarmonicInteraction (interactions.cpp:268-278)
            const int a = (int)dv.xy[3 * idx];
            const double rx = pe[3 * a] - dv.xy[3 * idx + 1];
            const double ry = pe[3 * a + 1] - dv.xy[3 * idx + 2];
            const double r = sqrt64(rx * rx + ry * ry);
            const double c = -2 * A.sub_k;
            put3(res, slot, r > 1e-10 ? V3{c * rx, c * ry, 0.0} : V3{0.0, 0.0, 0.0});
            break;
        }
        default:
            break;
    }
}

// Shared arrays of a block, 3 doubles per atom each.
struct Slice {
    double* pos;   // positions_
    double* vel;   // velocities_
    double* pe;    // positions of the current evaluation; the mixed velocities
    double* vk;    // RK4 v_k / midpoint v2
    double* fsum;  // RK4 force sum; forces_ of the last step otherwise
    double* vsum;  // RK4 velocity sum
    double* f;     // forces of the current evaluation
    double* dot;   // v_i . F_i
    double* en;    // energies of the tip's terms
    double* res;   // force slots
};

// What one thread decides for the block.
struct FlexCtl {
    double dt, alpha, e_tip, pw, e_eval;
    double ft[3];
    int conv, n_non_neg, col;
};

// One block of kFlexWarps warps relaxes one column.  An FP64 instruction of a
// warp takes 64 cycles whatever its lanes do, and an SM starts one every 19, so
// what counts is the number of warp instructions on the longest chain.  An
// evaluation therefore computes every interaction once, 32 of one kind to a
// warp, the kinds' chunks dealt to the warps by cost, into slots of shared
// memory; then one thread per atom and component adds the atom's slots in the
// reference's order.  The minimiser's per-atom parts run one thread per
// component, beside the convergence test on one warp and the power P on
// another.  A flexible C10H8 + H2 (25 columns x 6 heights): 505 -> 18.5 ms;
// before, a warp held a column, each lane evaluated its atoms' interactions
// one after another (the tip's 43 on one lane), and the kinds diverged.
__global__ void __launch_bounds__(32 * kFlexWarps, 2) flex_kernel(const __grid_constant__ FlexKernelArgs A) {
    extern __shared__ __align__(16) double flex_smem[];
    __shared__ FlexCtl ctl;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int kThreads = 32 * kFlexWarps;
    const int na = A.n_sys, nq = 3 * na;
    const size_t per = (size_t)nq;
    double* base = flex_smem;
    Slice S{base, base + per, base + 2 * per, base + 3 * per, base + 4 * per, base + 5 * per,
            base + 6 * per, base + 7 * per, base + 7 * per + na, nullptr};
    if (A.scratch) S.en = A.scratch + (size_t)blockIdx.x * (A.dv.n_energies + 3 * (size_t)A.n_slots);
    S.res = S.en + A.dv.n_energies;
    const ScanParams& P = A.P;
    const auto& dv = A.dv;
    const unsigned long long t0 = now_ns();
    unsigned long long my_steps = 0, my_evals = 0;   // thread 0
    unsigned err = 0;
    const int* fixed = dv.fixed;
    auto late = [&]() { return __syncthreads_or(tid == 0 && now_ns() - t0 > A.watchdog_ns) != 0; };

    // Forces at positions src into S.f and the tip's energy into ctl.e_eval;
    // tip_only: the tip–surface terms alone (System::evalTipSurfaceForces,
    // system.cpp:41-51), summed for the tip into ctl.ft.  Starts and ends with
    // a block barrier.
    auto evaluate = [&](const double* src, bool tip_only) {
        __syncthreads();
        for (int c = dv.warp_begin[warp]; c < dv.warp_begin[warp + 1]; ++c) {
            const int kind = dv.chunk_kind[c];
            if (tip_only && kind != FT_TS_VDW && kind != FT_TS_COUL) continue;
            const int idx = dv.task[32 * c + lane];
            if (idx >= 0) eval_task(A, src, kind, idx, S.res, S.en);
        }
        __syncthreads();
        const int n_f = tip_only ? 3 : nq;
        for (int q = tid; q < n_f; q += kThreads) {
            const int a = tip_only ? 1 : q / 3, d = tip_only ? q : q - 3 * a;
            double acc = 0;
            for (int i = dv.list_begin[a]; i < dv.list_begin[a + 1]; ++i) {
                const int s = dv.list[i];
                if (tip_only && (s >> 1) >= A.n_ts) continue;
                const double v = S.res[3 * (s >> 1) + d];
                acc += (s & 1) ? -v : v;
            }
            if (tip_only) ctl.ft[d] = acc;
            else S.f[q] = acc;
        }
        if (tid == kThreads - 1) {
            double E = 0;
            for (int i = dv.list_begin[1]; i < dv.list_begin[2]; ++i) {
                const int s = dv.list[i] >> 1;
                if (!(tip_only && s >= A.n_ts)) E += S.en[s];
            }
            ctl.e_eval = E;
        }
        if (tid == 0 && !tip_only) my_evals += 1;
        __syncthreads();
    };

    for (;;) {
        __syncthreads();
        if (tid == 0) {
            const unsigned long long t = atomicAdd(&A.ctr->next_work, 1ull);
            ctl.col = (t < (unsigned long long)(A.col_end - A.col_begin)) ? A.col_begin + (int)t : -1;
        }
        __syncthreads();
        const int col = ctl.col;
        if (col < 0) break;
        if (late()) {
            err |= ERR_WATCHDOG;
            break;
        }
        // System min_system = system (simulation.cpp:93): the initial state
        for (int q = tid; q < nq; q += kThreads) {
            S.pos[q] = dv.pos0[q];
            S.vel[q] = 0.0;
            S.fsum[q] = 0.0;
        }
        __syncthreads();
        if (tid == 0) {
            // setDummyXY / setDummyZ (system.cpp:139-162, system.hpp:46-49)
            const int i = col / P.ny, j = col % P.ny;
            double x = i * P.dx, y = j * P.dy;
            if (P.tip_pbc) {
                const double* ci = P.cell_inv;
                const double* c = P.cell;
                const double tx = x - P.offset[0], ty = y - P.offset[1], tz = 0 - P.offset[2];
                double cx = ci[0] * tx + ci[1] * ty + ci[2] * tz;
                double cy = ci[3] * tx + ci[4] * ty + ci[5] * tz;
                const double cz = ci[6] * tx + ci[7] * ty + ci[8] * tz;
                cx -= floor(cx);
                cy -= floor(cy);
                x = (c[0] * cx + c[1] * cy + c[2] * cz) + P.offset[0];
                y = (c[3] * cx + c[4] * cy + c[5] * cz) + P.offset[1];
            }
            S.pos[0] = x; S.pos[1] = y; S.pos[2] = P.zhigh;
            S.pos[3] = x; S.pos[4] = y; S.pos[5] = P.zhigh - P.tip_dummy_d;
            ctl.e_tip = 0.0;   // System::energies_[1], carried between heights
        }
        for (int k = 0; k < P.nz; ++k) {
            // ---- FIREMinimisation / SDMinimisation (minimiser.cpp:39-129) ----
            __syncthreads();
            if (tid == 0) {
                ctl.alpha = 0.1;
                ctl.dt = P.dt;
                ctl.n_non_neg = 0;
            }
            int n = 1;
            for (; n < P.maxsteps; ++n) {
                if ((n & 1023) == 0 && late()) {
                    err |= ERR_WATCHDOG;
                    break;
                }
                double e1 = 0, e2 = 0, e3 = 0;
                evaluate(S.pos, false);
                const double dt = ctl.dt;
                if (P.minimiser == MAFM_MIN_SD) {
                    for (int q = tid; q < nq; q += kThreads) S.fsum[q] = S.f[q];
                } else if (P.integrator == MAFM_INT_EULER) {
                    for (int q = tid; q < nq; q += kThreads) {
                        S.fsum[q] = S.f[q];
                        if (fixed[q / 3] != 1) {
                            S.pos[q] += dt * S.vel[q];
                            S.vel[q] += dt * S.f[q];
                        }
                    }
                } else if (P.integrator == MAFM_INT_MIDPOINT) {
                    for (int q = tid; q < nq; q += kThreads) {
                        double p2 = S.pos[q], v2 = S.vel[q];
                        if (fixed[q / 3] != 1) {
                            p2 += dt / 2 * S.vel[q];
                            v2 += dt / 2 * S.f[q];
                        }
                        S.pe[q] = p2;
                        S.vk[q] = v2;
                    }
                    evaluate(S.pe, false);
                    for (int q = tid; q < nq; q += kThreads) {
                        if (fixed[q / 3] != 1) {
                            S.pos[q] += dt * S.vk[q];
                            S.vel[q] += dt * S.f[q];
                        }
                        S.fsum[q] = S.f[q];
                    }
                } else {   // RK4 (integrators.cpp:56-111)
                    e1 = ctl.e_eval;
                    for (int q = tid; q < nq; q += kThreads) {
                        S.fsum[q] = S.f[q];                 // f1
                        S.vsum[q] = S.vel[q];               // v
                        double p2 = S.pos[q], v2 = S.vel[q];
                        if (fixed[q / 3] != 1) {
                            p2 += dt / 2 * S.vel[q];
                            v2 += dt / 2 * S.f[q];
                        }
                        S.pe[q] = p2;
                        S.vk[q] = v2;
                    }
                    evaluate(S.pe, false);
                    e2 = ctl.e_eval;
                    for (int q = tid; q < nq; q += kThreads) {
                        S.fsum[q] = S.fsum[q] + 2 * S.f[q];
                        S.vsum[q] = S.vsum[q] + 2 * S.vk[q];
                        const double v2 = S.vk[q];
                        double p3 = S.pos[q], v3 = S.vel[q];
                        if (fixed[q / 3] != 1) {
                            p3 += dt / 2 * v2;
                            v3 += dt / 2 * S.f[q];
                        }
                        S.pe[q] = p3;
                        S.vk[q] = v3;
                    }
                    evaluate(S.pe, false);
                    e3 = ctl.e_eval;
                    for (int q = tid; q < nq; q += kThreads) {
                        S.fsum[q] = S.fsum[q] + 2 * S.f[q];
                        S.vsum[q] = S.vsum[q] + 2 * S.vk[q];
                        const double v3 = S.vk[q];
                        double p4 = S.pos[q], v4 = S.vel[q];
                        if (fixed[q / 3] != 1) {
                            p4 += dt * v3;
                            v4 += dt * S.f[q];
                        }
                        S.pe[q] = p4;
                        S.vk[q] = v4;
                    }
                    evaluate(S.pe, false);
                    for (int q = tid; q < nq; q += kThreads) {
                        const double fs = S.fsum[q] + S.f[q];    // f1 + 2f2 + 2f3 + f4
                        const double vs = S.vsum[q] + S.vk[q];   // v + 2v2 + 2v3 + v4
                        if (fixed[q / 3] != 1) {
                            S.pos[q] += dt / 6 * vs;
                            S.vel[q] += dt / 6 * fs;
                        }
                        S.fsum[q] = fs / 6;
                    }
                }
                __syncthreads();
                // beside one another: the convergence test (the last warp), the
                // power P (the last warp but one), the mixing (the others)
                if (warp == kFlexWarps - 1) {
                    if (lane == 0) {
                        // checkConvergence on the tip (minimiser.cpp:15-37)
                        const bool rk4 = P.minimiser != MAFM_MIN_SD && P.integrator == MAFM_INT_RK4;
                        const double e_new = rk4 ? (e1 + 2 * e2 + 2 * e3 + ctl.e_eval) / 6 : ctl.e_eval;
                        const double ediff = e_new - ctl.e_tip;
                        bool conv;
                        if (P.minterm == MAFM_TERM_E) conv = fabs(ediff) < P.etol;
                        else {
                            conv = len3(v3(S.fsum + 3)) < P.ftol;
                            if (P.minterm != MAFM_TERM_F) conv = conv && fabs(ediff) < P.etol;
                        }
                        ctl.e_tip = e_new;
                        ctl.conv = conv;
                    }
                } else if (P.minimiser != MAFM_MIN_SD) {
                    if (warp == kFlexWarps - 2) {
                        // P = sum_i v_i . F_i in atom order
                        for (int a = lane; a < na; a += 32)
                            S.dot[a] = dot3(v3(S.vel + 3 * a), v3(S.fsum + 3 * a));
                        __syncwarp();
                        if (lane == 0) {
                            double pw = 0;
                            for (int a = 0; a < na; ++a) pw += S.dot[a];
                            ctl.pw = pw;
                        }
                    } else {
                        // (1 - alpha) v + alpha F.normalized() |v|  (minimiser.cpp:112-113)
                        const double alpha = ctl.alpha;
                        for (int q = tid; q < nq; q += kThreads - 64) {
                            const int a = q / 3;
                            if (fixed[a] == 1) {
                                S.pe[q] = S.vel[q];
                                continue;
                            }
                            const double lf = len3(v3(S.fsum + 3 * a));
                            const double fh = lf > 1e-10 ? div64(S.fsum[q], lf) : 0.0;
                            S.pe[q] = (1 - alpha) * S.vel[q] + (alpha * fh) * len3(v3(S.vel + 3 * a));
                        }
                    }
                }
                __syncthreads();
                if (ctl.conv) break;
                if (P.minimiser == MAFM_MIN_SD) {
                    for (int q = tid; q < nq; q += kThreads)
                        if (fixed[q / 3] != 1) S.pos[q] += P.dt * S.fsum[q];
                    continue;
                }
                const bool neg = ctl.pw < 0;
                for (int q = tid; q < nq; q += kThreads) S.vel[q] = neg ? 0.0 : S.pe[q];
                if (tid == kThreads - 1) {
                    if (neg) {
                        ctl.n_non_neg = 0;
                        ctl.dt = ctl.dt * 0.5;
                        ctl.alpha = 0.1;
                    } else {
                        if (ctl.n_non_neg > 5) {
                            ctl.dt = fmin(ctl.dt * 1.1, 10 * P.dt);
                            ctl.alpha *= 0.99;
                        }
                        ctl.n_non_neg++;
                    }
                }
            }
            if (err & ERR_WATCHDOG) break;
            // System::getOutput (system.cpp:28-51)
            evaluate(S.pos, true);
            if (tid == 0) {
                const double et = ctl.e_eval;
                const V3 ft = v3(ctl.ft);
                int st = n >= P.maxsteps ? MAFM_PT_MAXSTEPS : 0;
                if (!isfinite(ft.x) || !isfinite(ft.y) || !isfinite(ft.z) || !isfinite(et))
                    st |= MAFM_PT_NONFINITE;
                mafm_point r;
                r.tip[0] = S.pos[3]; r.tip[1] = S.pos[4]; r.tip[2] = S.pos[5];
                r.force[0] = ft.x; r.force[1] = ft.y; r.force[2] = ft.z;
                r.energy = et;
                r.steps = n;
                r.status = st;
                A.out[(size_t)(col - A.col_begin) * P.nz + k] = r;
                my_steps += (unsigned long long)n;
            }
            if (A.states && col == A.state_column)
                for (int q = tid; q < nq; q += kThreads) A.states[(size_t)k * nq + q] = S.pos[q];
            __syncthreads();
            // System::lowerTip (system.hpp:51-54)
            if (tid == 0) {
                S.pos[2] -= P.dz;
                S.pos[5] -= P.dz;
            }
            // the time limit once per height too: a height usually converges in
            // far fewer than the 1024 steps between the checks above
            if (late()) {
                err |= ERR_WATCHDOG;
                break;
            }
        }
        if (err & ERR_WATCHDOG) break;
    }
    if (tid == 0) {
        atomicAdd(&A.ctr->total_steps, my_steps);
        atomicAdd(&A.ctr->force_evals, my_evals);
        if (err) atomicOr(&A.ctr->error_word, err);
    }
}

}  // namespace
}  // namespace mafm

using namespace mafm;

extern "C" int mafm_flex_create(int device, const mafm_scan_desc* d, const mafm_flex_desc* f,
                                mafm_flex** out) {
    return guarded([&] {
        if (!d || !f || !out) fail(MAFM_E_INVALID, "null argument");
        *out = nullptr;
        if (!d->flexible) fail(MAFM_E_INVALID, "the descriptor is not a flexible molecule");
        if (d->rigidgrid || d->use_external_potential)
            fail(MAFM_E_UNSUPPORTED, "flexible molecules run with pair and Coulomb terms only");
        if (d->n_atoms < 1 || !d->pos || !d->type || !d->tip_pair || !f->fixed)
            fail(MAFM_E_INVALID, "flexible descriptor without atoms");
        if (d->n_atoms + 2 > 1024) fail(MAFM_E_RANGE, "flexible molecules of up to 1022 atoms");
        if (device >= 0) cuda_check(cudaSetDevice(device), "cudaSetDevice");
        auto* s = new mafm_flex();
        try {
            cuda_check(cudaGetDevice(&s->device), "cudaGetDevice");
            s->d = *d;
            const int ns = d->n_atoms, na = ns + 2;
            s->n_sys = na;
            // scan parameters shared with the rigid kernels
            ScanParams& P = s->P;
            P.td_kind = d->dummy_pair.kind;
            for (int k = 0; k < 3; ++k) P.td_p[k] = d->dummy_pair.p[k];
            P.td_coul = d->tip_dummy_coulomb && d->dummy_charge != 0 && d->tip_charge != 0;
            P.td_qq = P.td_coul ? d->qbase * d->dummy_charge * d->tip_charge : 0.0;
            P.harm_k = d->harm_k;
            P.harm_r0 = d->harm_r0;
            P.tip_dummy_d = d->tip_dummy_d;
            P.nx = d->nx; P.ny = d->ny; P.nz = d->nz;
            P.tip_pbc = d->tip_pbc;
            P.dx = d->dx; P.dy = d->dy; P.dz = d->dz; P.zhigh = d->zhigh;
            std::memcpy(P.cell, d->cell, sizeof P.cell);
            if (d->tip_pbc) {
                // the inverse in the reference's order (matrices.hpp:117-133)
                const double* m = d->cell;
                const double a = m[0], b = m[1], c = m[2], dd = m[3], e = m[4], ff = m[5], g = m[6],
                             h = m[7], ii = m[8];
                double det = a * (e * ii - ff * h);
                det += b * (ff * g - dd * ii);
                det += c * (dd * h - e * g);
                const double id = 1 / det;
                const double inv[9] = {id * (e * ii - ff * h), -id * (b * ii - c * h), id * (b * ff - c * e),
                                       -id * (dd * ii - ff * g), id * (a * ii - c * g), -id * (a * ff - c * dd),
                                       id * (dd * h - e * g), -id * (a * h - b * g), id * (a * e - b * dd)};
                std::memcpy(P.cell_inv, inv, sizeof inv);
            }
            std::memcpy(P.offset, d->offset, sizeof P.offset);
            P.minimiser = d->minimiser;
            P.integrator = d->integrator;
            P.minterm = d->minterm;
            P.maxsteps = d->maxsteps;
            P.etol = d->etol; P.ftol = d->ftol; P.dt = d->dt;

            // ---- host-side lists, in the reference's interaction order ----
            std::vector<double> pos0(3 * (size_t)na, 0.0);
            for (int a = 0; a < ns; ++a)
                for (int k = 0; k < 3; ++k) pos0[3 * (size_t)(a + 2) + k] = d->pos[3 * (size_t)a + k];
            std::vector<int> fixed(na, 0);
            fixed[0] = 1;
            for (int a = 0; a < ns; ++a) fixed[a + 2] = f->fixed[a];
            struct Entry { int kind, role, idx; };
            std::vector<std::vector<Entry>> lists(na);
            std::vector<std::vector<int>> tasks(FT_XY + 1);   // interactions of every kind
            auto add = [&](int atom, int kind, int role, int idx) {
                lists[atom].push_back({kind, role, idx});
                if (tasks[kind].empty() || tasks[kind].back() != idx) tasks[kind].push_back(idx);
            };
            std::vector<FlexTS> ts;
            // buildTipSurfaceInteractions (simulation.cpp:297-320)
            const int images = d->vdw_pbc ? 9 : 1;
            for (int im = 0; im < 9; ++im) {
                const int ia = im / 3 - 1, ib = im % 3 - 1;
                if (images == 1 && (ia != 0 || ib != 0)) continue;
                double sh[3] = {0, 0, 0};
                if (d->vdw_pbc)
                    for (int k = 0; k < 3; ++k) sh[k] = ia * d->cell[3 * k] + ib * d->cell[3 * k + 1];
                for (int a = 0; a < ns; ++a) {
                    const mafm_pair& pr = d->tip_pair[d->type[a]];
                    FlexTS t{};
                    t.atom = a + 2;
                    t.kind = pr.kind;
                    for (int k = 0; k < 3; ++k) { t.shift[k] = sh[k]; t.p[k] = pr.p[k]; }
                    ts.push_back(t);
                    add(1, FT_TS_VDW, 0, (int)ts.size() - 1);
                    add(a + 2, FT_TS_VDW, 1, (int)ts.size() - 1);
                    if (!d->vdw_pbc && d->coulomb && d->tip_charge != 0 && d->charge[a] != 0) {
                        FlexTS c{};
                        c.atom = a + 2;
                        c.coul = 1;
                        c.qq = d->qbase * d->tip_charge * d->charge[a];
                        ts.push_back(c);
                        add(1, FT_TS_COUL, 0, (int)ts.size() - 1);
                        add(a + 2, FT_TS_COUL, 1, (int)ts.size() - 1);
                    }
                }
            }
            // buildTipDummyInteractions (simulation.cpp:503-515)
            add(0, FT_TD_VDW, 0, 0);
            add(1, FT_TD_VDW, 1, 0);
            if (P.td_coul) {
                add(0, FT_TD_COUL, 0, 0);
                add(1, FT_TD_COUL, 1, 0);
            }
            add(0, FT_TD_HARM, 0, 0);
            add(1, FT_TD_HARM, 1, 0);
            // buildSurfaceSurfaceInteractions (simulation.cpp:557-693): bonds,
            // angles, dihedrals, then the non-bonded pairs
            std::vector<int> bonds, angles, dihedrals, pairs;
            for (int b = 0; b < f->n_bonds; ++b) {
                const int i = f->bond_atoms[2 * b] + 2, j = f->bond_atoms[2 * b + 1] + 2;
                bonds.insert(bonds.end(), {i, j});
            }
            for (int g = 0; g < f->n_angles; ++g)
                for (int k = 0; k < 3; ++k) angles.push_back(f->angle_atoms[3 * g + k] + 2);
            for (int g = 0; g < f->n_dihedrals; ++g)
                for (int k = 0; k < 4; ++k) dihedrals.push_back(f->dihedral_atoms[4 * g + k] + 2);
            std::vector<FlexPair> pp;
            for (int q = 0; q < f->n_pairs; ++q) {
                pairs.insert(pairs.end(), {f->pair_atoms[2 * q] + 2, f->pair_atoms[2 * q + 1] + 2});
                FlexPair x{};
                x.kind = f->pair_vdw[q].kind;
                for (int k = 0; k < 3; ++k) x.p[k] = f->pair_vdw[q].p[k];
                pp.push_back(x);
            }
            for (int a : bonds)
                if (a < 2 || a >= na) fail(MAFM_E_INVALID, "bond atom out of range");
            for (int a : angles)
                if (a < 2 || a >= na) fail(MAFM_E_INVALID, "angle atom out of range");
            for (int a : dihedrals)
                if (a < 2 || a >= na) fail(MAFM_E_INVALID, "dihedral atom out of range");
            for (int a : pairs)
                if (a < 2 || a >= na) fail(MAFM_E_INVALID, "pair atom out of range");
            for (int b = 0; b < f->n_bonds; ++b) {
                add(bonds[2 * b], FT_BOND, 0, b);
                add(bonds[2 * b + 1], FT_BOND, 1, b);
            }
            for (int g = 0; g < f->n_angles; ++g) {
                add(angles[3 * g + 1], FT_ANGLE, 1, g);
                add(angles[3 * g + 2], FT_ANGLE, 2, g);
                add(angles[3 * g], FT_ANGLE, 0, g);
            }
            for (int g = 0; g < f->n_dihedrals; ++g)
                for (int r = 0; r < 4; ++r) add(dihedrals[4 * g + r], FT_DIHEDRAL, r, g);
            std::vector<FlexCoul> coul;
            for (int q = 0; q < f->n_pairs; ++q) {
                add(pairs[2 * q], FT_PAIR_VDW, 0, q);
                add(pairs[2 * q + 1], FT_PAIR_VDW, 1, q);
                if (f->pair_qq && f->pair_qq[q] != 0) {
                    const int c = (int)coul.size();
                    coul.push_back({pairs[2 * q], pairs[2 * q + 1], f->pair_qq[q]});
                    add(pairs[2 * q], FT_PAIR_COUL, 0, c);
                    add(pairs[2 * q + 1], FT_PAIR_COUL, 1, c);
                }
            }
            // buildSubstrateInteractions (simulation.cpp:516-528)
            const double eps = f->substrate[0], sig = f->substrate[1], lambda = f->substrate[2],
                         rc = f->substrate[3];
            const double kPi = 3.14159265358979323846;
            s->sub[0] = 2 * kPi * eps * pow(sig / lambda, 2);
            s->sub[1] = (kPi / (lambda * lambda)) * 4 * eps * (pow(sig / rc, 12) - pow(sig / rc, 6));
            s->sub[2] = s->sub[0] * ((12. / 5) * pow(sig / rc, 10) - 3 * pow(sig / rc, 4));
            s->sub[3] = -sig;
            s->sub[4] = rc;
            s->sub[5] = sig;
            s->sub_k = f->substrate[4];
            std::vector<double> xy;
            for (int a = 2; a < na; ++a) {
                add(a, FT_SUBSTRATE, 0, a);
                if (fixed[a] == 2) {
                    xy.insert(xy.end(), {(double)a, pos0[3 * (size_t)a], pos0[3 * (size_t)a + 1]});
                    add(a, FT_XY, 0, (int)xy.size() / 3 - 1);
                }
            }
            // force slots, kind after kind: the tip's terms first (both kinds of
            // tip–surface terms index one list)
            const int n_ts = (int)ts.size();
            const int count[12] = {0, n_ts, 1, 1, 1, f->n_bonds, f->n_angles, f->n_dihedrals,
                                   f->n_pairs, (int)coul.size(), na, (int)xy.size() / 3};
            int slots = 0;
            for (int kd = FT_TS_VDW; kd <= FT_XY; ++kd) {
                s->dv.slot_base[kd] = slots;
                slots += count[kd] * flex_slots(kd);
                if (kd == FT_TD_HARM) s->dv.n_energies = slots;
            }
            s->n_slots = slots;
            // every atom's slots in the reference's order: a pair's second atom
            // (role 1; of the dummy's terms the tip, of an angle the shared atom,
            // role 0) takes the negative
            std::vector<int> begin(na + 1, 0), list;
            for (int a = 0; a < na; ++a) {
                begin[a] = (int)list.size();
                for (const Entry& e : lists[a]) {
                    const int first = s->dv.slot_base[e.kind] + e.idx * flex_slots(e.kind);
                    if (e.kind == FT_ANGLE) list.push_back(e.role == 0 ? (first + 2) << 1 | 1 : (first + e.role - 1) << 1);
                    else if (e.kind == FT_DIHEDRAL) list.push_back((first + e.role) << 1);
                    else list.push_back(first << 1 | (e.role == 1));
                }
            }
            begin[na] = (int)list.size();
            // chunks of up to 32 interactions of one kind, the costliest first,
            // each to the warp with the least to do (costs: FP64 instructions)
            const int cost[12] = {48, 30, 50, 30, 25, 32, 180, 220, 48, 30, 35, 18};
            std::vector<std::pair<int, int>> chunks;   // kind, first task
            for (int kd = FT_TS_VDW; kd <= FT_XY; ++kd)
                for (size_t i = 0; i < tasks[kd].size(); i += 32) chunks.push_back({kd, (int)i});
            std::stable_sort(chunks.begin(), chunks.end(),
                             [&](const auto& x, const auto& y) { return cost[x.first] > cost[y.first]; });
            std::vector<std::vector<std::pair<int, int>>> of_warp(kFlexWarps);
            std::vector<long long> load(kFlexWarps, 0);
            for (const auto& c : chunks) {
                const size_t w = std::min_element(load.begin(), load.end()) - load.begin();
                of_warp[w].push_back(c);
                load[w] += cost[c.first];
            }
            std::vector<int> warp_begin(1, 0), chunk_kind, task;
            for (const auto& w : of_warp) {
                for (const auto& c : w) {
                    chunk_kind.push_back(c.first);
                    for (size_t i = c.second; i < (size_t)c.second + 32; ++i)
                        task.push_back(i < tasks[c.first].size() ? tasks[c.first][i] : -1);
                }
                warp_begin.push_back((int)chunk_kind.size());
            }
            s->n_ts = n_ts;

            // one device block for every array (256-byte aligned pieces)
            struct Piece { const void* src; size_t bytes; size_t off; };
            std::vector<Piece> pieces;
            size_t off = 0;
            auto piece = [&](const void* src, size_t bytes) {
                pieces.push_back({src, bytes, off});
                const size_t at = off;
                off += (bytes + 255) & ~(size_t)255;
                return at;
            };
            const size_t o_pos = piece(pos0.data(), pos0.size() * sizeof(double));
            const size_t o_fixed = piece(fixed.data(), fixed.size() * sizeof(int));
            const size_t o_ts = piece(ts.data(), ts.size() * sizeof(FlexTS));
            const size_t o_b = piece(bonds.data(), bonds.size() * sizeof(int));
            const size_t o_bp = piece(f->bond_param, (size_t)f->n_bonds * 2 * sizeof(double));
            const size_t o_a = piece(angles.data(), angles.size() * sizeof(int));
            const size_t o_ap = piece(f->angle_param, (size_t)f->n_angles * 2 * sizeof(double));
            const size_t o_dh = piece(dihedrals.data(), dihedrals.size() * sizeof(int));
            const size_t o_dp = piece(f->dihedral_param, (size_t)f->n_dihedrals * 2 * sizeof(double));
            const size_t o_pr = piece(pairs.data(), pairs.size() * sizeof(int));
            const size_t o_pp = piece(pp.data(), pp.size() * sizeof(FlexPair));
            const size_t o_cp = piece(coul.data(), coul.size() * sizeof(FlexCoul));
            const size_t o_xy = piece(xy.data(), xy.size() * sizeof(double));
            const size_t o_lb = piece(begin.data(), begin.size() * sizeof(int));
            const size_t o_l = piece(list.data(), list.size() * sizeof(int));
            const size_t o_wb = piece(warp_begin.data(), warp_begin.size() * sizeof(int));
            const size_t o_ck = piece(chunk_kind.data(), chunk_kind.size() * sizeof(int));
            const size_t o_tk = piece(task.data(), task.size() * sizeof(int));
            s->block_bytes = std::max<size_t>(off, 256);
            cuda_check(cudaMalloc(&s->dev_block, s->block_bytes), "cudaMalloc");
            char* dev = static_cast<char*>(s->dev_block);
            for (const Piece& p : pieces)
                if (p.bytes)
                    cuda_check(cudaMemcpy(dev + p.off, p.src, p.bytes, cudaMemcpyHostToDevice), "upload");
            s->dv.pos0 = reinterpret_cast<const double*>(dev + o_pos);
            s->dv.fixed = reinterpret_cast<const int*>(dev + o_fixed);
            s->dv.ts = dev + o_ts;
            s->dv.bonds = reinterpret_cast<const int*>(dev + o_b);
            s->dv.bond_par = reinterpret_cast<const double*>(dev + o_bp);
            s->dv.angles = reinterpret_cast<const int*>(dev + o_a);
            s->dv.angle_par = reinterpret_cast<const double*>(dev + o_ap);
            s->dv.dihedrals = reinterpret_cast<const int*>(dev + o_dh);
            s->dv.dihedral_par = reinterpret_cast<const double*>(dev + o_dp);
            s->dv.pairs = reinterpret_cast<const int*>(dev + o_pr);
            s->dv.pair_par = dev + o_pp;
            s->dv.coul = dev + o_cp;
            s->dv.xy = reinterpret_cast<const double*>(dev + o_xy);
            s->dv.list_begin = reinterpret_cast<const int*>(dev + o_lb);
            s->dv.list = reinterpret_cast<const int*>(dev + o_l);
            s->dv.warp_begin = reinterpret_cast<const int*>(dev + o_wb);
            s->dv.chunk_kind = reinterpret_cast<const int*>(dev + o_ck);
            s->dv.task = reinterpret_cast<const int*>(dev + o_tk);
            cuda_check(cudaMalloc(&s->ctr, sizeof(RunCounters)), "cudaMalloc");
            cuda_check(cudaMallocHost(&s->host_ctr, sizeof(RunCounters)), "cudaMallocHost");
        } catch (...) {
            if (s->dev_block) cudaFree(s->dev_block);
            if (s->ctr) cudaFree(s->ctr);
            if (s->host_ctr) cudaFreeHost(s->host_ctr);
            delete s;
            throw;
        }
        *out = s;
    });
}

extern "C" int mafm_flex_destroy(mafm_flex* s) {
    if (s) {
        cudaSetDevice(s->device);
        if (s->dev_block) cudaFree(s->dev_block);
        if (s->ctr) cudaFree(s->ctr);
        if (s->host_ctr) cudaFreeHost(s->host_ctr);
        delete s;
    }
    return MAFM_OK;
}

extern "C" int mafm_flex_run(mafm_flex* s, int32_t col_begin, int32_t col_end, mafm_point* out,
                             mafm_run_stats* stats, int32_t state_column, double* states,
                             void* stream) {
    return guarded([&] {
        if (!s || !out) fail(MAFM_E_INVALID, "null argument");
        cuda_check(cudaSetDevice(s->device), "cudaSetDevice");
        const int n_cols = s->d.nx * s->d.ny;
        if (col_begin == 0 && col_end == 0) col_end = n_cols;
        if (col_begin < 0 || col_end > n_cols || col_begin > col_end)
            fail(MAFM_E_INVALID, "column range [%d, %d) outside [0, %d)", col_begin, col_end, n_cols);
        const size_t n_pts = (size_t)(col_end - col_begin) * s->d.nz;
        cudaStream_t st = (cudaStream_t)stream;
        // outputs: device or pinned memory directly, pageable through a copy
        mafm_point* dout = out;
        double* dstates = states;
        void* tmp_out = nullptr;
        void* tmp_states = nullptr;
        const size_t states_bytes = (size_t)s->d.nz * s->n_sys * 3 * sizeof(double);
        auto device_view = [](void* p) -> void* {
            cudaPointerAttributes a{};
            if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
                cudaGetLastError();
                return nullptr;
            }
            if (a.type == cudaMemoryTypeDevice || a.type == cudaMemoryTypeManaged) return p;
            if (a.type == cudaMemoryTypeHost) return a.devicePointer;
            return nullptr;
        };
        struct Frees {
            void* a = nullptr;
            void* b = nullptr;
            double* scratch = nullptr;
            ~Frees() {
                if (a) cudaFree(a);
                if (b) cudaFree(b);
                if (scratch) cudaFree(scratch);
            }
        } frees;
        if (void* v = device_view(out)) {
            dout = static_cast<mafm_point*>(v);
        } else {
            cuda_check(cudaMalloc(&tmp_out, n_pts * sizeof(mafm_point)), "cudaMalloc");
            frees.a = tmp_out;
            dout = static_cast<mafm_point*>(tmp_out);
        }
        if (states) {
            if (void* v = device_view(states)) {
                dstates = static_cast<double*>(v);
            } else {
                cuda_check(cudaMalloc(&tmp_states, states_bytes), "cudaMalloc");
                frees.b = tmp_states;
                dstates = static_cast<double*>(tmp_states);
                cuda_check(cudaMemsetAsync(tmp_states, 0, states_bytes, st), "memset states");
            }
        }
        FlexKernelArgs A{};
        A.dv = s->dv;
        A.P = s->P;
        std::memcpy(A.sub, s->sub, sizeof A.sub);
        A.sub_k = s->sub_k;
        A.n_sys = s->n_sys;
        A.n_ts = s->n_ts;
        A.n_slots = s->n_slots;
        A.col_begin = col_begin;
        A.col_end = col_end;
        A.out = dout;
        A.state_column = state_column;
        A.states = dstates;
        A.watchdog_ns = watchdog_ns_from_env();
        A.ctr = s->ctr;
        cuda_check(cudaMemsetAsync(s->ctr, 0, sizeof(RunCounters), st), "reset counters");
        // the atoms' arrays and v.F; the tip's energies and the force slots
        // while they fit (about 8,000 slots), else in global memory
        const size_t atom_bytes = (size_t)22 * s->n_sys * sizeof(double);
        const size_t block_doubles = (size_t)s->dv.n_energies + 3 * (size_t)s->n_slots;
        const bool in_smem = atom_bytes + block_doubles * sizeof(double) <= 200u * 1024u;
        const size_t smem = atom_bytes + (in_smem ? block_doubles * sizeof(double) : 0);
        cuda_check(cudaFuncSetAttribute(flex_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem),
                   "flex smem");
        int per_sm = 0;
        cuda_check(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, flex_kernel, 32 * kFlexWarps, smem),
                   "flex occupancy");
        const int cols = col_end - col_begin;
        int blocks = std::max(1, std::min(cols, sm_count() * (in_smem ? std::max(per_sm, 1) : 1)));
        if (!in_smem) {
            // Slots of this call, 24 B each and a set per block: 12 MB a block (25 MB
            // with charges) for the 520,000 pairs of 1,022 atoms in small fragments.
            // They are given back when the call ends, and where they do not fit
            // fewer blocks take the columns.
            cudaError_t e;
            while ((e = cudaMalloc(&frees.scratch, blocks * block_doubles * sizeof(double))) ==
                       cudaErrorMemoryAllocation && blocks > 1) {
                cudaGetLastError();
                blocks /= 2;
            }
            cuda_check(e, "cudaMalloc");
        }
        A.scratch = frees.scratch;
        if (cols > 0) {
            flex_kernel<<<blocks, 32 * kFlexWarps, smem, st>>>(A);
            cuda_check(cudaGetLastError(), "flex launch");
        }
        if (tmp_out)
            cuda_check(cudaMemcpyAsync(out, tmp_out, n_pts * sizeof(mafm_point), cudaMemcpyDeviceToHost, st),
                       "copy points");
        if (tmp_states)
            cuda_check(cudaMemcpyAsync(states, tmp_states, states_bytes, cudaMemcpyDeviceToHost, st),
                       "copy states");
        cuda_check(cudaMemcpyAsync(s->host_ctr, s->ctr, sizeof(RunCounters), cudaMemcpyDeviceToHost, st),
                   "counters");
        cuda_check(cudaStreamSynchronize(st), "flex relax");
        const RunCounters c = *s->host_ctr;
        if (stats) {
            *stats = mafm_run_stats{};
            stats->total_steps = c.total_steps;
            stats->force_evals = c.force_evals;
            stats->error_word = c.error_word;
        }
        if (c.error_word & ERR_WATCHDOG)
            fail(MAFM_E_DEVICE, "the flexible relaxation exceeded its time limit (MAFM_WATCHDOG_S)");
    });
}
