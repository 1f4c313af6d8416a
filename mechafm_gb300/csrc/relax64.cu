// relax64.cu — the plain FP64 GPU path (precision MAFM_FP64).
//
// A group of 4 to 32 lanes of a warp per pixel column (one thread where columns
// are many and terms few), columns handed out by a global atomic counter.  Every
// floating-point expression keeps the reference's operation order and this
// translation unit is compiled with -fmad=false, so no a*b+c is fused:
// with LJ and Coulomb terms the results are bit-identical to the reference's
// x86-64 build (division and square root are correctly rounded in both; exp
// in the Morse term may differ in the last bit).
//
// Reference correspondence (src/):
//   vdW / Coulomb terms        interactions.cpp:15-51
//   tip–dummy terms            interactions.cpp:252-266, simulation.cpp:503-515
//   trilinear grid lookup      force_grid.cpp:88-275
//   integrators                integrators.cpp:8-111
//   FIRE / SD / convergence    minimiser.cpp:15-129
//   pixel column, z descent    simulation.cpp:93-122, system.cpp:28-51, 139-162
//   rigid grid build           simulation.cpp:420-501
#include <algorithm>
#include <climits>

#include "relax64_dev.cuh"

namespace mafm {
namespace {

// Stage the terms into shared memory when they fit.
__device__ const AtomRec64* stage64(const ScanParams& p, AtomRec64* sm, int cap) {
    if (p.n_terms_direct <= cap) {
        for (int i = threadIdx.x; i < p.n_terms_direct; i += blockDim.x) sm[i] = p.atoms64[i];
        __syncthreads();
        return sm;
    }
    return p.atoms64;
}

// ---- the relaxation: G lanes a column ------------------------------------------

// One component of a trilinear lookup (ForceGrid::interpolate, interp64's
// expressions): lane component c (0-2 force, 3 energy) of a quad, position
// component q_c on lane c.
__device__ double interp64_quad(const GridView& g, double pos, int c, int quad, int& outside,
                                unsigned& err) {
    const int a = min(c, 2);
    const double q = pos - g.origin[a];
    double pb;
    if (g.orthogonal) {
        pb = quo64(q, g.basis[4 * a]);
    } else {
        const double qx = __shfl_sync(0xffffffffu, q, quad), qy = __shfl_sync(0xffffffffu, q, quad + 1),
                     qz = __shfl_sync(0xffffffffu, q, quad + 2);
        pb = g.inv[3 * a] * qx + g.inv[3 * a + 1] * qy + g.inv[3 * a + 2] * qz;
    }
    int gp = (int)floor(pb);
    if (!g.periodic && c < 3) {
        if (gp < 0) { gp = 0; outside = 1; }
        else if (gp >= g.n[a]) { gp = g.n[a] - 1; outside = 1; }
    }
    const double d = pb - gp;
    const int gx = __shfl_sync(0xffffffffu, gp, quad), gy = __shfl_sync(0xffffffffu, gp, quad + 1),
              gz = __shfl_sync(0xffffffffu, gp, quad + 2);
    const double dx = __shfl_sync(0xffffffffu, d, quad), dy = __shfl_sync(0xffffffffu, d, quad + 1),
                 dz = __shfl_sync(0xffffffffu, d, quad + 2);
    double s[8];
#pragma unroll
    for (int m = 0; m < 8; ++m)
        s[m] = reinterpret_cast<const double*>(
            g.g64 + grid_index64(g, gx + (m >> 2), gy + ((m >> 1) & 1), gz + (m & 1), err))[c];
    const double v00 = s[0] * (1 - dx) + s[4] * dx;
    const double v01 = s[1] * (1 - dx) + s[5] * dx;
    const double v10 = s[2] * (1 - dx) + s[6] * dx;
    const double v11 = s[3] * (1 - dx) + s[7] * dx;
    const double v0 = v00 * (1 - dy) + v10 * dy;
    const double v1 = v01 * (1 - dy) + v11 * dy;
    return v0 * (1 - dz) + v1 * dz;
}

// Force records a group's buffer holds: two rounds of its lanes, each with a
// van der Waals and a Coulomb record, and 32 B so that the groups of a warp
// read different banks.
template <int G>
constexpr int kGroupBuf = 2 * (2 * G) + 1;
// Terms of one pass of a block of several warps (both records of each).
constexpr int kWideTerms = 128;

// Term j of a scan for the separation tip - (its position); term n: the
// tip–dummy term.  With tip - dummy for the reference's dummy - tip every force
// component of it has the opposite sign, so it is added.
__device__ __forceinline__ AtomRec64 term64(const ScanParams& p, int j, int n, V3 dum) {
    if (j < n) return p.atoms64[j];
    AtomRec64 t;
    t.x = dum.x; t.y = dum.y; t.z = dum.z;
    t.qq = p.td_qq;
    t.p0 = p.td_p[0]; t.p1 = p.td_p[1]; t.p2 = p.td_p[2];
    t.kind = p.td_kind;
    t.coul = p.td_coul;
    return t;
}

// The XY spring (add_tip_dummy): what is added to component c.
__device__ __forceinline__ double spring64(const ScanParams& p, V3 tip, V3 dum, int c) {
    const double rx = dum.x - tip.x, ry = dum.y - tip.y;
    const double rr = root64(rx * rx + ry * ry);
    const double dr = rr - p.harm_r0;
    double add = -0.0;                      // no z force
    if (c == 3) {
        add = p.harm_k * dr * dr;
    } else if (c < 2 && rr > 1e-10) {
        const double s = quo64(-2 * p.harm_k * dr, rr);
        add = -(s * (c == 0 ? rx : ry));
    }
    return add;
}

// One column, or the list's next one, on G lanes (4, 8, 16 or 32) of a warp; one
// warp a block.  An FP64 instruction of a warp takes 64 cycles whatever its
// lanes do and an SM starts one every 19, so FP64 instructions are what the
// kernel counts: lane l of a group computes terms l, l + G, ... into the group's
// buffer, the tip–dummy term as one more, then lane c of every quad adds
// component c (x, y, z, E) of the records in the reference's order, and keeps
// component c of the tip's state through the integrator and FIRE.  Every sum and
// expression is formed as in Eval64 and fire_t / sd_t: the same bits.
//
// All groups of a warp take a minimiser step together (as many evaluations as
// the integrator has; a group that writes a height's record does so in the
// first one), so no group waits in another's branch; a group whose column is
// done takes the next one.
//
// W = 4 (G = 32): a block of four warps holds one column, for calls of so few
// columns that the length of an evaluation is what counts.  The first warp runs
// the minimiser and the sums; all four compute the terms, van der Waals and
// Coulomb records on different warps, the last one the spring.
//
// 51 x 51 x 11 graphene (2,601 columns, G = 8): 178 -> 26 ms; one thread per
// column used 21 of the 152 SMs there, and kept half of its lanes waiting.  301
// columns of the 60-atom cluster x 41 (W = 4): 255 -> 131 ms; one warp per
// column took 219 ms.
template <int G, int W>
__global__ void __launch_bounds__(32 * W) relax64_kernel(const __grid_constant__ ScanParams p, mafm_point* out,
                                                     RunCounters* ctr, const int* list, int col_begin,
                                                     long long n_cols, int pairs_per_eval, bool by_column) {
    constexpr unsigned kAll = 0xffffffffu;
    __shared__ __align__(32) Node64 buf_all[W == 1 ? (32 / G) * kGroupBuf<G> : 2 * kWideTerms];
    __shared__ double wide_pos[6], wide_spring[4];
    __shared__ int wide_quit;
    const int lane = threadIdx.x & 31;
    const int sub = lane & (G - 1), grp = lane / G;
    const int c = lane & 3, quad = lane & ~3;
    const int va = min(c, 2);              // the vector component of the lane's state
    Node64* buf = buf_all + grp * kGroupBuf<G>;
    const bool writer = sub < 4;           // the group's first quad writes its records
    const int n = p.ts_mode == 2 ? 0 : p.n_terms_direct;
    const bool coul_records = p.has_coulomb || p.td_coul;

    // W > 1: the block's records of terms base .. base + kWideTerms - 1 (up to n),
    // and with the first of them the spring
    auto wide_terms = [&](int base) {
        const int warp = threadIdx.x >> 5;
        const V3 tip = {wide_pos[0], wide_pos[1], wide_pos[2]}, dum = {wide_pos[3], wide_pos[4], wide_pos[5]};
        const int chunks = (min(kWideTerms, n + 1 - base) + 31) / 32;
        for (int q = warp; q < (coul_records ? 2 : 1) * chunks; q += W) {
            const int j = base + 32 * (coul_records ? q >> 1 : q) + lane;
            if (j > n) continue;
            const AtomRec64 t = term64(p, j, n, dum);
            const V3 r = {tip.x - t.x, tip.y - t.y, tip.z - t.z};
            V3 f = {0, 0, 0};
            double e = 0;
            const int part = coul_records ? q & 1 : 0;
            if (part == 0) vdw64(t.kind, t.p0, t.p1, t.p2, r, f, e);
            else if (t.coul) coul64(t.qq, r, f, e);
            buf_all[2 * (j - base) + part] = Node64{f.x, f.y, f.z, e};
        }
        if (base == 0 && warp == W - 1 && lane < 4) wide_spring[lane] = spring64(p, tip, dum, lane);
    };
    if (W > 1 && threadIdx.x >= 32) {
        for (;;) {
            __syncthreads();
            if (wide_quit) return;
            for (int base = 0;; base += kWideTerms) {
                if (base) __syncthreads();
                wide_terms(base);
                __syncthreads();
                if (n < base + kWideTerms) break;
            }
        }
    }

    long long w = -1;                      // work index of the group's column, -1: none
    bool done = false;
    double pp = 0, v = 0, u = 0, dm = 0, ex = 0;   // tip, velocity, v2 / v_k, dummy, evaluation position
    double fs = 0, vs = 0, es = 0;         // RK4 sums
    double energy = 0, alpha = 0, dt = 0;
    int k = 0, nst = 0, nnn = 0, outside = 0;
    bool writing = false;                  // the next evaluation is the height's record
    mafm_point* o = nullptr;
    unsigned err = 0, status_or = 0;
    long long steps = 0;
    unsigned long long evals = 0;

    auto bc = [&](double x, int m) { return __shfl_sync(kAll, x, quad + m); };
    // x . y over the quad's components, in vectors.hpp's order
    auto dot = [&](double x, double y) {
        const double s = x * y;
        return bc(s, 0) + bc(s, 1) + bc(s, 2);
    };

    // Force component c (c < 3) or energy (c = 3) at ex; with the tip–dummy terms
    // unless the group writes.  live: the group makes this evaluation (the others
    // of the warp go along; nothing of theirs is kept).
    auto evaluate = [&](bool live) {
        const V3 tip = {bc(ex, 0), bc(ex, 1), bc(ex, 2)};
        const V3 dum = {bc(dm, 0), bc(dm, 1), bc(dm, 2)};
        double acc = 0;
        int base = 0;
        constexpr int kPass = W == 1 ? 2 * G : kWideTerms;
        if (W > 1) {
            if (lane < 3) {
                wide_pos[lane] = ex;
                wide_pos[3 + lane] = dm;
            }
            if (lane == 0) wide_quit = 0;
        }
        for (;; base += kPass) {
            if (W > 1) {
                __syncthreads();
                wide_terms(base);
                __syncthreads();
            } else {
#pragma unroll 1
                for (int j = base + sub; j < base + kPass; j += G) {
                    if (j > n) break;
                    const AtomRec64 t = term64(p, j, n, dum);
                    const V3 r = {tip.x - t.x, tip.y - t.y, tip.z - t.z};
                    V3 f;
                    double e;
                    Node64* b = buf + 2 * (j - base);
                    vdw64(t.kind, t.p0, t.p1, t.p2, r, f, e);
                    b[0] = Node64{f.x, f.y, f.z, e};
                    if (coul_records) {
                        if (t.coul) coul64(t.qq, r, f, e);
                        // a term without Coulomb adds an exact +0: a sum that
                        // starts at +0 is left as it is
                        b[1] = t.coul ? Node64{f.x, f.y, f.z, e} : Node64{0.0, 0.0, 0.0, 0.0};
                    }
                }
                __syncwarp();
            }
            const double* b = reinterpret_cast<const double*>(buf) + c;
            const int cnt = (coul_records ? 2 : 1) * min(kPass, n - base), step = coul_records ? 4 : 8;
            int j = 0;
            for (; j + 8 <= cnt; j += 8) {   // loads ahead of the chain of additions
                double x[8];
#pragma unroll
                for (int m = 0; m < 8; ++m) x[m] = b[step * (j + m)];
#pragma unroll
                for (int m = 0; m < 8; ++m) acc += x[m];
            }
            for (; j < cnt; ++j) acc += b[step * j];
            if (n < base + kPass) break;
            if (W == 1) __syncwarp();
        }
        // the term sum is complete; the field, then the tip–dummy records
        int clamped = 0;
        unsigned bad = 0;
        if (p.ts_mode == 1) acc += interp64_quad(p.es, ex, c, quad, clamped, bad);
        if (p.ts_mode == 2) acc += interp64_quad(p.grid, ex, c, quad, clamped, bad);
        if (live) {
            outside |= p.ts_mode == 2 ? clamped : 0;
            err |= bad;
        }
        const double* td = reinterpret_cast<const double*>(buf + 2 * (n - base)) + c;
        const double with_td = acc + td[0];
        const double with_tc = p.td_coul ? with_td + td[4] : with_td;
        const double add = W > 1 ? wide_spring[c] : spring64(p, tip, dum, c);
        const double all = with_tc + add;
        if (W == 1) __syncwarp();           // the buffer may be written again
        if (live && sub == 0) evals += 1;
        return writing ? acc : all;
    };

    auto start_height = [&]() {
        outside = 0;
        alpha = 0.1;
        dt = p.dt;
        nnn = 0;
        nst = 1;
        writing = nst >= p.maxsteps;
        ex = pp;
    };

    for (;;) {
        const unsigned idle = __ballot_sync(kAll, sub == 0 && w < 0 && !done);
        if (idle) {
            unsigned long long base = 0;
            if (lane == 0) base = atomicAdd(&ctr->next_work, (unsigned long long)__popc(idle));
            base = __shfl_sync(kAll, base, 0);
            if (w < 0 && !done) {
                const long long g = (long long)base + __popc(idle & ((1u << (grp * G)) - 1u));
                if (g >= n_cols) {
                    done = true;
                } else {
                    // a new column (Simulation::run, simulation.cpp:93-99)
                    w = g;
                    const int col = list ? list[g] : col_begin + (int)g;
                    o = out + (by_column ? (size_t)(col - col_begin) : (size_t)g) * p.nz;
                    double x, y;
                    dummy_xy_t<double>(p, p.tip_pbc && p.ts_mode != 2, (col / p.ny) * p.dx, (col % p.ny) * p.dy,
                                       x, y);
                    dm = va == 0 ? x : va == 1 ? y : p.zhigh;
                    pp = va == 2 ? p.zhigh - p.tip_dummy_d : dm;
                    v = 0;
                    energy = 0;
                    k = 0;
                    start_height();
                }
            }
        }
        if (__all_sync(kAll, done)) break;

        double F = evaluate(w >= 0);
        double E = bc(F, 3);
        const bool was_writing = writing && w >= 0;
        const unsigned bad = __ballot_sync(kAll, !isfinite(F));
        const unsigned out_mask = __ballot_sync(kAll, outside != 0);
        if (was_writing) {
            // System::getOutput (system.cpp:28-51)
            const unsigned quad_bits = 0xfu << quad;
            int st = (nst >= p.maxsteps ? MAFM_PT_MAXSTEPS : 0) | ((out_mask & quad_bits) ? MAFM_PT_OUTSIDE : 0);
            if (bad & quad_bits) st |= MAFM_PT_NONFINITE;
            if (writer) {
                mafm_point* r = o + k;
                if (c < 3) {
                    r->tip[c] = pp;
                    r->force[c] = F;
                } else {
                    r->energy = F;
                    r->steps = nst;
                    r->status = st;
                    steps += nst;
                    status_or |= (unsigned)st;
                }
            }
            // System::lowerTip (system.hpp:51-54)
            if (va == 2) {
                dm = dm - p.dz;
                pp = pp - p.dz;
            }
            if (++k < p.nz) start_height();
            else w = -1;
        }
        // the groups in the middle of a height take their step
        const bool act = w >= 0 && !was_writing;
        double SF = F, SE = E;
        if (p.minimiser == MAFM_MIN_SD) {
        } else if (p.integrator == MAFM_INT_EULER) {
            if (act) {
                const double p1 = pp + dt * v;
                v = v + dt * F;
                pp = p1;
            }
        } else if (p.integrator == MAFM_INT_MIDPOINT) {
            if (act) {
                const double h = dt * 0.5;
                ex = pp + h * v;
                u = v + h * F;
            }
            SF = evaluate(act);
            SE = bc(SF, 3);
            if (act) {
                pp = pp + dt * u;
                v = v + dt * SF;
            }
        } else {   // RK4 (integrators.cpp:56-111)
            const double h = dt * 0.5;
            if (act) {
                fs = F;
                es = E;
                vs = v;
                ex = pp + h * v;
                u = v + h * F;
            }
#pragma unroll 1
            for (int s = 0; s < 2; ++s) {
                F = evaluate(act);
                E = bc(F, 3);
                if (act) {
                    fs = fs + 2.0 * F;
                    es = es + 2.0 * E;
                    vs = vs + 2.0 * u;
                    const double hs = s == 0 ? h : dt;
                    ex = pp + hs * u;
                    u = v + hs * F;
                }
            }
            F = evaluate(act);
            E = bc(F, 3);
            if (act) {
                fs = fs + F;
                es = es + E;
                vs = vs + u;
                const double s6 = quo64(dt, 6.0);
                pp = pp + s6 * vs;
                v = v + s6 * fs;
                SF = quo64(fs, 6.0);
                SE = quo64(es, 6.0);
            }
        }
        // FIREMinimisation / SDMinimisation (minimiser.cpp:39-129)
        if (c == 3) SF = 0;                 // the energy's lane has no vector component
        const double fl = root64(dot(SF, SF));
        const double ediff = SE - energy;
        if (act) energy = SE;
        bool conv;
        if (p.minterm == MAFM_TERM_E) conv = fabs(ediff) < p.etol;
        else if (p.minterm == MAFM_TERM_F) conv = fl < p.ftol;
        else conv = fabs(ediff) < p.etol && fl < p.ftol;
        const bool go = act && !conv;
        if (p.minimiser == MAFM_MIN_SD) {
            if (go) pp = pp + p.dt * SF;
        } else {
            const double pw = dot(v, SF);
            const double vl = root64(dot(v, v));
            const double fh = fl > 1e-10 ? quo64(SF, fl) : 0.0;
            const double mixed = (1.0 - alpha) * v + alpha * fh * vl;
            if (go) {
                if (pw < 0.0) {
                    v = 0;
                    nnn = 0;
                    dt = dt * 0.5;
                    alpha = 0.1;
                } else {
                    v = mixed;
                    if (nnn > 5) {
                        const double g = dt * 1.1, dt_max = 10.0 * p.dt;
                        dt = dt_max < g ? dt_max : g;   // std::min(g, dt_max)
                        alpha = alpha * 0.99;
                    }
                    nnn++;
                }
            }
        }
        if (act) {
            if (conv) writing = true;
            else if (++nst >= p.maxsteps) writing = true;
            ex = pp;
        }
    }

    if (W > 1) {
        __syncwarp();
        if (lane == 0) wide_quit = 1;
        __syncthreads();
    }
    for (int off = 16; off > 0; off >>= 1) {
        steps += __shfl_xor_sync(kAll, steps, off);
        evals += __shfl_xor_sync(kAll, evals, off);
        status_or |= __shfl_xor_sync(kAll, status_or, off);
        err |= __shfl_xor_sync(kAll, err, off);
    }
    if (lane == 0) {
        atomicAdd(&ctr->total_steps, (unsigned long long)steps);
        atomicAdd(&ctr->force_evals, evals);
        atomicAdd(&ctr->pair_evals, evals * (unsigned long long)pairs_per_eval);
        if (status_or | err) atomicOr(&ctr->error_word, status_or | err);
    }
}

// One thread a column: the same bits, for so many columns that they fill the GPU by
// themselves and evaluations of so few terms that the rest of a step, which a quad's
// lanes repeat, is most of the work (thread_per_column).  One warp a block.
__global__ void __launch_bounds__(32) relax64_thread_kernel(const __grid_constant__ ScanParams p, mafm_point* out,
                                                             RunCounters* ctr, const int* list, int col_begin,
                                                             long long n_cols, bool by_column, int smem_cap) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const AtomRec64* atoms = stage64(p, reinterpret_cast<AtomRec64*>(smem_raw), smem_cap);
    Eval64 ev{p, atoms, p.n_terms_direct, p.ts_mode, 0u, 0ull};
    long long steps = 0;
    unsigned long long evals = 0;
    unsigned status_or = 0;
    for (;;) {
        const long long w = (long long)atomicAdd(&ctr->next_work, 1ull);
        if (w >= n_cols) break;
        const int col = list ? list[w] : col_begin + (int)w;
        relax_column_t<double>(ev, p, col, out + (by_column ? (size_t)(col - col_begin) : (size_t)w) * p.nz, true,
                               false, steps, evals, status_or);
    }
    atomicAdd(&ctr->total_steps, (unsigned long long)steps);
    atomicAdd(&ctr->force_evals, evals);
    atomicAdd(&ctr->pair_evals, ev.pairs);
    if (status_or | ev.err) atomicOr(&ctr->error_word, status_or | ev.err);
}

// FP64 re-relaxation of the double-float kernel's near-tie columns (scan << 32 |
// column), one warp per column.  Persistent: each warp takes the next listed
// column and relaxes it from its top height with EvalWarp64, which forms every
// sum exactly as relax64_kernel does, so the column holds the plain FP64
// kernel's bits.  The step total is corrected by the difference; force and pair
// evaluations count every pass.
__global__ void __launch_bounds__(128) repair64_kernel(const BatchScan* __restrict__ scans,
                                                       const unsigned long long* __restrict__ list,
                                                       unsigned cap, RunCounters* ctr) {
    extern __shared__ __align__(32) unsigned char rraw[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    Node64* buf = reinterpret_cast<Node64*>(rraw) + (size_t)warp * 2 * kWarpChunk;
    const unsigned listed = min(ctr->n_tie, cap);
    long long steps = 0;
    unsigned long long evals = 0, pairs = 0;
    unsigned status_or = 0, err = 0;
    for (;;) {
        unsigned long long t = 0;
        if (lane == 0) t = atomicAdd(&ctr->repair_next, 1ull);
        t = __shfl_sync(0xffffffffu, t, 0);
        if (t >= listed) break;
        const unsigned long long e = list[t];
        const BatchScan& B = scans[(int)(e >> 32)];
        const long long c = (long long)(unsigned)(e & 0xffffffffull);
        const ScanParams& p = B.p;
        EvalWarp64 ev{p, p.atoms64, p.n_terms_direct, p.ts_mode, lane, buf, B.n_pairs_per_eval, 0u, 0ull};
        relax_column_t<double>(ev, p, c, B.out + (size_t)(c - B.col_begin) * p.nz, lane == 0, true, steps,
                               evals, status_or);
        pairs += ev.pairs;
        err |= ev.err;
        __syncwarp();
    }
    if (lane == 0) {
        atomicAdd(&ctr->total_steps, (unsigned long long)steps);
        atomicAdd(&ctr->force_evals, evals);
        atomicAdd(&ctr->pair_evals, pairs);
        if (status_or | err) atomicOr(&ctr->error_word, status_or | err);
    }
}

__global__ void sample64_kernel(const ScanParams p, int what, const double* pts, long long n,
                                double* out, RunCounters* ctr) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    Eval64 ev{p, p.atoms64, p.n_terms_direct, p.ts_mode, 0u, 0ull};
    V3 tip = {pts[3 * i], pts[3 * i + 1], pts[3 * i + 2]};
    V3 F = {0, 0, 0};
    double E = 0;
    int outside = 0;
    if (what == 1) {
        if (p.es.g64) interp64(p.es, tip, F, E, outside, ev.err);
    } else {
        ev.ts(tip, F, E, outside);
    }
    out[4 * i] = F.x; out[4 * i + 1] = F.y; out[4 * i + 2] = F.z; out[4 * i + 3] = E;
    if (ev.err) atomicOr(&ctr->error_word, ev.err);
}

// Simulation::buildTipGridInteractions: one thread per node, the tip-surface
// terms (and the external field) evaluated with the tip on the node.
__global__ void __launch_bounds__(128) grid_build64_kernel(const ScanParams p, const GridView g,
                                                           Node64* out, int smem_cap,
                                                           RunCounters* ctr) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const AtomRec64* atoms = stage64(p, reinterpret_cast<AtomRec64*>(smem_raw), smem_cap);
    Eval64 ev{p, atoms, p.n_terms_direct, p.es.g64 ? 1 : 0, 0u, 0ull};
    const long long total = (long long)g.n[0] * g.n[1] * g.n[2];
    for (long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
         idx += (long long)gridDim.x * blockDim.x) {
        const int k = (int)(idx % g.n[2]);
        const long long ij = idx / g.n[2];
        const int j = (int)(ij % g.n[1]), i = (int)(ij / g.n[1]);
        double x, y;
        dummy_xy_t<double>(p, p.tip_pbc != 0, i * g.basis[0] + g.origin[0],
                           j * g.basis[4] + g.origin[1], x, y);
        V3 tip = {x, y, k * g.basis[8] + g.origin[2]};
        V3 F;
        double E;
        int outside = 0;
        ev.ts(tip, F, E, outside);
        out[idx] = Node64{F.x, F.y, F.z, E};
    }
    if (ev.err) atomicOr(&ctr->error_word, ev.err);
}

int smem_cap64(int bytes_limit) { return bytes_limit / (int)sizeof(AtomRec64); }

}  // namespace

static size_t smem_bytes64(const ScanParams& p, int& cap) {
    const int limit = 96 * 1024;
    cap = smem_cap64(limit);
    const int n = p.n_terms_direct;
    return n <= cap ? (size_t)n * sizeof(AtomRec64) : 0;
}

template <int G, int W>
static cudaError_t launch_relax64_g(const ScanParams& p, mafm_point* out, RunCounters* ctr, const int* list,
                                    int col_begin, long long n_cols, int pairs_per_eval, bool by_column,
                                    cudaStream_t s) {
    int per_sm = 0;
    const cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, relax64_kernel<G, W>, 32 * W, 0);
    if (e != cudaSuccess) return e;
    const long long need = (n_cols * G + 31) / 32;
    const long long blocks = std::max(1ll, std::min(need, (long long)sm_count() * std::max(per_sm, 1)));
    relax64_kernel<G, W><<<(unsigned)blocks, 32 * W, 0, s>>>(p, out, ctr, list, col_begin, n_cols, pairs_per_eval,
                                                             by_column);
    return cudaGetLastError();
}

// Whether a thread a column is faster than four lanes a column.  The lanes share the
// terms and nothing else, so lookups and few terms are in favour of a thread; a
// thread waits for the slowest of 32 columns at every height, so columns that cost
// differently are in favour of lanes: close to the atoms, not while the tip starts
// every height 3.5 A above the topmost one (calm).  Times in ms, thread / lanes, of
// scans at 0.05 A a pixel whose tip starts at 6 A (cluster) and 10 A (plain grid and
// field) above the atoms, 0.1 A a height:
//   rigid grid, calm  6,400 columns x 21 10.1 / 8.5, 8,100 10.1 / 12.4, 90,000 x 41 84 /
//     180; down to 2 A  8,100 233 / 117, 19,600 254 / 267, 90,000 607 / 874
//   field and 16 terms, calm  10,000 x 11 17.3 / 13.4, 19,600 21 / 29; down to 2.5 A
//     19,600 410 / 302, 40,000 643 / 661; 36 terms  40,000 x 26 480 / 504, 90,000 935 /
//     1122, x 36 2294 / 2305; 64 terms  90,000 x 26 2766 / 2527
//   4 LJ and Coulomb terms, calm  10,000 x 11 14.5 / 11.6, 19,600 x 21 33 / 40, 90,000 89 /
//     142; down to 2 A  90,000 328 / 337; LJ alone 209 / 206
//   10 terms  19,600 x 21 82 / 91, 90,000 210 / 293; down to 2 A  90,000 950 / 780
//   20 terms  19,600 x 21 295 / 219, 90,000 525 / 588; 60 terms  90,000 x 21 2557 / 2212
static bool thread_per_column(const ScanParams& p, long long n_cols, bool calm) {
    const int terms = p.n_terms_direct;
    int per_sm = INT_MAX;   // columns that an SM needs
    if (p.ts_mode == 2) per_sm = calm ? 48 : 100;
    else if (p.ts_mode == 1 && terms <= 16) per_sm = calm ? 110 : 260;
    else if (p.ts_mode == 1 && terms <= 40) per_sm = 400;
    else if (p.ts_mode == 0 && calm && terms <= 20) per_sm = terms <= 10 ? 110 : 400;
    return n_cols >= (long long)sm_count() * per_sm;
}

static cudaError_t launch_relax64_thread(const ScanParams& p, mafm_point* out, RunCounters* ctr, const int* list,
                                         int col_begin, long long n_cols, bool by_column, cudaStream_t s) {
    int cap = 0, per_sm = 0;
    const size_t smem = smem_bytes64(p, cap);
    // One warp a block spreads the columns over the SMs (20 terms, 40,000 columns x 2
    // heights: 59.5 -> 50.5 ms with blocks of 128).
    constexpr int threads = 32;
    cudaError_t e = cudaFuncSetAttribute(relax64_thread_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 96 * 1024);
    if (e == cudaSuccess)
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, relax64_thread_kernel, threads, smem);
    if (e != cudaSuccess) return e;
    const long long blocks = std::min((n_cols + threads - 1) / threads, (long long)sm_count() * std::max(per_sm, 1));
    relax64_thread_kernel<<<(unsigned)blocks, threads, smem, s>>>(p, out, ctr, list, col_begin, n_cols, by_column, cap);
    return cudaGetLastError();
}

// Lanes per column: the fewest that give every SM four warps (an SM starts an
// FP64 instruction every 19 cycles and a warp one every 64).  More lanes leave more
// of them idle in the in-order sums.  G = 4 / 8 / 16 / 32: 2,601 columns (graphene, 11
// heights) 37.4 / 25.4 / 27.6 / 42.1 ms; 22,500 (cluster, 2 heights) 89 / 106 / 130 /
// 182; 5,041 (cluster, 4 heights) 37.9 / 36.7 / 43.4 / 56.3; 1,296 35.1 / 21.8 / 16.0 /
// 18.0.
// Four warps per column while there are few columns: cluster, 41 heights, one warp /
// four warps: 1 column 163 / 103 ms, 301 190 / 125, 1,000 247 / 200; graphene without
// Coulomb, 11 heights: 576 columns 12.0 / 10.3, 800 14.5 / 15.5, 961 16.6 / 18.7.  (They
// are faster for 2 to 15 terms too, 100 columns of 4 atoms 5.1 / 3.3 ms, which the
// bound of 16 terms leaves out.)
cudaError_t launch_relax64(const ScanParams& p, mafm_point* out, RunCounters* ctr, const int* list,
                           int col_begin, long long n_cols, int pairs_per_eval, bool by_column, bool calm,
                           cudaStream_t s) {
    if (n_cols <= 0) return cudaSuccess;
    if (thread_per_column(p, n_cols, calm))
        return launch_relax64_thread(p, out, ctr, list, col_begin, n_cols, by_column, s);
    int G = 4;
    while (G < 32 && n_cols * G < 32ll * 4 * sm_count()) G *= 2;
    const long long wide_cols = (p.has_coulomb ? 7ll : 4ll) * sm_count();
    if (n_cols <= wide_cols && p.n_terms_direct >= 16)
        return launch_relax64_g<32, 4>(p, out, ctr, list, col_begin, n_cols, pairs_per_eval, by_column, s);
    switch (G) {
        case 4: return launch_relax64_g<4, 1>(p, out, ctr, list, col_begin, n_cols, pairs_per_eval, by_column, s);
        case 8: return launch_relax64_g<8, 1>(p, out, ctr, list, col_begin, n_cols, pairs_per_eval, by_column, s);
        case 16: return launch_relax64_g<16, 1>(p, out, ctr, list, col_begin, n_cols, pairs_per_eval, by_column, s);
        default: return launch_relax64_g<32, 1>(p, out, ctr, list, col_begin, n_cols, pairs_per_eval, by_column, s);
    }
}

cudaError_t launch_repair64(const BatchScan* scans, const unsigned long long* list, unsigned cap,
                            RunCounters* ctr, cudaStream_t s) {
    constexpr int kThreads = 128;
    const size_t smem = (size_t)(kThreads / 32) * 2 * kWarpChunk * sizeof(Node64);
    repair64_kernel<<<(unsigned)sm_count(), kThreads, smem, s>>>(scans, list, cap, ctr);
    return cudaGetLastError();
}

cudaError_t launch_sample64(const ScanParams& p, int what, const double* pts, int64_t n,
                            double* out, RunCounters* ctr, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    sample64_kernel<<<(unsigned)((n + 127) / 128), 128, 0, s>>>(p, what, pts, n, out, ctr);
    return cudaGetLastError();
}

cudaError_t launch_grid_build64(const ScanParams& p, const GridView& g, Node64* out,
                                RunCounters* ctr, cudaStream_t s) {
    int cap;
    size_t sm = smem_bytes64(p, cap);
    cudaError_t e = cudaFuncSetAttribute(grid_build64_kernel,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, 96 * 1024);
    if (e != cudaSuccess) return e;
    const long long total = (long long)g.n[0] * g.n[1] * g.n[2];
    long long blocks = (total + 127) / 128;
    const long long cap_blocks = (long long)sm_count() * 16;
    if (blocks > cap_blocks) blocks = cap_blocks;
    if (blocks < 1) blocks = 1;
    grid_build64_kernel<<<(unsigned)blocks, 128, sm, s>>>(p, g, out, cap, ctr);
    return cudaGetLastError();
}

}  // namespace mafm
