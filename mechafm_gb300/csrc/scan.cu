// scan.cu — device-resident scans and the relax / sample / grid entry points
// of the C ABI.
//
//   mafm_scan_create   packs the tip–atom terms in the reference's interaction
//                      order (simulation.cpp:238-320, 503-515), uploads them,
//                      computes the external field by FFT on the GPU
//                      (ElectrostaticPotentialInteraction ctor,
//                      interactions.cpp:53-234, with cuFFT in FP64) and
//                      records the rigid-grid geometry (simulation.cpp:428-441).
//   rigid grids        are built on first use, FP64 for MAFM_FP64 runs and
//                      FP32 for MAFM_FP32C runs (simulation.cpp:445-501).
//   mafm_run           plain FP64 kernel or the FP32 persistent kernel.
//   mafm_run_batch     many scans in one persistent FP32 launch.
#include <cufft.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "mafm_df.h"
#include "mafm_internal.h"

namespace mafm {
namespace {

constexpr double kPi = 3.14159265358979323846;

// Device buffer owned by a scan.
template <class T>
struct DevBuf {
    T* p = nullptr;
    size_t n = 0;
    DevBuf() = default;
    DevBuf(const DevBuf&) = delete;
    DevBuf& operator=(const DevBuf&) = delete;
    ~DevBuf() { release(); }
    void release() {
        if (p) cudaFree(p);
        p = nullptr;
        n = 0;
    }
    void alloc(size_t count) {
        if (count <= n && p) return;
        release();
        if (count == 0) return;
        cudaError_t e = cudaMalloc(&p, count * sizeof(T));
        if (e != cudaSuccess) {
            p = nullptr;
            fail(MAFM_E_NOMEM, "cudaMalloc of %zu bytes failed: %s", count * sizeof(T),
                 cudaGetErrorString(e));
        }
        n = count;
    }
};

struct M3 {
    double v[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};
};

double det3(const M3& m) {
    double d = 0;
    d = m.v[0][0] * (m.v[1][1] * m.v[2][2] - m.v[1][2] * m.v[2][1]);
    d += m.v[0][1] * (m.v[1][2] * m.v[2][0] - m.v[1][0] * m.v[2][2]);
    d += m.v[0][2] * (m.v[1][0] * m.v[2][1] - m.v[1][1] * m.v[2][0]);
    return d;
}

// Matrix3::inverse (matrices.hpp:89-116)
M3 inv3(const M3& m) {
    M3 r;
    const double inv_det = 1 / det3(m);
    const double a = m.v[0][0], b = m.v[0][1], c = m.v[0][2];
    const double d = m.v[1][0], e = m.v[1][1], f = m.v[1][2];
    const double g = m.v[2][0], h = m.v[2][1], i = m.v[2][2];
    r.v[0][0] = inv_det * (e * i - f * h);
    r.v[0][1] = -inv_det * (b * i - c * h);
    r.v[0][2] = inv_det * (b * f - c * e);
    r.v[1][0] = -inv_det * (d * i - f * g);
    r.v[1][1] = inv_det * (a * i - c * g);
    r.v[1][2] = -inv_det * (a * f - c * d);
    r.v[2][0] = inv_det * (d * h - e * g);
    r.v[2][1] = -inv_det * (a * h - b * g);
    r.v[2][2] = inv_det * (a * e - b * d);
    return r;
}

bool is_diagonal(const M3& m) {   // Matrix3::isDiagonal (matrices.hpp:71-86)
    double ds = 0, nd = 0;
    for (int i = 0; i < 3; i++)
        for (int j = 0; j < 3; j++) {
            if (i == j) ds += std::abs(m.v[i][i]);
            else nd += std::abs(m.v[i][j]);
        }
    return nd < 1.0e-10 * ds;
}

M3 from_rowmajor(const double* a) {
    M3 m;
    for (int r = 0; r < 3; ++r)
        for (int c = 0; c < 3; ++c) m.v[r][c] = a[3 * r + c];
    return m;
}

void to_rowmajor(const M3& m, double* a) {
    for (int r = 0; r < 3; ++r)
        for (int c = 0; c < 3; ++c) a[3 * r + c] = m.v[r][c];
}

// ---- external field kernels (FP64) ----------------------------------------

__global__ void real_to_complex(const double* v, cufftDoubleComplex* c, long long n) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x)
        c[i] = make_cuDoubleComplex(v[i], 0.0);
}

// E(k) = V(k) * (vol * rho(k))  (interactions.cpp:139-146)
__global__ void kspace_product(cufftDoubleComplex* V, const cufftDoubleComplex* R, double vol,
                               long long n) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x) {
        const double ar = vol * R[i].x, ai = vol * R[i].y;
        const double vr = V[i].x, vi = V[i].y;
        V[i] = make_cuDoubleComplex(vr * ar - vi * ai, vr * ai + vi * ar);
    }
}

struct KBasis {
    double kb[9];   // reciprocal basis (B diag(n))^-1^T, row-major
    int n[3];
};

// -2 pi i (ka + kb + kc)_comp E(k), Nyquist wrap at i >= n/2 (interactions.cpp:165-225)
__global__ void gradient_mult(const cufftDoubleComplex* E, cufftDoubleComplex* out, KBasis K,
                              int comp) {
    const long long N = (long long)K.n[0] * K.n[1] * K.n[2];
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < N;
         i += (long long)gridDim.x * blockDim.x) {
        const int iz = (int)(i % K.n[2]);
        const long long r = i / K.n[2];
        const int iy = (int)(r % K.n[1]), ix = (int)(r / K.n[1]);
        double ka = ix * K.kb[3 * comp + 0];
        if (ix >= K.n[0] / 2) ka -= K.n[0] * K.kb[3 * comp + 0];
        double kbv = iy * K.kb[3 * comp + 1];
        if (iy >= K.n[1] / 2) kbv -= K.n[1] * K.kb[3 * comp + 1];
        double kc = iz * K.kb[3 * comp + 2];
        if (iz >= K.n[2] / 2) kc -= K.n[2] * K.kb[3 * comp + 2];
        const double kk = ka + kbv + kc;
        out[i] = make_cuDoubleComplex(2.0 * kPi * kk * E[i].y, -2.0 * kPi * kk * E[i].x);
    }
}

// Real part / N into one component of the node array; imaginary residue check
// of ffti_data_grid (fft.cpp:79-83): only positive residues are checked.
__global__ void take_real(const cufftDoubleComplex* in, Node64* out, int comp, long long N,
                          unsigned long long* max_bits) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < N;
         i += (long long)gridDim.x * blockDim.x) {
        const double v = in[i].x / N;
        double* o = reinterpret_cast<double*>(out + i);
        o[comp] = v;
        const double im = in[i].y / N;
        if (im > 1.0e-8) atomicMax(max_bits, (unsigned long long)__double_as_longlong(im));
    }
}

__global__ void nodes_to_float4(const Node64* in, float4* out, long long n) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x) {
        const Node64 v = in[i];
        out[i] = make_float4((float)v.x, (float)v.y, (float)v.z, (float)v.w);
    }
}

__global__ void write_batch(BatchScan* dst, BatchScan v) { *dst = v; }
__global__ void write_batch_df(BatchDF* dst, BatchDF v) { *dst = v; }

// Expected relaxation cost of each pixel column: the density of tip–atom terms
// under the pixel (Gaussian of 2 A in xy).  Columns over the molecule take up
// to ten times more FIRE steps than columns over vacuum; running the
// expensive ones first shortens the tail of the persistent launch.
__global__ void column_cost_proxy(const AtomRec32* terms, int n_terms, int nx, int ny, double dx,
                                  double dy, float* w) {
    const long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= (long long)nx * ny) return;
    const float x = (float)((c / ny) * dx), y = (float)((c % ny) * dy);
    float acc = 0.f;
    for (int t = 0; t < n_terms; ++t) {
        const float ex = x - terms[t].a.x, ey = y - terms[t].a.y;
        acc += __expf(-(ex * ex + ey * ey) * 0.125f);
    }
    w[c] = acc;
}

// FIRE steps of each pixel column (the sum over its heights) of a relaxed scan.
__global__ void column_steps(const mafm_point* pts, int nz, long long n_cols, unsigned* steps) {
    const long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= n_cols) return;
    unsigned s = 0;
    for (int k = 0; k < nz; ++k) s += (unsigned)pts[c * nz + k].steps;
    steps[c] = s;
}

unsigned grid_blocks(long long n) {
    long long b = (n + 255) / 256;
    const long long cap = (long long)sm_count() * 32;
    return (unsigned)std::max(1ll, std::min(b, cap));
}

}  // namespace
}  // namespace mafm

struct mafm_scan {
    int device = 0;
    mafm_scan_desc d{};                 // scalars of the descriptor (pointers not kept)
    mafm::ScanParams P{};               // shared parameters; pointers filled per precision
    mafm::DevBuf<mafm::AtomRec64> atoms64;
    mafm::DevBuf<mafm::AtomRec32> atoms32;
    mafm::DevBuf<mafm::TermPair32> units32;
    mafm::DevBuf<int32_t> index32;       // FP64 term index of each atoms32 record
    mafm::DevBuf<mafm::Node64> es64, grid64;
    mafm::DevBuf<float4> es32, grid32;
    mafm::GridView es_view{}, grid_view{};
    bool grid64_built = false, grid32_built = false;
    mafm::DevBuf<mafm::RunCounters> ctr;
    mafm::DevBuf<mafm::BatchScan> batch;
    mafm::DevBuf<mafm_point> stage;
    mafm::DevBuf<int> order;             // columns by descending expected cost
    mafm::DevBuf<mafm::TermPairDF> pairsdf;    // terms in double-float pairs (MAFM_DF)
    int df_lj_pairs = 0, df_morse_pairs = 0;
    mafm::DevBuf<mafm::NodeDF> esdf;           // external field in double-float
    mafm::DevBuf<mafm::NodeDF> griddf;         // rigid grid built in double-float
    mafm::DevBuf<mafm::Node64> griddf64;       //   and its FP64 copy (re-relaxation)
    bool griddf_built = false;
    // the interpolated build of it: laid out at the first build, where it pays
    std::vector<float> df_xyz;                 // positions of the term pairs (rigid grids)
    bool far_planned = false, far_used = false;
    mafm::FarViewDF far{};
    mafm::DevBuf<unsigned char> far_tables;
    mafm::DevBuf<unsigned> far_mask;
    mafm::DevBuf<mafm::NodeDF> far_coef;
    mafm::DevBuf<mafm::BatchDF> batchdf;       // descriptor of a double-float run
    mafm::DevBuf<unsigned long long> repair;   // columns to re-relax in FP64
    bool order_built = false;
    bool order_measured = false;          // order from a relaxation's step counts
    mafm::RunCounters* host_ctr = nullptr;   // pinned
    int n_pairs_per_eval = 0;
    bool calm = false;                         // every height starts 3.5 A above the topmost atom
    int has_coulomb = 0;
    std::vector<int32_t> atom_type;      // type index of each surface atom (adjoint folding)
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    ~mafm_scan() {
        if (host_ctr) cudaFreeHost(host_ctr);
        if (ev0) cudaEventDestroy(ev0);
        if (ev1) cudaEventDestroy(ev1);
    }
};

namespace mafm {
namespace {

void validate(const mafm_scan_desc* d) {
    if (!d) fail(MAFM_E_INVALID, "null descriptor");
    if (d->flexible) fail(MAFM_E_UNSUPPORTED, "a flexible molecule runs through mafm_flex_create");
    if (d->n_atoms < 0 || d->n_types < 0) fail(MAFM_E_INVALID, "negative atom or type count");
    if (d->n_atoms > 0 && (!d->pos || !d->type || !d->tip_pair))
        fail(MAFM_E_INVALID, "descriptor has atoms but null pos/type/tip_pair");
    if (d->n_atoms > 0 && d->coulomb && !d->charge)
        fail(MAFM_E_INVALID, "coulomb on but charge is null");
    for (int a = 0; a < d->n_atoms; ++a)
        if (d->type[a] < 0 || d->type[a] >= d->n_types)
            fail(MAFM_E_INVALID, "atom %d has type index %d outside [0, %d)", a, d->type[a], d->n_types);
    for (int t = 0; t < d->n_types; ++t)
        if (d->tip_pair[t].kind != MAFM_PAIR_LJ && d->tip_pair[t].kind != MAFM_PAIR_MORSE)
            fail(MAFM_E_INVALID, "pair kind %d of type %d", d->tip_pair[t].kind, t);
    if (d->dummy_pair.kind != MAFM_PAIR_LJ && d->dummy_pair.kind != MAFM_PAIR_MORSE)
        fail(MAFM_E_INVALID, "dummy pair kind %d", d->dummy_pair.kind);
    if (d->nx < 1 || d->ny < 1 || d->nz < 1) fail(MAFM_E_INVALID, "empty scan grid %d x %d x %d", d->nx, d->ny, d->nz);
    if ((long long)d->nx * d->ny > 0x7fffffffll) fail(MAFM_E_RANGE, "more than 2^31 pixel columns");
    if (d->minimiser != MAFM_MIN_SD && d->minimiser != MAFM_MIN_FIRE) fail(MAFM_E_INVALID, "minimiser %d", d->minimiser);
    if (d->integrator < MAFM_INT_EULER || d->integrator > MAFM_INT_RK4) fail(MAFM_E_INVALID, "integrator %d", d->integrator);
    if (d->minterm < MAFM_TERM_E || d->minterm > MAFM_TERM_EF) fail(MAFM_E_INVALID, "minterm %d", d->minterm);
    if (d->use_external_potential) {
        if (!d->epot) fail(MAFM_E_INVALID, "external potential on but epot is null");
        if (d->epot_n[0] < 1 || d->epot_n[1] < 1 || d->epot_n[2] < 1) fail(MAFM_E_INVALID, "empty potential grid");
    }
}

// Tip–atom terms in the reference's interaction order.
void pack_terms(mafm_scan& s, const mafm_scan_desc& d) {
    const M3 cell = from_rowmajor(d.cell);
    std::vector<AtomRec64> t64;
    const int images = d.vdw_pbc ? 9 : 1;
    t64.reserve((size_t)d.n_atoms * images);
    for (int ia = -1; ia <= 1; ++ia)
        for (int ib = -1; ib <= 1; ++ib) {
            if (!d.vdw_pbc && (ia != 0 || ib != 0)) continue;
            double sx = 0, sy = 0, sz = 0;
            if (d.vdw_pbc) {   // simulation.cpp:303-306
                sx = ia * cell.v[0][0] + ib * cell.v[0][1];
                sy = ia * cell.v[1][0] + ib * cell.v[1][1];
                sz = ia * cell.v[2][0] + ib * cell.v[2][1];
            }
            for (int a = 0; a < d.n_atoms; ++a) {
                const mafm_pair& p = d.tip_pair[d.type[a]];
                AtomRec64 r{};
                if (d.vdw_pbc) {
                    r.x = d.pos[3 * a] + sx;
                    r.y = d.pos[3 * a + 1] + sy;
                    r.z = d.pos[3 * a + 2] + sz;
                } else {
                    r.x = d.pos[3 * a];
                    r.y = d.pos[3 * a + 1];
                    r.z = d.pos[3 * a + 2];
                }
                r.kind = p.kind;
                r.p0 = p.p[0];
                r.p1 = p.p[1];
                r.p2 = p.p[2];
                // addCoulombInteraction (simulation.cpp:269-295): only without
                // vdw_pbc, and only if both charges are non-zero.
                r.coul = d.coulomb && !d.vdw_pbc && d.tip_charge != 0 && d.charge[a] != 0;
                r.qq = r.coul ? d.qbase * d.tip_charge * d.charge[a] : 0.0;
                t64.push_back(r);
            }
        }
    // FP32 copy, LJ terms first so that lanes sharing a column rarely diverge on the kind.
    std::vector<AtomRec32> t32;
    std::vector<int32_t> t32_index;   // FP64 term of each FP32 record
    t32.reserve(t64.size());
    int n_coul = 0;
    for (int pass = 0; pass < 2; ++pass)
        for (const AtomRec64& r : t64) {
            if ((pass == 0) != (r.kind == MAFM_PAIR_LJ)) continue;
            t32_index.push_back((int32_t)(&r - t64.data()));
            AtomRec32 q;
            q.a = make_float4((float)r.x, (float)r.y, (float)r.z, (float)r.qq);
            int kind = r.kind;
            float kf;
            std::memcpy(&kf, &kind, sizeof kf);
            q.b = make_float4((float)r.p0, (float)r.p1, (float)r.p2, kf);
            t32.push_back(q);
            n_coul += r.coul;
        }
    // Paired copy for the packed relax loop (TermPair32).
    std::vector<TermPair32> u32;
    int n_units_lj = 0;
    for (int pass = 0; pass < 2; ++pass) {
        std::vector<const AtomRec64*> run;
        for (const AtomRec64& r : t64)
            if ((pass == 0) == (r.kind == MAFM_PAIR_LJ)) run.push_back(&r);
        for (size_t i = 0; i < run.size(); i += 2) {
            const AtomRec64* t[2] = {run[i], i + 1 < run.size() ? run[i + 1] : nullptr};
            float f[16];
            for (int c = 0; c < 2; ++c) {
                AtomRec64 z{};
                z.x = z.y = z.z = 1.0e4;   // padding: zero parameters, far away
                const AtomRec64& r = t[c] ? *t[c] : z;
                f[0 + c] = (float)-r.x;
                f[2 + c] = (float)-r.y;
                f[4 + c] = (float)-r.z;
                f[6 + c] = (float)-r.qq;
                if (pass == 0) {
                    f[8 + c] = (float)-r.p0;
                    f[10 + c] = (float)r.p1;
                    f[12 + c] = (float)(-12.0 * r.p1);
                    f[14 + c] = (float)(6.0 * r.p0);
                } else {
                    f[8 + c] = (float)r.p0;
                    f[10 + c] = (float)-r.p1;
                    f[12 + c] = (float)-r.p2;
                    f[14 + c] = (float)(-2.0 * r.p0 * r.p1);
                }
            }
            TermPair32 q;
            q.xy = make_float4(f[0], f[1], f[2], f[3]);
            q.zq = make_float4(f[4], f[5], f[6], f[7]);
            q.pa = make_float4(f[8], f[9], f[10], f[11]);
            q.pb = make_float4(f[12], f[13], f[14], f[15]);
            u32.push_back(q);
        }
        if (pass == 0) n_units_lj = (int)u32.size();
    }
    s.units32.alloc(std::max<size_t>(u32.size(), 1));
    if (!u32.empty())
        cuda_check(cudaMemcpy(s.units32.p, u32.data(), u32.size() * sizeof(TermPair32),
                              cudaMemcpyHostToDevice), "upload terms");
    s.P.n_units = (int)u32.size();
    s.P.n_units_lj = n_units_lj;
    s.atoms64.alloc(std::max<size_t>(t64.size(), 1));
    s.atoms32.alloc(std::max<size_t>(t32.size(), 1));
    s.index32.alloc(std::max<size_t>(t32.size(), 1));
    if (!t64.empty()) {
        cuda_check(cudaMemcpy(s.index32.p, t32_index.data(), t32_index.size() * sizeof(int32_t),
                              cudaMemcpyHostToDevice), "upload terms");
        cuda_check(cudaMemcpy(s.atoms64.p, t64.data(), t64.size() * sizeof(AtomRec64),
                              cudaMemcpyHostToDevice), "upload terms");
        cuda_check(cudaMemcpy(s.atoms32.p, t32.data(), t32.size() * sizeof(AtomRec32),
                              cudaMemcpyHostToDevice), "upload terms");
    }
    // double-float pairs for MAFM_DF
    const std::vector<TermPairDF> tdf = term_pairs_df(t64, s.df_lj_pairs, s.df_morse_pairs);
    if (d.rigidgrid)
        for (const TermPairDF& q : tdf)
            s.df_xyz.insert(s.df_xyz.end(), {q.xh.x, q.yh.x, q.zh.x, q.xh.y, q.yh.y, q.zh.y});
    s.pairsdf.alloc(std::max<size_t>(tdf.size(), 1));
    if (!tdf.empty())
        cuda_check(cudaMemcpy(s.pairsdf.p, tdf.data(), tdf.size() * sizeof(TermPairDF),
                              cudaMemcpyHostToDevice), "upload terms");
    s.P.n_terms = (int)t64.size();
    s.P.n_terms_direct = d.rigidgrid ? 0 : s.P.n_terms;
    s.has_coulomb = n_coul > 0;
    s.P.has_coulomb = s.has_coulomb;
    s.n_pairs_per_eval = d.rigidgrid ? 0 : (int)t64.size() + n_coul;
    double top = -INFINITY;
    for (int a = 0; a < d.n_atoms; ++a) top = std::max(top, d.pos[3 * a + 2]);
    s.calm = d.zhigh - (d.nz - 1) * d.dz - d.tip_dummy_d - top > 3.5;
}

// ElectrostaticPotentialInteraction ctor (interactions.cpp:53-234) on the GPU.
void build_external_field(mafm_scan& s, const mafm_scan_desc& d) {
    const int n0 = d.epot_n[0], n1 = d.epot_n[1], n2 = d.epot_n[2];
    const long long N = (long long)n0 * n1 * n2;
    const M3 B = from_rowmajor(d.epot_basis);
    const bool orth = is_diagonal(B);
    // Gaussian tip charge on the host, in the reference's order (interactions.cpp:63-105).
    std::vector<double> rho((size_t)N, 0.0);
    {
        const double w = 0.5;   // g_tip_gaussian_width (globals.hpp:17)
        const double w2 = pow(w, 2);
        const double norm = 1.0 / pow(w * sqrt(2.0 * kPi), 3);
        const int nmin = std::min(std::min(n0, n1), n2);
        int cut[3] = {nmin, nmin, nmin};
        for (int a = 0; a < 3; ++a)
            for (int i = 0; i < nmin - 1; i++) {
                const double vx = i * B.v[0][a], vy = i * B.v[1][a], vz = i * B.v[2][a];
                const double sq = vx * vx + vy * vy + vz * vz;
                if (exp(-0.5 * sq / w2) < 1.0e-10) {   // g_gaussian_cutoff_value
                    cut[a] = i;
                    break;
                }
            }
        const int n[3] = {n0, n1, n2};
        for (int ix = -cut[0]; ix <= cut[0]; ix++)
            for (int iy = -cut[1]; iy <= cut[1]; iy++)
                for (int iz = -cut[2]; iz < cut[2]; iz++) {
                    double px, py, pz;
                    if (orth) {
                        px = 0 + ix * B.v[0][0];
                        py = 0 + iy * B.v[1][1];
                        pz = 0 + iz * B.v[2][2];
                    } else {
                        px = 0 + (B.v[0][0] * ix + B.v[0][1] * iy + B.v[0][2] * iz);
                        py = 0 + (B.v[1][0] * ix + B.v[1][1] * iy + B.v[1][2] * iz);
                        pz = 0 + (B.v[2][0] * ix + B.v[2][1] * iy + B.v[2][2] * iz);
                    }
                    const double r2 = px * px + py * py + pz * pz;
                    int g[3] = {ix, iy, iz};
                    for (int a = 0; a < 3; ++a)
                        if (g[a] < 0 || g[a] >= n[a]) {
                            const int k = (int)floor((double)g[a] / n[a]);
                            g[a] -= k * n[a];
                        }
                    rho[((size_t)g[0] * n1 + g[1]) * n2 + g[2]] +=
                        d.tip_charge * norm * exp(-0.5 * r2 / w2);
                }
    }
    DevBuf<double> real;
    DevBuf<cufftDoubleComplex> V, R;
    real.alloc((size_t)N);
    V.alloc((size_t)N);
    R.alloc((size_t)N);
    const unsigned nb = grid_blocks(N);
    cuda_check(cudaMemcpy(real.p, d.epot, N * sizeof(double), cudaMemcpyHostToDevice), "upload potential");
    real_to_complex<<<nb, 256>>>(real.p, V.p, N);
    cuda_check(cudaMemcpy(real.p, rho.data(), N * sizeof(double), cudaMemcpyHostToDevice), "upload rho");
    real_to_complex<<<nb, 256>>>(real.p, R.p, N);
    cuda_check(cudaGetLastError(), "external field setup");
    real.release();
    cufftHandle plan;
    if (cufftPlan3d(&plan, n0, n1, n2, CUFFT_Z2Z) != CUFFT_SUCCESS)
        fail(MAFM_E_CUDA, "cufftPlan3d(%d, %d, %d) failed", n0, n1, n2);
    struct PlanGuard { cufftHandle h; ~PlanGuard() { cufftDestroy(h); } } guard{plan};
    if (cufftExecZ2Z(plan, V.p, V.p, CUFFT_FORWARD) != CUFFT_SUCCESS ||
        cufftExecZ2Z(plan, R.p, R.p, CUFFT_FORWARD) != CUFFT_SUCCESS)
        fail(MAFM_E_CUDA, "forward FFT of the external potential failed");
    kspace_product<<<nb, 256>>>(V.p, R.p, det3(B), N);
    // reciprocal basis (fft.cpp:41-47)
    M3 bn;
    for (int r = 0; r < 3; ++r)
        for (int c = 0; c < 3; ++c) bn.v[r][c] = B.v[r][c] * d.epot_n[c];
    const M3 bi = inv3(bn);
    KBasis K;
    for (int r = 0; r < 3; ++r)
        for (int c = 0; c < 3; ++c) K.kb[3 * r + c] = bi.v[c][r];
    K.n[0] = n0; K.n[1] = n1; K.n[2] = n2;
    s.es64.alloc((size_t)N);
    DevBuf<unsigned long long> maxbits;
    maxbits.alloc(1);
    cuda_check(cudaMemset(maxbits.p, 0, sizeof(unsigned long long)), "memset");
    for (int comp = -1; comp < 3; ++comp) {
        if (comp < 0) cuda_check(cudaMemcpy(R.p, V.p, N * sizeof(cufftDoubleComplex), cudaMemcpyDeviceToDevice), "copy");
        else gradient_mult<<<nb, 256>>>(V.p, R.p, K, comp);
        if (cufftExecZ2Z(plan, R.p, R.p, CUFFT_INVERSE) != CUFFT_SUCCESS)
            fail(MAFM_E_CUDA, "inverse FFT of the external field failed");
        take_real<<<nb, 256>>>(R.p, s.es64.p, comp < 0 ? 3 : comp, N, maxbits.p);
    }
    s.es32.alloc((size_t)N);
    nodes_to_float4<<<nb, 256>>>(s.es64.p, s.es32.p, N);
    s.esdf.alloc((size_t)N);
    cuda_check(launch_nodes_to_df(s.es64.p, s.esdf.p, N, nullptr), "external field (double-float)");
    cuda_check(cudaDeviceSynchronize(), "external field");
    unsigned long long bits = 0;
    cuda_check(cudaMemcpy(&bits, maxbits.p, sizeof bits, cudaMemcpyDeviceToHost), "readback");
    if (bits) {
        double im;
        std::memcpy(&im, &bits, sizeof im);
        fail(MAFM_E_RANGE, "Imaginary part of inverse FFT exceeded threshold 1.0e-8! Value: %e",
             im * (double)N);
    }
    GridView& g = s.es_view;
    g.g64 = s.es64.p;
    g.g32 = s.es32.p;
    g.n[0] = n0; g.n[1] = n1; g.n[2] = n2;
    g.periodic = 1;
    g.orthogonal = orth;
    to_rowmajor(B, g.basis);
    to_rowmajor(inv3(B), g.inv);
    for (int a = 0; a < 3; ++a) g.origin[a] = d.epot_origin[a];
}

// Geometry of the rigid grid (simulation.cpp:428-441).
void rigid_grid_geometry(mafm_scan& s, const mafm_scan_desc& d) {
    GridView& g = s.grid_view;
    const double sp[3] = {d.dx / 2, d.dy / 2, d.dz / 2};
    int border[3];
    for (int a = 0; a < 3; ++a) border[a] = (int)ceil(1.5 / sp[a]);   // g_force_grid_margin
    const double nx = floor(d.area[0] / sp[0]) + 2 * border[0] + 1;
    const double ny = floor(d.area[1] / sp[1]) + 2 * border[1] + 1;
    const double nz = floor((d.zhigh - d.zlow) / sp[2]) + 2 * border[2] + 1;
    if (nx * ny * nz > 4.0e9) fail(MAFM_E_RANGE, "rigid grid of %.0f nodes is too large", nx * ny * nz);
    g.n[0] = (int)nx;
    g.n[1] = (int)ny;
    g.n[2] = (int)nz;
    g.origin[0] = -border[0] * sp[0];
    g.origin[1] = -border[1] * sp[1];
    g.origin[2] = d.zlow - d.tip_dummy_d - border[2] * sp[2];
    std::memset(g.basis, 0, sizeof g.basis);
    std::memset(g.inv, 0, sizeof g.inv);
    for (int a = 0; a < 3; ++a) {
        g.basis[4 * a] = sp[a];
        g.inv[4 * a] = 1 / sp[a];
    }
    g.periodic = 0;
    g.orthogonal = 1;
}

ScanParams build_params(const mafm_scan& s) {
    ScanParams p = s.P;
    p.n_terms_direct = s.d.rigidgrid ? 0 : p.n_terms;
    return p;
}

// The FP64 descriptor that a double-float launch's re-relaxation reads: over
// a rigid grid, the FP64 copy of the double-float grid.
ScanParams build_params_for(const mafm_scan& s, bool df) {
    ScanParams p = build_params(s);
    if (df && s.d.rigidgrid) p.grid.g64 = s.griddf64.p;
    return p;
}

// Parameters of the grid build: every tip–surface term plus the external field.
ScanParams build_grid_params(const mafm_scan& s) {
    ScanParams p = s.P;
    p.n_terms_direct = p.n_terms;
    p.ts_mode = s.d.use_external_potential ? 1 : 0;
    p.es = s.es_view;
    return p;
}

void zero_counters(mafm_scan& s, cudaStream_t st) {
    cuda_check(cudaMemsetAsync(s.ctr.p, 0, sizeof(RunCounters), st), "reset counters");
}

void ensure_grid(mafm_scan& s, bool fp64, cudaStream_t st, bool rebuild = false) {
    if (!s.d.rigidgrid) return;
    const long long N = (long long)s.grid_view.n[0] * s.grid_view.n[1] * s.grid_view.n[2];
    if (rebuild) {
        if (fp64) s.grid64_built = false;
        else s.grid32_built = false;
    }
    if (fp64 && !s.grid64_built) {
        if (!s.grid64.p) s.grid64.alloc((size_t)N);
        zero_counters(s, st);
        cuda_check(launch_grid_build64(build_grid_params(s), s.grid_view, s.grid64.p, s.ctr.p, st), "grid build");
        s.grid_view.g64 = s.grid64.p;
        s.grid64_built = true;
    }
    if (!fp64 && !s.grid32_built) {
        if (!s.grid32.p) s.grid32.alloc((size_t)N);
        zero_counters(s, st);
        cuda_check(launch_grid_build32(build_grid_params(s), s.grid_view, s.grid32.p, s.ctr.p, st), "grid build");
        s.grid_view.g32 = s.grid32.p;
        s.grid32_built = true;
    }
    s.P.grid = s.grid_view;
}

// The interpolated build's plan on the device (once per scan).
void ensure_far_plan(mafm_scan& s, cudaStream_t st) {
    if (s.far_planned) return;
    FarPlanDF plan;
    if (plan_far_df(build_grid_params(s), s.grid_view, s.df_xyz, s.df_lj_pairs, plan)) {
        std::vector<unsigned char> host;
        auto piece = [&](const void* p, size_t bytes) {
            const size_t at = (host.size() + 63) & ~(size_t)63;
            host.resize(at + bytes);
            std::memcpy(host.data() + at, p, bytes);
            return at;
        };
        size_t at[3][5];
        long long blocks = 1, strips = 1;
        for (int a = 0; a < 3; ++a) {
            const FarAxisDF& A = plan.axis[a];
            at[a][0] = piece(A.begin.data(), A.begin.size() * sizeof(int));
            at[a][1] = piece(A.pos.data(), A.pos.size() * sizeof(dfloat));
            at[a][2] = piece(A.cheb.data(), A.cheb.size() * sizeof(dfloat));
            at[a][3] = piece(A.lag.data(), A.lag.size() * sizeof(dfloat));
            at[a][4] = piece(A.box.data(), A.box.size() * sizeof(float2));
            s.far.nb[a] = (int)A.begin.size() - 1;
            blocks *= s.far.nb[a];
            int most = 0;
            for (int b = 0; b < s.far.nb[a]; ++b) most = std::max(most, A.begin[b + 1] - A.begin[b]);
            if (a == 0) s.far.max_planes = most;
            strips *= a == 2 ? (most + 3) / 4 : most;
        }
        try {
            s.far_tables.alloc(host.size());
            const size_t chunk = (size_t)std::min<long long>(blocks, kFarChunk);
            s.far_mask.alloc(chunk * plan.words);
            s.far_coef.alloc(chunk * kFarPoints * kFarPoints * kFarPoints);
        } catch (const Failure&) {   // no room beside the grid: the direct sum needs none
            cudaGetLastError();
            s.far_tables.release();
            s.far_mask.release();
            s.far_coef.release();
            s.far_planned = true;
            return;
        }
        cuda_check(cudaMemcpyAsync(s.far_tables.p, host.data(), host.size(), cudaMemcpyHostToDevice, st),
                   "upload grid plan");
        cuda_check(cudaStreamSynchronize(st), "upload grid plan");
        for (int a = 0; a < 3; ++a) {
            const unsigned char* t = s.far_tables.p;
            s.far.begin[a] = reinterpret_cast<const int*>(t + at[a][0]);
            s.far.pos[a] = reinterpret_cast<const dfloat*>(t + at[a][1]);
            s.far.cheb[a] = reinterpret_cast<const dfloat*>(t + at[a][2]);
            s.far.lag[a] = reinterpret_cast<const dfloat*>(t + at[a][3]);
            s.far.box[a] = reinterpret_cast<const float2*>(t + at[a][4]);
        }
        s.far.words = plan.words;
        s.far.first = 0;
        s.far.max_strips = (int)strips;
        s.far.mask = s.far_mask.p;
        s.far.coef = s.far_coef.p;
        s.far_used = true;
    }
    s.far_planned = true;
}

// The double-float rigid grid (MAFM_DF) and its FP64 copy, built on first use
// (rebuild: again).
void ensure_grid_df(mafm_scan& s, cudaStream_t st, bool rebuild = false) {
    if (!s.d.rigidgrid) return;
    if (rebuild) s.griddf_built = false;
    if (s.griddf_built) return;
    const long long N = (long long)s.grid_view.n[0] * s.grid_view.n[1] * s.grid_view.n[2];
    if (!s.griddf.p) s.griddf.alloc((size_t)N);
    if (!s.griddf64.p) s.griddf64.alloc((size_t)N);
    ensure_far_plan(s, st);
    zero_counters(s, st);
    ScanParams bp = build_grid_params(s);
    bp.grid = s.grid_view;
    const ScanParamsDF q = params_df(bp, s.pairsdf.p, s.df_lj_pairs, s.df_morse_pairs, s.esdf.p, s.griddf.p);
    cuda_check(launch_grid_builddf(q, s.griddf.p, s.griddf64.p, s.far_used ? &s.far : nullptr, st),
               "grid build");
    s.griddf_built = true;
}

// The grid a relaxation in precision prec reads, built if needed.
void ensure_grid_for(mafm_scan& s, int prec, cudaStream_t st, bool rebuild = false) {
    if (prec == MAFM_DF) ensure_grid_df(s, st, rebuild);
    else ensure_grid(s, prec == MAFM_FP64, st, rebuild);
}

// Cost-ordered schedule of a scan's columns, built once: proxy on the GPU,
// counting sort into 1024 buckets (descending) on the host.
Relax32Config default_config(long long n_cols, int max_terms, const mafm_run_opts* o, int n_scans);

void ensure_order(mafm_scan& s, cudaStream_t st, bool measured = false) {
    if (s.order_built && (s.order_measured || !measured)) return;
    const long long n = (long long)s.d.nx * s.d.ny;
    if (s.d.rigidgrid || s.P.n_terms == 0 || n < 2) {
        s.order_built = true;
        return;
    }
    if (!s.order_built) {
        s.order_built = true;
        DevBuf<float> w;
        w.alloc((size_t)n);
        column_cost_proxy<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(s.atoms32.p, s.P.n_terms, s.d.nx,
                                                                      s.d.ny, s.d.dx, s.d.dy, w.p);
        cuda_check(cudaGetLastError(), "cost proxy");
        std::vector<float> hw((size_t)n);
        cuda_check(cudaMemcpyAsync(hw.data(), w.p, (size_t)n * sizeof(float), cudaMemcpyDeviceToHost, st),
                   "cost proxy");
        cuda_check(cudaStreamSynchronize(st), "cost proxy");
        float wmax = 0.f;
        for (float v : hw) wmax = std::max(wmax, v);
        constexpr int kBuckets = 1024;
        std::vector<int> count(kBuckets + 1, 0);
        std::vector<int> bucket((size_t)n);
        for (long long c = 0; c < n; ++c) {
            int b = wmax > 0.f ? (int)((1.f - hw[c] / wmax) * (kBuckets - 1)) : 0;
            b = std::min(std::max(b, 0), kBuckets - 1);
            bucket[c] = b;
            count[b + 1]++;
        }
        for (int b = 0; b < kBuckets; ++b) count[b + 1] += count[b];
        std::vector<int> ord((size_t)n);
        for (long long c = 0; c < n; ++c) ord[count[bucket[c]]++] = (int)c;
        s.order.alloc((size_t)n);
        cuda_check(cudaMemcpyAsync(s.order.p, ord.data(), (size_t)n * sizeof(int), cudaMemcpyHostToDevice, st),
                   "upload order");
        cuda_check(cudaStreamSynchronize(st), "upload order");
    }
    if (!measured) return;
    // Measured costs, for plans (replayed many times): a launch takes as
    // long as its last-finishing lanes, and the proxy's order leaves lanes
    // idle at the end.  One FP32C relaxation of the scan (ordered by the
    // proxy) gives every column's FIRE steps, which track FP64's on 99.5 %
    // of the points; longest first.  The order is kept with the scan, so later
    // runs of it use it too.  On the 401 x 401 cluster: double-float launch
    // 572 -> 541 ms, FP32C 93 -> 77 ms, for one FP32C run at plan creation.
    s.order_measured = true;
    DevBuf<mafm_point> pts;
    pts.alloc((size_t)n * s.d.nz);
    BatchScan b{};
    b.p = build_params(s);
    b.out = pts.p;
    b.col_begin = 0;
    b.col_end = (int)n;
    b.n_pairs_per_eval = s.n_pairs_per_eval;
    b.has_coulomb = s.has_coulomb;
    b.order = s.order.p;
    write_batch<<<1, 1, 0, st>>>(s.batch.p, b);
    cuda_check(cudaGetLastError(), "descriptor upload");
    const Relax32Config cfg = default_config(n, b.p.n_terms_direct, nullptr, 1);
    zero_counters(s, st);
    cuda_check(launch_relax32(s.batch.p, 1, n, nullptr, cfg, s.ctr.p, st), "cost pilot");
    DevBuf<unsigned> steps;
    steps.alloc((size_t)n);
    column_steps<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(pts.p, s.d.nz, n, steps.p);
    cuda_check(cudaGetLastError(), "cost pilot");
    std::vector<unsigned> hs((size_t)n);
    cuda_check(cudaMemcpyAsync(hs.data(), steps.p, (size_t)n * sizeof(unsigned), cudaMemcpyDeviceToHost, st),
               "cost pilot");
    cuda_check(cudaStreamSynchronize(st), "cost pilot");
    std::vector<int> ord((size_t)n);
    for (long long c = 0; c < n; ++c) ord[(size_t)c] = (int)c;
    std::stable_sort(ord.begin(), ord.end(), [&](int x, int y) { return hs[(size_t)x] > hs[(size_t)y]; });
    cuda_check(cudaMemcpyAsync(s.order.p, ord.data(), (size_t)n * sizeof(int), cudaMemcpyHostToDevice, st),
               "upload order");
    cuda_check(cudaStreamSynchronize(st), "upload order");
}

bool is_device_ptr(const void* p) {
    cudaPointerAttributes a{};
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return a.type == cudaMemoryTypeDevice || a.type == cudaMemoryTypeManaged;
}

// Device-visible address of pinned (page-locked) host memory, or nullptr for
// anything else.  Kernels write points straight into such buffers (over the
// host link while they run), so no staging buffer and no copy are needed.
mafm_point* pinned_view(void* p) {
    cudaPointerAttributes a{};
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    if (a.type != cudaMemoryTypeHost || !a.devicePointer) return nullptr;
    return static_cast<mafm_point*>(a.devicePointer);
}

void check_device_errors(const RunCounters& c) {
    if (c.error_word & ERR_GRID_INDEX)
        fail(MAFM_E_RANGE, "Invalid grid point: the tip left the rigid force grid "
                           "(force_grid.cpp:236-240 stops the reference here)");
    if (c.error_word & ERR_STAGE_TIMEOUT)
        fail(MAFM_E_DEVICE, "a bounded wait on the term staging barrier expired; the kernel "
                            "ended without its results and the device context's state is "
                            "unspecified (destroy and recreate it)");
    if (c.error_word & ERR_WATCHDOG)
        fail(MAFM_E_DEVICE, "the relax kernel stopped at its watchdog time limit");
    if (c.error_word & ERR_REPAIR_WAIT)
        fail(MAFM_E_DEVICE, "a bounded wait for a near-tie column's re-relaxation entry expired; "
                            "that column holds no results");
}

// Descriptor of a double-float run over columns [cb, ce) of a scan.
BatchDF batch_df_entry(const mafm_scan& s, mafm_point* out, int cb, int ce, bool whole,
                       long long col_first) {
    BatchDF b{};
    b.p = params_df(s.P, s.pairsdf.p, s.df_lj_pairs, s.df_morse_pairs, s.esdf.p, s.griddf.p);
    b.out = out;
    b.col_first = col_first;
    b.col_begin = cb;
    b.col_end = ce;
    b.order = whole && s.order_built ? s.order.p : nullptr;
    b.n_pairs_per_eval = s.n_pairs_per_eval;
    return b;
}

// Default FP32 launch shape (the autotuner's measurements behind it: 401 x 401
// cluster, 101 x 101 graphene, 128 x 128 cluster, 256-scan batch).
// Lanes per column: the fewest that give a quarter of the resident lanes a
// column each; one lane per column does the least work per term, and small
// scans gain from a few lanes more, but not from filling every lane (101 x
// 101: G = 2 in 26.9 ms, G = 8 in 47 ms).
// Tile: one column when the scan has at least twice as many columns as there
// are groups, so that a group takes its next column from the shared queue
// when it frees up and the queue (in descending expected cost) stays shared
// until the last columns; longer tiles reserve columns for a warp's lanes
// early and leave the end of a launch statically assigned (401 x 401 at G =
// 1: 100 ms at one column per tile, 114 ms at 32).  Otherwise, and for several
// scans, one column per group, so that a warp that starts is a full warp:
// spreading few columns over every warp lowers the active lanes per issued
// instruction (201 x 201 at G = 1: 49 ms, 57-66 ms at one column per tile).
// Several scans: every scan has its own queue and a warp changes scan only
// when its scan's queue is empty, because a change waits for all its groups.
// 12 molecules (98,304 columns): 342 ms, at four columns per group 612 ms;
// with one queue through all scans, where nearly every tile was a change,
// 669 ms at four and 420 ms at one column per group; 5 small ones (12,801
// columns) 56 ms against 261 ms.
// Block: 256 threads; several scans 128, whose warps spread over more SMs when
// there are few (5 molecules 68 -> 56 ms, 12 molecules the same).
Relax32Config default_config(long long n_cols, int max_terms, const mafm_run_opts* o, int n_scans) {
    Relax32Config c{};
    c.block = (o && o->block_threads) ? o->block_threads : n_scans > 1 ? 128 : 256;
    const long long lanes_cap = (long long)sm_count() * 512;   // two 256-thread blocks per SM
    int G = 1;
    while (G < 32 && n_cols * G < lanes_cap / 4) G *= 2;
    if (max_terms <= 1) G = 1;
    c.lanes = (o && o->lanes_per_column) ? o->lanes_per_column : G;
    const bool long_queue = n_scans <= 1 && n_cols >= 2 * (lanes_cap / c.lanes);
    const int tile = (o && o->columns_per_tile) ? o->columns_per_tile : long_queue ? 1 : 32 / c.lanes;
    c.cols_per_tile = std::min(std::max(tile, 1), 1 << 16);   // queue heads are 32-bit
    // Shared slice per warp, in 32 B term slots: the paired records of up to
    // 400 terms (each kind's run padded to even: + 2); 12.9 KB per warp keeps
    // two 8-warp blocks per SM.
    c.smem_terms = std::min(std::max(max_terms, 1) + 2, 402);
    c.smem_terms = (c.smem_terms + 1) & ~1;
    c.blocks = 0;
    c.watchdog_ns = watchdog_ns_from_env();
    return c;
}

}  // namespace
}  // namespace mafm

using namespace mafm;

extern "C" {

int mafm_scan_create(int device, const mafm_scan_desc* desc, mafm_scan** out) {
    return guarded([&] {
        if (!out) fail(MAFM_E_INVALID, "null output handle");
        *out = nullptr;
        validate(desc);
        if (device >= 0) cuda_check(cudaSetDevice(device), "cudaSetDevice");
        auto* s = new mafm_scan();
        try {
            cuda_check(cudaGetDevice(&s->device), "cudaGetDevice");
            const mafm_scan_desc& d = *desc;
            s->d = d;
            s->d.pos = nullptr;
            s->d.charge = nullptr;
            s->d.type = nullptr;
            s->d.tip_pair = nullptr;
            s->d.epot = nullptr;
            s->atom_type.assign(d.type, d.type + d.n_atoms);
            ScanParams& P = s->P;
            std::memset(&P, 0, sizeof P);
            pack_terms(*s, d);
            P.atoms64 = s->atoms64.p;
            P.atoms32 = s->atoms32.p;
            P.units32 = s->units32.p;
            P.ts_mode = d.rigidgrid ? 2 : (d.use_external_potential ? 1 : 0);
            P.td_kind = d.dummy_pair.kind;
            for (int k = 0; k < 3; ++k) P.td_p[k] = d.dummy_pair.p[k];
            P.td_coul = d.tip_dummy_coulomb && d.dummy_charge != 0 && d.tip_charge != 0;
            P.td_qq = P.td_coul ? d.qbase * d.dummy_charge * d.tip_charge : 0.0;
            P.harm_k = d.harm_k;
            P.harm_r0 = d.harm_r0;
            P.tip_dummy_d = d.tip_dummy_d;
            P.nx = d.nx; P.ny = d.ny; P.nz = d.nz;
            P.tip_pbc = d.tip_pbc;
            P.dx = d.dx; P.dy = d.dy; P.dz = d.dz; P.zhigh = d.zhigh;
            std::memcpy(P.cell, d.cell, sizeof P.cell);
            if (d.tip_pbc) to_rowmajor(inv3(from_rowmajor(d.cell)), P.cell_inv);
            std::memcpy(P.offset, d.offset, sizeof P.offset);
            P.minimiser = d.minimiser;
            P.integrator = d.integrator;
            P.minterm = d.minterm;
            P.maxsteps = d.maxsteps;
            P.etol = d.etol; P.ftol = d.ftol; P.dt = d.dt;
            if (d.use_external_potential) build_external_field(*s, d);
            P.es = s->es_view;
            if (d.rigidgrid) rigid_grid_geometry(*s, d);
            P.grid = s->grid_view;
            s->ctr.alloc(1);
            s->batch.alloc(1);
            cuda_check(cudaMallocHost(&s->host_ctr, sizeof(RunCounters)), "cudaMallocHost");
            cuda_check(cudaEventCreate(&s->ev0), "cudaEventCreate");
            cuda_check(cudaEventCreate(&s->ev1), "cudaEventCreate");
        } catch (...) {
            delete s;
            throw;
        }
        *out = s;
    });
}

int mafm_scan_destroy(mafm_scan* scan) {
    if (scan) {
        cudaSetDevice(scan->device);
        delete scan;
    }
    return MAFM_OK;
}

int mafm_scan_size(const mafm_scan* scan, int64_t* n_points, int64_t* n_columns) {
    return guarded([&] {
        if (!scan) fail(MAFM_E_INVALID, "null scan");
        const int64_t cols = (int64_t)scan->d.nx * scan->d.ny;
        if (n_columns) *n_columns = cols;
        if (n_points) *n_points = cols * scan->d.nz;
    });
}

int mafm_run(mafm_scan* scan, const mafm_run_opts* opts, mafm_point* out, mafm_run_stats* stats,
             void* stream) {
    return guarded([&] {
        if (!scan || !out) fail(MAFM_E_INVALID, "null scan or output");
        cuda_check(cudaSetDevice(scan->device), "cudaSetDevice");
        cudaStream_t st = (cudaStream_t)stream;
        const long long n_cols_all = (long long)scan->d.nx * scan->d.ny;
        int cb = 0, ce = (int)n_cols_all;
        if (opts && (opts->col_begin || opts->col_end)) {
            cb = opts->col_begin;
            ce = opts->col_end;
            if (cb < 0 || ce > n_cols_all || cb > ce)
                fail(MAFM_E_INVALID, "column range [%d, %d) outside [0, %lld)", cb, ce, n_cols_all);
        }
        const int prec = opts ? opts->precision : MAFM_FP64;
        if (prec != MAFM_FP64 && prec != MAFM_FP32C && prec != MAFM_DF)
            fail(MAFM_E_INVALID, "precision %d", prec);
        const size_t n_pts = (size_t)(ce - cb) * scan->d.nz;
        if (n_pts == 0) {
            if (stats) *stats = mafm_run_stats{};
            return;
        }
        // host outputs: pinned memory is written directly, pageable memory
        // through the scan's device staging buffer
        const bool host_out = !is_device_ptr(out);
        mafm_point* const pinned = host_out ? pinned_view(out) : nullptr;
        const bool staged = host_out && !pinned;
        mafm_point* dout = pinned ? pinned : out;
        if (staged) {
            scan->stage.alloc(n_pts);
            dout = scan->stage.p;
        }
        ensure_grid_for(*scan, prec, st);
        const bool whole = cb == 0 && ce == n_cols_all;
        if (prec == MAFM_DF && whole) ensure_order(*scan, st);
        zero_counters(*scan, st);
        cuda_check(cudaEventRecord(scan->ev0, st), "cudaEventRecord");
        if (prec == MAFM_FP64) {
            ScanParams p = build_params(*scan);
            cuda_check(launch_relax64(p, dout, scan->ctr.p, nullptr, cb, ce - cb, scan->n_pairs_per_eval, true, scan->calm, st),
                       "relax64 launch");
        } else if (prec == MAFM_DF) {
            // double-float relaxation, then FP64 for the columns it lists
            BatchScan b{};
            b.p = build_params_for(*scan, true);
            b.out = dout;
            b.col_begin = cb;
            b.col_end = ce;
            b.n_pairs_per_eval = scan->n_pairs_per_eval;
            b.has_coulomb = scan->has_coulomb;
            write_batch<<<1, 1, 0, st>>>(scan->batch.p, b);
            scan->batchdf.alloc(1);
            write_batch_df<<<1, 1, 0, st>>>(scan->batchdf.p, batch_df_entry(*scan, dout, cb, ce, whole, 0));
            cuda_check(cudaGetLastError(), "descriptor upload");
            const unsigned cap = (unsigned)(ce - cb);
            scan->repair.alloc(cap);
            cuda_check(launch_relaxdf(scan->batchdf.p, scan->batch.p, 1, ce - cb, scan->ctr.p, scan->repair.p, cap,
                                      watchdog_ns_from_env(), opts ? opts->lanes_per_column : 0, st),
                       "double-float relax launch");
            cuda_check(launch_repair64(scan->batch.p, scan->repair.p, cap, scan->ctr.p, st),
                       "FP64 re-relaxation launch");
        } else {
            BatchScan b{};
            b.p = build_params(*scan);
            b.out = dout;
            b.col_begin = cb;
            b.col_end = ce;
            b.n_pairs_per_eval = scan->n_pairs_per_eval;
            b.has_coulomb = scan->has_coulomb;
            if (cb == 0 && ce == n_cols_all) {
                ensure_order(*scan, st);
                b.order = scan->order.p;
            }
            write_batch<<<1, 1, 0, st>>>(scan->batch.p, b);
            const Relax32Config cfg = default_config(ce - cb, b.p.n_terms_direct, opts, 1);
            cuda_check(launch_relax32(scan->batch.p, 1, ce - cb, nullptr, cfg, scan->ctr.p, st), "relax32 launch");
        }
        cuda_check(cudaEventRecord(scan->ev1, st), "cudaEventRecord");
        if (staged)
            cuda_check(cudaMemcpyAsync(out, dout, n_pts * sizeof(mafm_point), cudaMemcpyDeviceToHost, st),
                       "copy points to host");
        if (stats || host_out) {
            cuda_check(cudaMemcpyAsync(scan->host_ctr, scan->ctr.p, sizeof(RunCounters),
                                       cudaMemcpyDeviceToHost, st), "copy counters");
            cuda_check(cudaStreamSynchronize(st), "relax");
            const RunCounters c = *scan->host_ctr;
            if (stats) {
                float ms = 0.f;
                cudaEventElapsedTime(&ms, scan->ev0, scan->ev1);
                stats->total_steps = c.total_steps;
                stats->force_evals = c.force_evals;
                stats->pair_evals = c.pair_evals;
                stats->error_word = c.error_word;
                stats->fp64_columns = prec == MAFM_DF ? std::min<unsigned>(c.n_tie, ce - cb) : 0;
                stats->kernel_ms = ms;
            }
            check_device_errors(c);
        }
    });
}

int mafm_run_batch(mafm_scan* const* scans, int32_t n_scans, const mafm_run_opts* opts,
                   mafm_point* const* outs, mafm_run_stats* stats, void* stream) {
    return guarded([&] {
        if (!scans || !outs || n_scans <= 0) fail(MAFM_E_INVALID, "empty batch");
        const int prec = opts ? opts->precision : MAFM_FP32C;
        if (prec != MAFM_FP32C && prec != MAFM_DF)
            fail(MAFM_E_UNSUPPORTED, "batched runs use MAFM_FP32C or MAFM_DF");
        if (opts && (opts->col_begin || opts->col_end))
            fail(MAFM_E_INVALID, "column ranges are per scan; batches relax whole scans");
        const bool dfp = prec == MAFM_DF;
        cudaStream_t st = (cudaStream_t)stream;
        mafm_scan* s0 = scans[0];
        if (!s0) fail(MAFM_E_INVALID, "null scan in batch");
        cuda_check(cudaSetDevice(s0->device), "cudaSetDevice");
        const bool host_out = !is_device_ptr(outs[0]);
        std::vector<BatchScan> bs((size_t)n_scans);
        std::vector<size_t> offsets((size_t)n_scans);
        size_t total_pts = 0;
        long long max_cols = 0, total_cols = 0;
        int max_terms = 0;
        for (int i = 0; i < n_scans; ++i) {
            mafm_scan* s = scans[i];
            if (!s || !outs[i]) fail(MAFM_E_INVALID, "null scan or output %d in batch", i);
            if (s->device != s0->device) fail(MAFM_E_INVALID, "scans of one batch must share a device");
            if (is_device_ptr(outs[i]) == host_out) fail(MAFM_E_INVALID, "batch outputs mix host and device memory");
            offsets[i] = total_pts;
            const long long cols = (long long)s->d.nx * s->d.ny;
            total_pts += (size_t)cols * s->d.nz;
            max_cols = std::max(max_cols, cols);
            total_cols += cols;
            ensure_grid_for(*s, prec, st);
            ensure_order(*s, st);
            max_terms = std::max(max_terms, s->d.rigidgrid ? 0 : s->P.n_terms);
        }
        Relax32Config cfg = default_config(total_cols, max_terms, opts, n_scans);
        // host outputs: pinned ones are written directly, pageable ones staged
        std::vector<mafm_point*> pinned((size_t)n_scans, nullptr);
        bool any_staged = false;
        for (int i = 0; i < n_scans && host_out; ++i) {
            pinned[i] = pinned_view(outs[i]);
            any_staged |= !pinned[i];
        }
        if (any_staged) s0->stage.alloc(total_pts);
        for (int i = 0; i < n_scans; ++i) {
            mafm_scan* s = scans[i];
            BatchScan& b = bs[i];
            b.p = build_params_for(*s, dfp);
            b.out = !host_out ? outs[i] : pinned[i] ? pinned[i] : s0->stage.p + offsets[i];
            b.col_begin = 0;
            b.col_end = s->d.nx * s->d.ny;
            b.n_pairs_per_eval = s->n_pairs_per_eval;
            b.has_coulomb = s->has_coulomb;
            b.order = s->order.p;
        }
        set_batch_shares(bs.data(), n_scans);
        DevBuf<BatchScan> dbs;
        dbs.alloc(bs.size());
        cuda_check(cudaMemcpyAsync(dbs.p, bs.data(), bs.size() * sizeof(BatchScan), cudaMemcpyHostToDevice, st),
                   "upload batch");
        DevBuf<BatchDF> dbd;
        DevBuf<unsigned long long> rlist;
        DevBuf<unsigned> next_col;
        if (!dfp) next_col.alloc((size_t)n_scans);
        if (dfp) {
            std::vector<BatchDF> bd((size_t)n_scans);
            long long first = 0;
            for (int i = 0; i < n_scans; ++i) {
                bd[i] = batch_df_entry(*scans[i], bs[i].out, 0, bs[i].col_end, true, first);
                first += bs[i].col_end;
            }
            dbd.alloc(bd.size());
            cuda_check(cudaMemcpyAsync(dbd.p, bd.data(), bd.size() * sizeof(BatchDF),
                                       cudaMemcpyHostToDevice, st), "upload batch");
            rlist.alloc((size_t)total_cols);
            // the descriptors must reach the device before the host vector goes
            cuda_check(cudaStreamSynchronize(st), "upload batch");
        }
        zero_counters(*s0, st);
        cuda_check(cudaEventRecord(s0->ev0, st), "cudaEventRecord");
        if (dfp) {
            cuda_check(launch_relaxdf(dbd.p, dbs.p, n_scans, total_cols, s0->ctr.p, rlist.p, (unsigned)total_cols,
                                      watchdog_ns_from_env(), opts ? opts->lanes_per_column : 0, st),
                       "double-float relax launch");
            cuda_check(launch_repair64(dbs.p, rlist.p, (unsigned)total_cols, s0->ctr.p, st),
                       "FP64 re-relaxation launch");
        } else {
            cuda_check(launch_relax32(dbs.p, n_scans, total_cols, next_col.p, cfg, s0->ctr.p, st),
                       "relax32 batch launch");
        }
        cuda_check(cudaEventRecord(s0->ev1, st), "cudaEventRecord");
        if (host_out)
            for (int i = 0; i < n_scans; ++i) {
                if (pinned[i]) continue;
                const size_t np = (size_t)scans[i]->d.nx * scans[i]->d.ny * scans[i]->d.nz;
                cuda_check(cudaMemcpyAsync(outs[i], s0->stage.p + offsets[i], np * sizeof(mafm_point),
                                           cudaMemcpyDeviceToHost, st), "copy points to host");
            }
        cuda_check(cudaMemcpyAsync(s0->host_ctr, s0->ctr.p, sizeof(RunCounters), cudaMemcpyDeviceToHost, st),
                   "copy counters");
        cuda_check(cudaStreamSynchronize(st), "batch relax");
        const RunCounters c = *s0->host_ctr;
        if (stats) {
            float ms = 0.f;
            cudaEventElapsedTime(&ms, s0->ev0, s0->ev1);
            stats->total_steps = c.total_steps;
            stats->force_evals = c.force_evals;
            stats->pair_evals = c.pair_evals;
            stats->error_word = c.error_word;
            stats->fp64_columns = dfp ? (unsigned)std::min<long long>(c.n_tie, total_cols) : 0;
            stats->kernel_ms = ms;
        }
        check_device_errors(c);
    });
}

int mafm_run_columns(mafm_scan* scan, const int32_t* columns, int64_t n, mafm_point* out,
                     mafm_run_stats* stats, void* stream) {
    return guarded([&] {
        if (!scan || (n > 0 && (!columns || !out))) fail(MAFM_E_INVALID, "null argument");
        if (n < 0) fail(MAFM_E_INVALID, "negative column count");
        if (stats) *stats = mafm_run_stats{};
        if (n == 0) return;
        const long long n_cols = (long long)scan->d.nx * scan->d.ny;
        if (n > 0xffffffffll) fail(MAFM_E_RANGE, "more than 2^32 columns in one call");
        for (int64_t i = 0; i < n; ++i)
            if (columns[i] < 0 || columns[i] >= n_cols)
                fail(MAFM_E_INVALID, "column %d outside [0, %lld)", columns[i], n_cols);
        cuda_check(cudaSetDevice(scan->device), "cudaSetDevice");
        cudaStream_t st = (cudaStream_t)stream;
        const size_t n_pts = (size_t)n * scan->d.nz;
        const bool host_out = !is_device_ptr(out);
        mafm_point* const pinned = host_out ? pinned_view(out) : nullptr;
        const bool staged = host_out && !pinned;
        mafm_point* dout = pinned ? pinned : out;
        if (staged) {
            scan->stage.alloc(n_pts);
            dout = scan->stage.p;
        }
        ensure_grid(*scan, true, st);
        DevBuf<int> dlist;
        dlist.alloc((size_t)n);
        cuda_check(cudaMemcpyAsync(dlist.p, columns, (size_t)n * sizeof(int), cudaMemcpyHostToDevice, st),
                   "upload columns");
        zero_counters(*scan, st);
        cuda_check(cudaEventRecord(scan->ev0, st), "cudaEventRecord");
        cuda_check(launch_relax64(build_params(*scan), dout, scan->ctr.p, dlist.p, 0, n, scan->n_pairs_per_eval,
                                  false, scan->calm, st), "FP64 column launch");
        cuda_check(cudaEventRecord(scan->ev1, st), "cudaEventRecord");
        if (staged)
            cuda_check(cudaMemcpyAsync(out, dout, n_pts * sizeof(mafm_point), cudaMemcpyDeviceToHost, st),
                       "copy points to host");
        cuda_check(cudaMemcpyAsync(scan->host_ctr, scan->ctr.p, sizeof(RunCounters),
                                   cudaMemcpyDeviceToHost, st), "copy counters");
        cuda_check(cudaStreamSynchronize(st), "relax columns");
        const RunCounters c = *scan->host_ctr;
        if (stats) {
            float ms = 0.f;
            cudaEventElapsedTime(&ms, scan->ev0, scan->ev1);
            stats->total_steps = c.total_steps;
            stats->force_evals = c.force_evals;
            stats->pair_evals = c.pair_evals;
            stats->error_word = c.error_word;
            stats->kernel_ms = ms;
        }
        check_device_errors(c);
    });
}

int mafm_scan_sample(mafm_scan* scan, int32_t precision, int32_t what, const double* pts,
                     int64_t n, double* out) {
    return guarded([&] {
        if (!scan || (n > 0 && (!pts || !out))) fail(MAFM_E_INVALID, "null argument");
        if (n <= 0) return;
        cuda_check(cudaSetDevice(scan->device), "cudaSetDevice");
        if (precision != MAFM_FP64 && precision != MAFM_FP32C)
            fail(MAFM_E_INVALID, "unknown precision %d", precision);
        const bool fp64 = precision == MAFM_FP64;
        ensure_grid(*scan, fp64, nullptr);
        DevBuf<double> dp, dout;
        dp.alloc((size_t)n * 3);
        dout.alloc((size_t)n * 4);
        cuda_check(cudaMemcpy(dp.p, pts, (size_t)n * 3 * sizeof(double), cudaMemcpyHostToDevice), "upload points");
        zero_counters(*scan, nullptr);
        ScanParams p = build_params(*scan);
        if (fp64) cuda_check(launch_sample64(p, what, dp.p, n, dout.p, scan->ctr.p, nullptr), "sample");
        else cuda_check(launch_sample32(p, what, dp.p, n, dout.p, scan->ctr.p, nullptr), "sample");
        cuda_check(cudaMemcpy(out, dout.p, (size_t)n * 4 * sizeof(double), cudaMemcpyDeviceToHost), "download");
    });
}

int mafm_scan_grid_info(const mafm_scan* scan, int32_t what, int32_t n[3], double basis[9],
                        double origin[3]) {
    return guarded([&] {
        if (!scan) fail(MAFM_E_INVALID, "null scan");
        const GridView& g = what == 1 ? scan->es_view : scan->grid_view;
        if ((what == 1 && !scan->d.use_external_potential) || (what != 1 && !scan->d.rigidgrid))
            fail(MAFM_E_INVALID, "the scan has no such grid");
        for (int a = 0; a < 3; ++a) {
            if (n) n[a] = g.n[a];
            if (origin) origin[a] = g.origin[a];
        }
        if (basis) std::memcpy(basis, g.basis, sizeof g.basis);
    });
}

int mafm_scan_build_grid(mafm_scan* scan, int32_t precision, void* stream) {
    return guarded([&] {
        if (!scan) fail(MAFM_E_INVALID, "null scan");
        if (precision != MAFM_FP64 && precision != MAFM_FP32C && precision != MAFM_DF)
            fail(MAFM_E_INVALID, "unknown precision %d", precision);
        if (!scan->d.rigidgrid) return;
        cuda_check(cudaSetDevice(scan->device), "cudaSetDevice");
        ensure_grid_for(*scan, precision, (cudaStream_t)stream, true);
    });
}

int mafm_scan_grid_copy(const mafm_scan* scan, int32_t what, double* out) {
    return guarded([&] {
        if (!scan || !out) fail(MAFM_E_INVALID, "null argument");
        mafm_scan* s = const_cast<mafm_scan*>(scan);
        cuda_check(cudaSetDevice(s->device), "cudaSetDevice");
        const GridView* g;
        const Node64* src;
        if (what == 1) {
            if (!s->d.use_external_potential) fail(MAFM_E_INVALID, "the scan has no external field");
            g = &s->es_view;
            src = s->es64.p;
        } else {
            if (!s->d.rigidgrid) fail(MAFM_E_INVALID, "the scan has no rigid grid");
            ensure_grid(*s, true, nullptr);
            g = &s->grid_view;
            src = s->grid64.p;
        }
        const size_t N = (size_t)g->n[0] * g->n[1] * g->n[2];
        cuda_check(cudaMemcpy(out, src, N * sizeof(Node64), cudaMemcpyDeviceToHost), "download grid");
    });
}

int mafm_scan_grid_df(mafm_scan* scan, int32_t blocks[3], double* out) {
    return guarded([&] {
        if (!scan) fail(MAFM_E_INVALID, "null scan");
        if (!scan->d.rigidgrid) fail(MAFM_E_INVALID, "the scan has no rigid grid");
        cuda_check(cudaSetDevice(scan->device), "cudaSetDevice");
        ensure_grid_df(*scan, nullptr);
        if (blocks)
            for (int a = 0; a < 3; ++a) blocks[a] = scan->far_used ? scan->far.nb[a] : 0;
        if (!out) return;
        const size_t N = (size_t)scan->grid_view.n[0] * scan->grid_view.n[1] * scan->grid_view.n[2];
        cuda_check(cudaMemcpy(out, scan->griddf64.p, N * sizeof(Node64), cudaMemcpyDeviceToHost), "download grid");
    });
}

}  // extern "C"

namespace mafm {

int scan_device(const mafm_scan* s) { return s->device; }

long long scan_columns(const mafm_scan* s) { return (long long)s->d.nx * s->d.ny; }

int scan_direct_terms(const mafm_scan* s) { return s->d.rigidgrid ? 0 : s->P.n_terms; }

bool scan_fp32_ready(const mafm_scan* s) { return !s->d.rigidgrid || s->grid32_built; }

BatchScan scan_batch_entry(const mafm_scan* s, mafm_point* out) {
    BatchScan b{};
    b.p = build_params(*s);
    b.out = out;
    b.col_begin = 0;
    b.col_end = s->d.nx * s->d.ny;
    b.n_pairs_per_eval = s->n_pairs_per_eval;
    b.has_coulomb = s->has_coulomb;
    b.order = s->order_built ? s->order.p : nullptr;
    return b;
}

Relax32Config relax32_config(long long n_cols, int max_terms, const mafm_run_opts* o, int n_scans) {
    return default_config(n_cols, max_terms, o, n_scans);
}

void check_run_errors(const RunCounters& c) { check_device_errors(c); }

// Expected work of a column: its term records, and about eight records' worth
// of minimiser per evaluation (the slot machine is 13 % of a 60-atom
// cluster's relaxation, 30 records).
void set_batch_shares(BatchScan* scans, int n_scans) {
    double total = 0;
    for (int i = 0; i < n_scans; ++i) {
        BatchScan& b = scans[i];
        b.weight = (float)((b.p.n_terms_direct > 0 ? b.p.n_units : 0) + 8);
        total += (double)b.weight * (b.col_end - b.col_begin);
    }
    double sum = 0;
    for (int i = 0; i < n_scans; ++i) {
        scans[i].share_begin = total > 0 ? (float)(sum / total) : 0.f;
        sum += (double)scans[i].weight * (scans[i].col_end - scans[i].col_begin);
    }
}

}  // namespace mafm

// ---- batch plans and the autotuner -----------------------------------------

struct mafm_plan {
    int device = 0;
    int n_scans = 0;
    mafm::Relax32Config cfg{};
    mafm::DevBuf<mafm::BatchScan> list;
    mafm::DevBuf<unsigned> next_col;           // queue head of every scan (FP32C)
    mafm::DevBuf<mafm::RunCounters> ctr;
    // MAFM_DF: the double-float descriptors and the re-relaxation list
    bool dfp = false;
    long long cols = 0;
    mafm::DevBuf<mafm::BatchDF> listdf;
    mafm::DevBuf<unsigned long long> repair;
    int df_lanes = 1;                          // lanes per column of the DF kernel
    mafm::RunCounters* host_ctr = nullptr;
    ~mafm_plan() {
        if (host_ctr) cudaFreeHost(host_ctr);
    }
};

namespace mafm {
namespace {

// Descriptor list of a batch.
std::vector<BatchScan> batch_entries(mafm_scan* const* scans, int n, mafm_point* const* outs, bool df) {
    std::vector<BatchScan> bs((size_t)n);
    for (int i = 0; i < n; ++i) {
        bs[i] = scan_batch_entry(scans[i], outs[i]);
        bs[i].p = build_params_for(*scans[i], df);
    }
    set_batch_shares(bs.data(), n);
    return bs;
}

void plan_build(mafm_plan& p, mafm_scan* const* scans, int n, const mafm_run_opts* opts,
                mafm_point* const* outs, cudaStream_t st) {
    if (!scans || !outs || n <= 0) fail(MAFM_E_INVALID, "empty batch");
    const int prec = opts ? opts->precision : MAFM_FP32C;
    if (prec != MAFM_FP32C && prec != MAFM_DF) fail(MAFM_E_UNSUPPORTED, "plans run MAFM_FP32C or MAFM_DF");
    if (opts && (opts->col_begin || opts->col_end)) fail(MAFM_E_INVALID, "plans relax whole scans");
    p.dfp = prec == MAFM_DF;
    p.device = scans[0]->device;
    cuda_check(cudaSetDevice(p.device), "cudaSetDevice");
    long long cols = 0;
    int max_terms = 0;
    for (int i = 0; i < n; ++i) {
        if (!scans[i] || !outs[i]) fail(MAFM_E_INVALID, "null scan or output %d", i);
        if (scans[i]->device != p.device) fail(MAFM_E_INVALID, "scans of one plan must share a device");
        if (!is_device_ptr(outs[i])) fail(MAFM_E_INVALID, "plan outputs must be device memory");
        ensure_grid_for(*scans[i], prec, st);
        ensure_order(*scans[i], st, true);
        cols += (long long)scans[i]->d.nx * scans[i]->d.ny;
        max_terms = std::max(max_terms, scan_direct_terms(scans[i]));
    }
    p.cfg = default_config(cols, max_terms, opts, n);
    std::vector<BatchScan> bs = batch_entries(scans, n, outs, p.dfp);
    p.n_scans = n;
    p.cols = cols;
    p.list.alloc(bs.size());
    if (!p.dfp) p.next_col.alloc(bs.size());
    p.ctr.alloc(1);
    cuda_check(cudaMemcpyAsync(p.list.p, bs.data(), bs.size() * sizeof(BatchScan),
                               cudaMemcpyHostToDevice, st), "upload plan");
    std::vector<BatchDF> bd;
    if (p.dfp) {
        p.df_lanes = df_lanes_per_column(cols, opts ? opts->lanes_per_column : 0);
        long long first = 0;
        for (int i = 0; i < n; ++i) {
            bd.push_back(batch_df_entry(*scans[i], outs[i], 0, bs[i].col_end, true, first));
            first += bs[i].col_end;
        }
        p.listdf.alloc(bd.size());
        cuda_check(cudaMemcpyAsync(p.listdf.p, bd.data(), bd.size() * sizeof(BatchDF),
                                   cudaMemcpyHostToDevice, st), "upload plan");
        p.repair.alloc((size_t)cols);
    }
    cuda_check(cudaStreamSynchronize(st), "upload plan");
    if (!p.host_ctr) cuda_check(cudaMallocHost(&p.host_ctr, sizeof(RunCounters)), "cudaMallocHost");
}

void plan_launch(mafm_plan& p, cudaStream_t st) {
    cuda_check(cudaMemsetAsync(p.ctr.p, 0, sizeof(RunCounters), st), "reset counters");
    if (p.dfp) {
        cuda_check(launch_relaxdf(p.listdf.p, p.list.p, p.n_scans, p.cols, p.ctr.p, p.repair.p,
                                  (unsigned)p.cols, p.cfg.watchdog_ns, p.df_lanes, st),
                   "double-float relax launch");
        cuda_check(launch_repair64(p.list.p, p.repair.p, (unsigned)p.cols, p.ctr.p, st),
                   "FP64 re-relaxation launch");
    } else {
        cuda_check(launch_relax32(p.list.p, p.n_scans, p.cols, p.next_col.p, p.cfg, p.ctr.p, st), "relax32 launch");
    }
}

}  // namespace
}  // namespace mafm

extern "C" {

int mafm_plan_create(mafm_scan* const* scans, int32_t n_scans, const mafm_run_opts* opts,
                     mafm_point* const* outs, mafm_plan** out) {
    return guarded([&] {
        if (!out) fail(MAFM_E_INVALID, "null output handle");
        *out = nullptr;
        auto* p = new mafm_plan();
        try {
            plan_build(*p, scans, n_scans, opts, outs, nullptr);
        } catch (...) {
            delete p;
            throw;
        }
        *out = p;
    });
}

int mafm_plan_launch(mafm_plan* plan, void* stream) {
    return guarded([&] {
        if (!plan) fail(MAFM_E_INVALID, "null plan");
        plan_launch(*plan, (cudaStream_t)stream);
    });
}

int mafm_plan_stats(mafm_plan* plan, mafm_run_stats* stats, void* stream) {
    return guarded([&] {
        if (!plan || !stats) fail(MAFM_E_INVALID, "null argument");
        cudaStream_t st = (cudaStream_t)stream;
        cuda_check(cudaMemcpyAsync(plan->host_ctr, plan->ctr.p, sizeof(RunCounters),
                                   cudaMemcpyDeviceToHost, st), "copy counters");
        cuda_check(cudaStreamSynchronize(st), "plan");
        const RunCounters c = *plan->host_ctr;
        *stats = mafm_run_stats{};
        stats->total_steps = c.total_steps;
        stats->force_evals = c.force_evals;
        stats->pair_evals = c.pair_evals;
        stats->error_word = c.error_word;
        stats->fp64_columns = plan->dfp ? (unsigned)std::min<long long>(c.n_tie, plan->cols) : 0;
        check_device_errors(c);
    });
}

int mafm_plan_destroy(mafm_plan* plan) {
    if (plan) {
        cudaSetDevice(plan->device);
        delete plan;
    }
    return MAFM_OK;
}

int mafm_plan_config(const mafm_plan* plan, mafm_run_opts* opts) {
    return guarded([&] {
        if (!plan || !opts) fail(MAFM_E_INVALID, "null argument");
        *opts = mafm_run_opts{};
        opts->precision = plan->dfp ? MAFM_DF : MAFM_FP32C;
        opts->lanes_per_column = plan->dfp ? plan->df_lanes : plan->cfg.lanes;
        opts->block_threads = plan->dfp ? 128 : plan->cfg.block;
        opts->columns_per_tile = plan->dfp ? 1 : plan->cfg.cols_per_tile;
    });
}

// Time launch shapes on the scans themselves and keep the fastest: lanes per
// column first (block 256; tiles of 1 and 32 / G columns for one scan, 32 / G
// and 128 / G for batches), then block size and tile length (1, 4, 32 / G and
// 128 / G columns) around the best lane count.
int mafm_autotune(mafm_scan* const* scans, int32_t n_scans, mafm_run_opts* best, double* best_ms,
                  void* stream) {
    return guarded([&] {
        if (!scans || n_scans <= 0 || !best) fail(MAFM_E_INVALID, "empty batch");
        cudaStream_t st = (cudaStream_t)stream;
        cuda_check(cudaSetDevice(scans[0]->device), "cudaSetDevice");
        size_t total = 0;
        int max_terms = 0;
        for (int i = 0; i < n_scans; ++i) {
            if (!scans[i]) fail(MAFM_E_INVALID, "null scan %d", i);
            total += (size_t)scans[i]->d.nx * scans[i]->d.ny * scans[i]->d.nz;
            max_terms = std::max(max_terms, scan_direct_terms(scans[i]));
        }
        DevBuf<mafm_point> buf;
        buf.alloc(total);
        std::vector<mafm_point*> outs((size_t)n_scans);
        size_t off = 0;
        for (int i = 0; i < n_scans; ++i) {
            outs[i] = buf.p + off;
            off += (size_t)scans[i]->d.nx * scans[i]->d.ny * scans[i]->d.nz;
        }
        cudaEvent_t e0, e1;
        cuda_check(cudaEventCreate(&e0), "cudaEventCreate");
        cuda_check(cudaEventCreate(&e1), "cudaEventCreate");
        struct EvGuard { cudaEvent_t a, b; ~EvGuard() { cudaEventDestroy(a); cudaEventDestroy(b); } } eg{e0, e1};
        // The sweep runs on the first kTrialScans scans of a batch; the winner
        // is then timed against the default shape on the whole batch (a
        // subset of a large batch can favour another shape, with more lanes a
        // column and shorter tiles).
        constexpr int kTrialScans = 32;
        int n_time = std::min(n_scans, (int32_t)kTrialScans);
        auto time_opts = [&](const mafm_run_opts& o, bool warm = true) {
            mafm_plan p;
            plan_build(p, scans, n_time, &o, outs.data(), st);
            if (warm) plan_launch(p, st);   // warm-up: module load, attributes
            cuda_check(cudaEventRecord(e0, st), "cudaEventRecord");
            plan_launch(p, st);
            cuda_check(cudaEventRecord(e1, st), "cudaEventRecord");
            cuda_check(cudaEventSynchronize(e1), "autotune");
            float ms = 0.f;
            cudaEventElapsedTime(&ms, e0, e1);
            cuda_check(cudaMemcpy(p.host_ctr, p.ctr.p, sizeof(RunCounters), cudaMemcpyDeviceToHost), "counters");
            check_device_errors(*p.host_ctr);
            return (double)ms;
        };
        mafm_run_opts o{};
        o.precision = MAFM_FP32C;
        o.block_threads = 256;
        mafm_run_opts keep = o;
        double keep_ms = 1e300;
        const int lane_set[6] = {1, 2, 4, 8, 16, 32};
        for (int G : lane_set) {
            if (G > 1 && G > std::max(max_terms, 1)) break;
            o.lanes_per_column = G;
            // one scan: one-column tiles balance large scans, whole-warp tiles
            // keep a warp's lanes busy when there are fewer columns than
            // groups; batches: one or four columns per group
            const int t_a = n_scans > 1 ? 32 / G : 1, t_b = n_scans > 1 ? 128 / G : 32 / G;
            for (int ti = 0; ti < (t_b == t_a ? 1 : 2); ++ti) {   // G = 32: one shape
                o.columns_per_tile = ti == 0 ? t_a : t_b;
                const double ms = time_opts(o);
                if (ms < keep_ms) { keep_ms = ms; keep = o; }
            }
        }
        mafm_run_opts base = keep;
        for (int block : {128, 256}) {
            const int G = base.lanes_per_column;
            int tiles[4] = {1, 4, 32 / G, 128 / G};
            for (int ti = 0; ti < 4; ++ti) {
                const int tile = tiles[ti];
                bool seen = false;
                for (int tj = 0; tj < ti; ++tj) seen |= tiles[tj] == tile;
                if (seen) continue;
                mafm_run_opts c = base;
                c.block_threads = block;
                c.columns_per_tile = tile;
                if (block == base.block_threads && c.columns_per_tile == base.columns_per_tile) continue;
                const double ms = time_opts(c);
                if (ms < keep_ms) { keep_ms = ms; keep = c; }
            }
        }
        if (n_scans > n_time) {
            n_time = n_scans;
            mafm_run_opts def{};
            def.precision = MAFM_FP32C;
            const double ms_keep = time_opts(keep, false), ms_def = time_opts(def, false);
            keep_ms = ms_keep;
            if (ms_def < ms_keep) {
                mafm_plan p;
                plan_build(p, scans, n_scans, &def, outs.data(), st);
                keep = def;
                keep.lanes_per_column = p.cfg.lanes;
                keep.block_threads = p.cfg.block;
                keep.columns_per_tile = p.cfg.cols_per_tile;
                keep_ms = ms_def;
            }
        }
        *best = keep;
        if (best_ms) *best_ms = keep_ms;
    });
}

}  // extern "C"

extern "C" int mafm_adjoint(mafm_scan* scan, const mafm_point* pts, const double* dl_dfz,
                            mafm_grad* out, void* stream) {
    return mafm_adjoint_ex(scan, MAFM_FP64, pts, dl_dfz, out, stream);
}

extern "C" int mafm_adjoint_ex(mafm_scan* scan, int32_t precision, const mafm_point* pts,
                               const double* dl_dfz, mafm_grad* out, void* stream) {
    return guarded([&] {
        if (!scan || !pts || !dl_dfz || !out) fail(MAFM_E_INVALID, "null argument");
        if (precision != MAFM_FP64 && precision != MAFM_FP32C)
            fail(MAFM_E_INVALID, "unknown precision %d", precision);
        if (scan->d.rigidgrid)
            fail(MAFM_E_UNSUPPORTED, "gradients through a rigid force grid are not provided");
        cuda_check(cudaSetDevice(scan->device), "cudaSetDevice");
        cudaStream_t st = (cudaStream_t)stream;
        const long long npts = (long long)scan->d.nx * scan->d.ny * scan->d.nz;
        DevBuf<mafm_point> dpts;
        DevBuf<double> dw, gterm;
        const mafm_point* pp = pts;
        const double* pw = dl_dfz;
        if (!is_device_ptr(pts)) {
            dpts.alloc((size_t)npts);
            cuda_check(cudaMemcpyAsync(dpts.p, pts, npts * sizeof(mafm_point), cudaMemcpyHostToDevice, st),
                       "upload points");
            pp = dpts.p;
        }
        if (!is_device_ptr(dl_dfz)) {
            dw.alloc((size_t)npts);
            cuda_check(cudaMemcpyAsync(dw.p, dl_dfz, npts * sizeof(double), cudaMemcpyHostToDevice, st),
                       "upload weights");
            pw = dw.p;
        }
        const int nt = scan->P.n_terms;
        gterm.alloc((size_t)std::max(nt, 1) * 7);
        cuda_check(cudaMemsetAsync(gterm.p, 0, (size_t)std::max(nt, 1) * 7 * sizeof(double), st), "memset");
        zero_counters(*scan, st);
        ScanParams p = build_params(*scan);
        cuda_check(launch_adjoint(p, precision, scan->index32.p, pp, pw, npts,
                                  scan->d.qbase * scan->d.tip_charge, gterm.p,
                                  scan->ctr.p, st), "adjoint launch");
        std::vector<double> g((size_t)std::max(nt, 1) * 7);
        cuda_check(cudaMemcpyAsync(g.data(), gterm.p, g.size() * sizeof(double), cudaMemcpyDeviceToHost, st),
                   "download gradients");
        cuda_check(cudaMemcpyAsync(scan->host_ctr, scan->ctr.p, sizeof(RunCounters), cudaMemcpyDeviceToHost, st),
                   "counters");
        cuda_check(cudaStreamSynchronize(st), "adjoint");
        if (scan->host_ctr->error_word & MAFM_PT_NONFINITE)
            fail(MAFM_E_DEVICE, "singular force Jacobian at a relaxed point");
        const int na = scan->d.n_atoms, ntypes = scan->d.n_types;
        if (out->dpos) std::memset(out->dpos, 0, sizeof(double) * 3 * na);
        if (out->dcharge) std::memset(out->dcharge, 0, sizeof(double) * na);
        if (out->dpair) std::memset(out->dpair, 0, sizeof(double) * 3 * ntypes);
        for (int t = 0; t < nt; ++t) {
            const int a = t % na;
            const double* v = g.data() + (size_t)t * 7;
            if (out->dpos)
                for (int k = 0; k < 3; ++k) out->dpos[3 * a + k] += v[k];
            if (out->dpair)
                for (int k = 0; k < 3; ++k) out->dpair[3 * scan->atom_type[a] + k] += v[3 + k];
            if (out->dcharge) out->dcharge[a] += v[6];
        }
    });
}
