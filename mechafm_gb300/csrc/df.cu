// df.cu — frequency-shift images from Fz stacks on the GPU.
//
// The reference turns the scan files into frequency-shift images with its
// post-processing script (simple-vafm-image.py:77-89, 204), Giessibl's
// small-amplitude formula: for every window of nosc consecutive heights
//   df(x, y) = -fshiftfac * dz * sum_m W[m] * Fz(x, y, z_m),
//   fshiftfac = f0 / (2 k) * 2 / (pi A^2),   W(z) = z / sqrt(|A^2 - z^2|)
// on the offsets z = (-zosc[L-1], ..., -zosc[2], zosc[0], ..., zosc[L-1])
// with zosc = 0, dz, 2 dz, ... (L = ceil((A + dz) / dz) values, numpy's
// arange), both end points dropped.  Heights are taken in ascending z (the
// script sorts the scan file names); window s covers heights s .. s+nosc-1.
// The operator is linear in Fz, so its adjoint is the transposed sum
// (mafm_df_adjoint), used to take gradients of a loss on df images.
#include <algorithm>
#include <cmath>
#include <vector>

#include "mafm_internal.h"

namespace mafm {
namespace {

constexpr int kMaxW = 4096;

// Python's float floor division and modulo (the script's `//` and `%`):
// both go through fmod, so 0.5 // 0.1 is 4.0 although floor(0.5 / 0.1) is 5.
double py_floordiv(double a, double b) {
    double mod = std::fmod(a, b);
    double div = (a - mod) / b;
    if (mod != 0 && ((b < 0) != (mod < 0))) div -= 1.0;
    if (div != 0) {
        double f = std::floor(div);
        if (div - f > 0.5) f += 1.0;
        return f;
    }
    return std::copysign(0.0, a / b);
}

double py_mod(double a, double b) {
    double mod = std::fmod(a, b);
    if (mod != 0) {
        if ((b < 0) != (mod < 0)) mod += b;
    } else {
        mod = std::copysign(0.0, b);
    }
    return mod;
}

// Weights and prefactor exactly as the script builds them.
void df_weights(const mafm_df_params& prm, double dz, std::vector<double>& w, double& fac) {
    double amplitude = prm.amplitude;
    const double k = prm.k_cantilever, f0 = prm.f0;
    fac = (f0 / (2 * k)) * (2 / (3.14159265358979323846 * amplitude * amplitude));
    // ampcut = (1+(amplitude/dz))%(1+(amplitude//dz)): W is infinite at +-A
    const double ampcut = py_mod(1 + (amplitude / dz), 1 + py_floordiv(amplitude, dz));
    if (ampcut < 0.01) amplitude += dz / 2;
    const double stop = amplitude + dz;
    const long long L = (long long)std::ceil((stop - 0.0) / dz);
    if (L < 3 || L > kMaxW) fail(MAFM_E_RANGE, "frequency-shift window of %lld heights", L);
    std::vector<double> zosc((size_t)L);
    for (long long i = 0; i < L; ++i) zosc[i] = 0.0 + i * dz;
    std::vector<double> full;
    for (long long i = L - 1; i > 1; --i) full.push_back(-zosc[i]);
    for (long long i = 0; i < L; ++i) full.push_back(zosc[i]);
    w.clear();
    for (size_t i = 1; i + 1 < full.size(); ++i) {
        const double z = full[i];
        w.push_back(z / std::sqrt(std::fabs(amplitude * amplitude - z * z)));
    }
}

// Window weights as a kernel argument: no device buffer, no upload and no
// allocation on the call path.  128 weights hold every height step down to
// about 0.008 A at the default amplitude; longer windows read a device buffer.
constexpr int kInlineW = 128;
struct InlineW {
    double w[kInlineW];
};

// Columns (x, y) a block handles, and its threads.  An Fz stack has z fastest
// and an image stack x, y fastest, so a block moves a tile of 32 columns
// through shared memory and both sides are read and written in whole
// sectors.  On 401 x 401 x 41 these kernels take 87.7 us (images) and 92.8 us
// (transpose); one thread per value with the stack read in place took 90.5
// and 105 us.  What bounds them is the FP64 pipe: one FMA per weight and value,
// 4.2e7 of them at that size, and an SM takes a warp's FMA every 19 cycles.
// The whole pass, images and gradient from Python (stream-ordered calls), went from
// 852 to 211 us there and from 654 to 212 us at 64 x 64 x 41: two allocations, two
// frees and a wait of each call are gone.
constexpr int kTileXY = 32;
constexpr int kTileThreads = 256;

// out[s][x][y] = -scale sum_m w[m] fz[x][y][nz - 1 - s - m].  fz is read with a
// stride (in doubles) so that it can be the force[2] field of mafm_point
// records.  Rows of the tile have an odd length, so that the 32 columns of a
// warp fall into different banks.
__global__ void __launch_bounds__(kTileThreads) df_kernel(const double* fz, long long stride,
                                                          long long nxy, int nz, const __grid_constant__ InlineW iw,
                                                          const double* wbuf, int nosc, double scale,
                                                          double* out, int nshift) {
    extern __shared__ __align__(16) double df_tile[];
    const double* w = wbuf ? wbuf : iw.w;
    const int pitch = nz | 1;
    const long long xy0 = (long long)blockIdx.x * kTileXY;
    const int cols = (int)min((long long)kTileXY, nxy - xy0);
    for (int i = threadIdx.x; i < cols * nz; i += kTileThreads) {
        const int c = i / nz, k = i - c * nz;
        df_tile[c * pitch + k] = fz[(xy0 * nz + i) * stride];
    }
    __syncthreads();
    const int c = threadIdx.x % kTileXY;
    if (c >= cols) return;
    for (int s = threadIdx.x / kTileXY; s < nshift; s += kTileThreads / kTileXY) {
        const double* f = df_tile + c * pitch + (nz - 1 - s);   // ascending z: level index falls
        double acc = 0;
        for (int m = 0; m < nosc; ++m) acc += w[m] * f[-m];
        out[(long long)s * nxy + xy0 + c] = -scale * acc;
    }
}

// Transpose: g_fz[x][y][k] = -scale * sum_{s,m: s+m = nz-1-k} w[m] g_df[s][x][y].
__global__ void __launch_bounds__(kTileThreads) df_adjoint_kernel(const double* gdf, long long nxy, int nz,
                                                                  const __grid_constant__ InlineW iw, const double* wbuf,
                                                                  int nosc, double scale, double* gfz,
                                                                  int nshift) {
    extern __shared__ __align__(16) double df_tile[];
    const double* w = wbuf ? wbuf : iw.w;
    double* res = df_tile + (size_t)nshift * kTileXY;   // results, one odd-length row per column
    const int pitch = nz | 1;
    const long long xy0 = (long long)blockIdx.x * kTileXY;
    const int cols = (int)min((long long)kTileXY, nxy - xy0);
    const int c = threadIdx.x % kTileXY, row = threadIdx.x / kTileXY;
    constexpr int kRows = kTileThreads / kTileXY;
    if (c < cols)
        for (int s = row; s < nshift; s += kRows) df_tile[s * kTileXY + c] = gdf[(long long)s * nxy + xy0 + c];
    __syncthreads();
    if (c < cols)
        for (int h = row; h < nz; h += kRows) {
            double acc = 0;
            const int m1 = min(nosc - 1, h);
            for (int m = max(0, h - nshift + 1); m <= m1; ++m) acc += w[m] * df_tile[(h - m) * kTileXY + c];
            res[c * pitch + nz - 1 - h] = -scale * acc;
        }
    __syncthreads();
    for (int i = threadIdx.x; i < cols * nz; i += kTileThreads) {
        const int cc = i / nz;
        gfz[xy0 * nz + i] = res[cc * pitch + (i - cc * nz)];
    }
}

// The same sums with one thread per value, for stacks of so many heights that
// a 32-column tile does not fit into shared memory.
__global__ void df_tall_kernel(const double* fz, long long stride, long long nxy, int nz, const double* w,
                               int nosc, double scale, double* out, int nshift) {
    const long long tid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (tid >= (long long)nshift * nxy) return;
    const int s = (int)(tid / nxy);
    const long long xy = tid % nxy;
    double acc = 0;
    for (int m = 0; m < nosc; ++m) acc += w[m] * fz[(xy * nz + (nz - 1 - s - m)) * stride];
    out[tid] = -scale * acc;
}

__global__ void df_tall_adjoint_kernel(const double* gdf, long long nxy, int nz, const double* w, int nosc,
                                       double scale, double* gfz, int nshift) {
    const long long tid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (tid >= nxy * nz) return;
    const int h = nz - 1 - (int)(tid % nz);
    const long long xy = tid / nz;
    double acc = 0;
    for (int m = 0; m < nosc; ++m) {
        const int s = h - m;
        if (s >= 0 && s < nshift) acc += w[m] * gdf[(long long)s * nxy + xy];
    }
    gfz[tid] = -scale * acc;
}

// Shared memory of a tile; 48 KB is what a block gets without opting in.
size_t tile_bytes(bool adjoint, int nz, int nshift) {
    return sizeof(double) * kTileXY * ((size_t)(nz | 1) + (adjoint ? (size_t)nshift : 0));
}
constexpr size_t kTileLimit = 48 * 1024;

bool dev_ptr(const void* p) {
    cudaPointerAttributes a{};
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return a.type == cudaMemoryTypeDevice || a.type == cudaMemoryTypeManaged;
}

// Memory the host can read in place (managed memory is on the device too).
bool host_readable(const void* p) {
    cudaPointerAttributes a{};
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return true;
    }
    return a.type != cudaMemoryTypeDevice;
}

mafm_df_params defaults(const mafm_df_params* p) {
    if (p) return *p;
    mafm_df_params d;
    d.amplitude = 0.50;                 // simple-vafm-image.py:78
    d.k_cantilever = 1800 * 1.438978;   // :79 (N/m in kcal/mol/A^2)
    d.f0 = 25.000e3;                    // :80
    return d;
}

}  // namespace
}  // namespace mafm

using namespace mafm;

extern "C" int mafm_df_weights(const mafm_df_params* params, double dz, double* w, int32_t cap,
                               int32_t* n_w, double* fshiftfac) {
    return guarded([&] {
        if (dz <= 0) fail(MAFM_E_INVALID, "dz must be positive");
        std::vector<double> ww;
        double fac;
        df_weights(defaults(params), dz, ww, fac);
        if (n_w) *n_w = (int32_t)ww.size();
        if (fshiftfac) *fshiftfac = fac;
        if (w) {
            if (cap < (int32_t)ww.size()) fail(MAFM_E_RANGE, "weight buffer of %d < %zu", cap, ww.size());
            for (size_t i = 0; i < ww.size(); ++i) w[i] = ww[i];
        }
    });
}

// Host or device buffers, one stream.  wait: the result is complete on return.
static int df_apply(bool wait, bool adjoint, const double* in, int64_t stride, int32_t nx, int32_t ny, int32_t nz,
                    double dz, const mafm_df_params* params, double* out, void* stream) {
    return guarded([&] {
        if (!in || !out || nx < 1 || ny < 1 || nz < 1) fail(MAFM_E_INVALID, "bad df arguments");
        std::vector<double> ww;
        double fac;
        df_weights(defaults(params), dz, ww, fac);
        const int nosc = (int)ww.size();
        const int nshift = nz - nosc;
        if (nshift <= 0) fail(MAFM_E_RANGE, "%d heights are fewer than the %d-height window", nz, nosc);
        cudaStream_t st = (cudaStream_t)stream;
        const long long nfz = (long long)nx * ny * nz, ndf = (long long)nshift * nx * ny;
        const long long n_in = adjoint ? ndf : (nfz - 1) * (stride > 0 ? stride : 1) + 1;
        const long long n_out = adjoint ? nfz : ndf;
        double *din = nullptr, *dout = nullptr, *dw = nullptr;
        struct Frees {
            std::vector<void*> p;
            ~Frees() { for (void* q : p) cudaFree(q); }
        } frees;
        auto dalloc = [&](double** p, long long n) {
            cuda_check(cudaMalloc(p, (size_t)n * sizeof(double)), "cudaMalloc");
            frees.p.push_back(*p);
        };
        const double* src = in;
        if (!dev_ptr(in)) {
            dalloc(&din, n_in);
            cuda_check(cudaMemcpyAsync(din, in, (size_t)n_in * sizeof(double), cudaMemcpyHostToDevice, st), "upload");
            src = din;
        }
        const bool host_out = !dev_ptr(out);
        double* dst = out;
        if (host_out) {
            dalloc(&dout, n_out);
            dst = dout;
        }
        const double scale = fac * dz;
        const long long nxy = (long long)nx * ny;
        const size_t smem = tile_bytes(adjoint, nz, nshift);
        const bool tiled = smem <= kTileLimit;
        InlineW iw{};
        const bool inl = tiled && nosc <= kInlineW;
        if (inl) {
            std::copy(ww.begin(), ww.end(), iw.w);
        } else {
            dalloc(&dw, nosc);
            cuda_check(cudaMemcpyAsync(dw, ww.data(), nosc * sizeof(double), cudaMemcpyHostToDevice, st), "upload");
        }
        const long long n_blocks = tiled ? (nxy + kTileXY - 1) / kTileXY : (n_out + 255) / 256;
        if (n_blocks > 0x7fffffffll) fail(MAFM_E_RANGE, "frequency-shift stack of %d x %d x %d is too large", nx, ny, nz);
        const unsigned blocks = (unsigned)n_blocks;
        const long long sd = stride > 0 ? stride : 1;
        if (tiled && adjoint) df_adjoint_kernel<<<blocks, kTileThreads, smem, st>>>(src, nxy, nz, iw, dw, nosc, scale, dst, nshift);
        else if (tiled) df_kernel<<<blocks, kTileThreads, smem, st>>>(src, sd, nxy, nz, iw, dw, nosc, scale, dst, nshift);
        else if (adjoint) df_tall_adjoint_kernel<<<blocks, 256, 0, st>>>(src, nxy, nz, dw, nosc, scale, dst, nshift);
        else df_tall_kernel<<<blocks, 256, 0, st>>>(src, sd, nxy, nz, dw, nosc, scale, dst, nshift);
        cuda_check(cudaGetLastError(), "df launch");
        if (host_out)
            cuda_check(cudaMemcpyAsync(out, dst, (size_t)n_out * sizeof(double), cudaMemcpyDeviceToHost, st), "download");
        // A stream-ordered call waits all the same where host (or managed) memory
        // takes part, and before buffers of its own are freed.
        if (wait || !frees.p.empty() || host_readable(in) || host_readable(out))
            cuda_check(cudaStreamSynchronize(st), "df");
    });
}

extern "C" int mafm_df(const double* fz, int64_t stride, int32_t nx, int32_t ny, int32_t nz, double dz,
                       const mafm_df_params* params, double* df, void* stream) {
    return df_apply(true, false, fz, stride, nx, ny, nz, dz, params, df, stream);
}

extern "C" int mafm_df_adjoint(const double* g_df, int32_t nx, int32_t ny, int32_t nz, double dz,
                               const mafm_df_params* params, double* g_fz, void* stream) {
    return df_apply(true, true, g_df, 1, nx, ny, nz, dz, params, g_fz, stream);
}

extern "C" int mafm_df_async(const double* fz, int64_t stride, int32_t nx, int32_t ny, int32_t nz, double dz,
                             const mafm_df_params* params, double* df, void* stream) {
    return df_apply(false, false, fz, stride, nx, ny, nz, dz, params, df, stream);
}

extern "C" int mafm_df_adjoint_async(const double* g_df, int32_t nx, int32_t ny, int32_t nz, double dz,
                                     const mafm_df_params* params, double* g_fz, void* stream) {
    return df_apply(false, true, g_df, 1, nx, ny, nz, dz, params, g_fz, stream);
}
