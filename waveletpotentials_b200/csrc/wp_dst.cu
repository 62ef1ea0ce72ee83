// wp_dst.cu -- Dirichlet Poisson solve -lap_h p = f by DST-I along x, y and z, in FP64.
//
// Reference behaviour: CuDst3D (cuDst3D.cu:202-341): odd extension into a 2(n+1)-point complex
// FFT per axis (cuFFT), orthonormal scaling sqrt(2/(n+1)), division by the eigenvalues
// sum_i (2 - 2 cos(k_i pi / (n_i + 1))) and the factor dx*dy (cuDstProj_dx, :172-200), then the
// same transforms again (the orthonormal DST-I is its own inverse).
//
// B200 design: no FFT library.  Each axis transform is a dense FP64 product with the DST-I matrix on the
// FP64 matrix units (mma.m16n8k8.f64), halved by the matrix's symmetry: with e_j = x_j + x_{N-j} and
// o_j = x_j - x_{N-j} (N = n + 1) the odd outputs are a product of half the size with e, the even ones
// with o.  It takes any extent; one kernel stages C whole lines folded in shared memory, and the
// spectral division rides on the z axis, whose two transforms are one kernel (five passes over the
// array in all).
//
// What bounds it: the FP64 units.  255^3 nodes are 2 x 128^2 x 65025 FMA = 4.3 GFLOP per transform,
// 115 us at 37 TFLOP/s, against 41 us for its 266 MB of HBM traffic.  Measured there (B200, 1965 MHz):
// 212 us per transform and 377 us for the z round trip, against 2358 us per transform of the unfolded
// product with one shared-memory load per FMA; the whole solve 14.3 -> 1.22 ms.
#include "wp_common.cuh"

#include <mutex>
#include <new>

namespace {

// Lines of one axis: element p of line (i, o) at o s_out + i s_in + p pstride.
struct Geom {
    long s_in, s_out, pstride;
    int ni, nouter;
};

// A transform of length n in folded form: `ho` odd outputs (1-based k = 1, 3, ...) of the ho folded sums,
// `he` even ones of the he folded differences; rows padded to tiles of 16, columns to steps of 8.
struct Fold {
    int n, ho, he, to, te, ko, ke;
    __host__ __device__ explicit Fold(int m)
        : n(m), ho((m + 1) / 2), he(m / 2), to((ho + 15) / 16), te((he + 15) / 16), ko((ho + 7) / 8), ke((he + 7) / 8) {}
    __host__ __device__ long words() const { return 128L * ((long)to * ko + (long)te * ke); }
};

// The folded matrices in the order the matrix instruction reads them: fragment (tile, step) is 128
// doubles, 4 consecutive ones per lane (rows lane / 4 and + 8, columns lane % 4 and + 4), so a warp
// fetches a fragment as 1 KB of consecutive 16-byte loads.  The product (j + 1)(k + 1) is reduced
// modulo 2(n + 1), so sinpi's argument is exact.
__global__ void dst_matrix_kernel(double* __restrict__ M, int n) {
    const Fold f(n);
    const long i = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (i >= f.words()) return;
    const long odd = 128L * f.to * f.ko;
    const bool even = i >= odd;
    const long q = even ? i - odd : i;
    const int steps = even ? f.ke : f.ko;
    const int e = (int)(q & 3), lane = (int)((q >> 2) & 31);
    const int step = (int)((q >> 7) % steps), tile = (int)((q >> 7) / steps);
    const int r = tile * 16 + (lane >> 2) + (e & 1) * 8, c = step * 8 + (lane & 3) + (e >> 1) * 4;
    double v = 0.0;
    if (r < (even ? f.he : f.ho) && c < (even ? f.he : f.ho)) {
        const long k = 2L * r + (even ? 2 : 1), j = c + 1;
        v = sqrt(2.0 / (n + 1)) * sinpi((double)((j * k) % (2L * (n + 1))) / (n + 1));
    }
    M[i] = v;
}

__device__ __forceinline__ void dmma(double* c, double2 a01, double2 a23, double b0, double b1) {
    asm volatile("mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
                 : "d"(a01.x), "d"(a01.y), "d"(a23.x), "d"(a23.y), "d"(b0), "d"(b1));
}

// eigenvalue 2 - 2 cos(pi (i + 1) / (n + 1)) of index i
__device__ __forceinline__ double dst_eig(int i, int n) {
    const double t = sinpi((double)(i + 1) / (2.0 * (n + 1)));
    return 4.0 * t * t;
}

enum { DST_STRIDED = 0, DST_CONTIGUOUS = 1, DST_ROUND = 2 };

// C lines per CTA, folded in shared memory as [row][C + 4] (the pitch is 4 modulo 16 doubles: the
// fragment reads of 4 rows x 8 columns meet no bank twice per half warp).  Warp w takes the row tiles
// w, w + W, ...; its TPW accumulators stay in registers until every warp has read the folded lines, so
// the result can replace them.
//   DST_STRIDED     lines along x or z: results stored straight from the accumulators
//   DST_CONTIGUOUS  lines along y: results leave through shared memory, coalesced along y
//   DST_ROUND       lines along z: transform, division by the eigenvalues, transform back
template <int C, int W, int TPW, int MODE>
__global__ void __launch_bounds__(W * 32) dst_mma_kernel(const double* src, double* dst, const double* __restrict__ M, int n,
                                                         Geom g, int nx, int ny, double scale) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr int P = C + 4, NT = W * 32, NN = C / 8;
    const Fold f(n);
    double* E = reinterpret_cast<double*>(smem_raw);
    double* O = E + (long)f.ko * 8 * P;
    double* lc = O + (long)f.ke * 8 * P;  // DST_ROUND: eigenvalue sums of the lines and of the outputs
    double* lr = lc + C;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int i0 = blockIdx.x * C;
    const long obase = (long)blockIdx.y * g.s_out;
    const int nc = min(C, g.ni - i0);

    // stage: pair (j, n - 1 - j) -> sum and difference; the middle of an odd line is its own sum
    for (int i = tid; i < C * f.ko * 8; i += NT) {
        int col, j;
        if (MODE == DST_CONTIGUOUS) { col = i / (f.ko * 8); j = i - col * (f.ko * 8); }
        else { col = i % C; j = i / C; }
        double e = 0.0, o = 0.0;
        if (col < nc && j < f.ho) {
            const double* line = src + obase + (long)(i0 + col) * g.s_in;
            e = line[(long)j * g.pstride];
            if (j < f.he) {
                const double b = line[(long)(n - 1 - j) * g.pstride];
                o = e - b;
                e += b;
            }
        }
        E[j * P + col] = e;
        if (j < f.ke * 8) O[j * P + col] = o;
    }
    if (MODE == DST_ROUND) {
        for (int i = tid; i < C; i += NT) {
            const int l = i0 + i;
            lc[i] = i < nc ? dst_eig(l / ny, nx) + dst_eig(l % ny, ny) : 1.0;
        }
        for (int i = tid; i < n; i += NT) lr[i] = dst_eig(i, n);
    }
    __syncthreads();

    double acc[TPW][NN][4];
    const int g4 = lane >> 2, t4 = lane & 3;
    // folded row of output q: q < he its sum's row, q >= n - he its difference's, the middle a sum's row
    auto slot = [&](int q) -> double* { return q < f.ho ? E + q * P : O + (n - 1 - q) * P; };
    auto product = [&]() {
#pragma unroll
        for (int t = 0; t < TPW; ++t) {
#pragma unroll
            for (int c = 0; c < NN; ++c)
#pragma unroll
                for (int e = 0; e < 4; ++e) acc[t][c][e] = 0.0;
            const int tile = warp + t * W;
            if (tile >= f.to + f.te) continue;
            const bool even = tile >= f.to;
            const int steps = even ? f.ke : f.ko;
            const double* B = (even ? O : E) + t4 * P + g4;
            const double2* A = reinterpret_cast<const double2*>(M + 128L * (even ? (long)f.to * f.ko + (long)(tile - f.to) * f.ke
                                                                                : (long)tile * f.ko)) + lane * 2;
            double2 a0 = __ldg(A), a1 = __ldg(A + 1);
            for (int s = 0; s < steps; ++s) {
                const double2 c0 = a0, c1 = a1;
                if (s + 1 < steps) {  // the next fragment's L2 latency hides behind this step's products
                    a0 = __ldg(A + 64L * (s + 1));
                    a1 = __ldg(A + 64L * (s + 1) + 1);
                }
#pragma unroll
                for (int c = 0; c < NN; ++c) dmma(acc[t][c], c0, c1, B[s * 8 * P + c * 8], B[s * 8 * P + 4 * P + c * 8]);
            }
        }
    };
    // visits the accumulators as (output index, line in the tile, value)
    auto each = [&](auto&& fn) {
#pragma unroll
        for (int t = 0; t < TPW; ++t) {
            const int tile = warp + t * W;
            if (tile >= f.to + f.te) continue;
            const bool even = tile >= f.to;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int r = (even ? tile - f.to : tile) * 16 + g4 + 8 * h;
                if (r >= (even ? f.he : f.ho)) continue;
#pragma unroll
                for (int c = 0; c < NN; ++c)
#pragma unroll
                    for (int e = 0; e < 2; ++e) fn(2 * r + (even ? 1 : 0), c * 8 + t4 * 2 + e, acc[t][c][2 * h + e]);
            }
        }
    };
    product();
    if (MODE == DST_ROUND) {
        __syncthreads();
        each([&](int q, int col, double v) { slot(q)[col] = v * (scale / (lc[col] + lr[q])); });
        __syncthreads();
        for (int i = tid; i < C * f.he; i += NT) {
            const int col = i % C, j = i / C;
            const double a = E[j * P + col], b = O[j * P + col];
            E[j * P + col] = a + b;
            O[j * P + col] = a - b;
        }
        __syncthreads();
        product();
    }
    if (MODE == DST_CONTIGUOUS) {
        __syncthreads();
        each([&](int q, int col, double v) { slot(q)[col] = v; });
        __syncthreads();
        for (int i = tid; i < nc * n; i += NT) {
            const int col = i / n, q = i - col * n;
            dst[obase + (long)(i0 + col) * g.s_in + q] = slot(q)[col];
        }
    } else {
        each([&](int q, int col, double v) {
            if (col < nc) dst[obase + (long)(i0 + col) * g.s_in + (long)q * g.pstride] = v;
        });
    }
}

template <int C, int W, int TPW, int MODE>
cudaError_t launch_axis(const double* src, double* dst, const double* M, int n, Geom g, int nx, int ny, double scale,
                        cudaStream_t s) {
    const Fold f(n);
    const size_t smem = sizeof(double) * ((size_t)(f.ko + f.ke) * 8 * (C + 4) + (MODE == DST_ROUND ? C + n : 0));
    auto k = dst_mma_kernel<C, W, TPW, MODE>;
    cudaError_t e = wp_set_smem(k, smem);
    if (e != cudaSuccess) return e;
    const int tok = wp_prof_start(s);
    k<<<dim3((g.ni + C - 1) / C, g.nouter), W * 32, smem, s>>>(src, dst, M, n, g, nx, ny, scale);
    e = cudaGetLastError();
    wp_prof_stop(tok, MODE == DST_ROUND ? "dst_round" : "dst_axis", 16.0 * n * (double)g.ni * g.nouter, s);
    return e;
}

// 32 lines and 8 warps up to 256 (74 KB of shared memory and some 120 registers: two CTAs per SM, whose loads and
// products overlap); longer lines take 16 columns so that the tile and the accumulators still fit (82 KB at 512,
// 164 KB at 1024).
template <int MODE>
cudaError_t launch_mode(const double* src, double* dst, const double* M, int n, Geom g, int nx, int ny, double scale,
                        cudaStream_t s) {
    if (n <= 256) return launch_axis<32, 8, 2, MODE>(src, dst, M, n, g, nx, ny, scale, s);
    if (n <= 512) return launch_axis<16, 16, 2, MODE>(src, dst, M, n, g, nx, ny, scale, s);
    return launch_axis<16, 16, 4, MODE>(src, dst, M, n, g, nx, ny, scale, s);
}

// Along y (and z) the lines of all planes form one run; along x they run within a plane.
cudaError_t apply_axis(const double* src, double* dst, const double* M, int DX, int DY, int DZ, char axis,
                       cudaStream_t s) {
    if (axis == 'y') return launch_mode<DST_CONTIGUOUS>(src, dst, M, DY, Geom{DY, 0, 1, DX * DZ, 1}, 0, 0, 0.0, s);
    return launch_mode<DST_STRIDED>(src, dst, M, DX, Geom{1, (long)DX * DY, DY, DY, DZ}, 0, 0, 0.0, s);
}

// x and y transforms, z transform with the spectral division and back, y and x transforms.  A CTA reads
// its lines whole before it writes them, so every pass after the first runs in place (dst may equal f).
cudaError_t solve_all(const double* f, double* dst, double* const M[3], int nx, int ny, int nz, double scale,
                      cudaStream_t s) {
    cudaError_t e = apply_axis(f, dst, M[0], nx, ny, nz, 'x', s);
    if (e == cudaSuccess) e = apply_axis(dst, dst, M[1], nx, ny, nz, 'y', s);
    if (e == cudaSuccess)
        e = launch_mode<DST_ROUND>(dst, dst, M[2], nz, Geom{1, 0, (long)nx * ny, nx * ny, 1}, nx, ny, scale, s);
    if (e == cudaSuccess) e = apply_axis(dst, dst, M[1], nx, ny, nz, 'y', s);
    if (e == cudaSuccess) e = apply_axis(dst, dst, M[0], nx, ny, nz, 'x', s);
    return e;
}

cudaError_t make_matrix(double* M, int n, cudaStream_t s) {
    const int tok = wp_prof_start(s);
    dst_matrix_kernel<<<wp_cdiv(Fold(n).words(), 256), 256, 0, s>>>(M, n);
    const cudaError_t e = cudaGetLastError();
    wp_prof_stop(tok, "dst_matrix", 8.0 * Fold(n).words(), s);
    return e;
}

}  // namespace

struct wp_dst3d {
    int n[3];
    double h[3];
    double* M[3];  // folded orthonormal DST-I matrices per axis
};

extern "C" CUWHHD_API wp_status wp_dst3d_create(wp_dst3d** out, int nx, int ny, int nz, double dx, double dy, double dz) {
    if (!out) { wp_set_error_msg("wp_dst3d_create: null handle"); return WP_ERR_INVALID_ARG; }
    *out = nullptr;
    if (nx < 1 || ny < 1 || nz < 1 || nx > 1024 || ny > 1024 || nz > 1024 || nz > 65535 || !(dx > 0) || !(dy > 0) ||
        !(dz > 0)) {
        wp_set_error_msg("wp_dst3d_create: extents must be in [1, 1024] and spacings > 0");
        return WP_ERR_INVALID_ARG;
    }
    wp_dst3d* h = new (std::nothrow) wp_dst3d();
    if (!h) return WP_ERR_INVALID_ARG;
    const int n[3] = {nx, ny, nz};
    const double hs[3] = {dx, dy, dz};
    for (int a = 0; a < 3; ++a) {
        h->n[a] = n[a];
        h->h[a] = hs[a];
        cudaError_t e = cudaMalloc((void**)&h->M[a], sizeof(double) * Fold(n[a]).words());
        if (e == cudaSuccess) e = make_matrix(h->M[a], n[a], nullptr);
        if (e != cudaSuccess) { wp_set_cuda_error(e, "dst3d create", __FILE__, __LINE__); wp_dst3d_destroy(h); return WP_ERR_CUDA; }
    }
    const cudaError_t e = cudaStreamSynchronize(nullptr);  // the solves may run on any stream
    if (e != cudaSuccess) { wp_set_cuda_error(e, "dst3d create", __FILE__, __LINE__); wp_dst3d_destroy(h); return WP_ERR_CUDA; }
    *out = h;
    return WP_OK;
}

extern "C" CUWHHD_API wp_status wp_dst3d_solve(wp_dst3d* h, double* dst, const double* f, void* stream) {
    if (!h || !dst || !f) { wp_set_error_msg("wp_dst3d_solve: null pointer"); return WP_ERR_INVALID_ARG; }
    cudaStream_t s = (cudaStream_t)stream;
    const cudaError_t e = solve_all(f, dst, h->M, h->n[0], h->n[1], h->n[2], h->h[0] * h->h[1], s);
    if (e != cudaSuccess) { wp_set_cuda_error(e, "dst3d solve", __FILE__, __LINE__); return WP_ERR_CUDA; }
    return WP_OK;
}

extern "C" CUWHHD_API wp_status wp_dst3d_destroy(wp_dst3d* h) {
    if (!h) return WP_OK;
    for (int a = 0; a < 3; ++a) if (h->M[a]) cudaFree(h->M[a]);
    wp_scratch_trim();
    delete h;
    return WP_OK;
}

// ------------------------------------------------------------------ allocation-free variant
// Same transforms as wp_dst3d_solve, with the three DST-I matrices in a file-scope device array instead
// of handle-owned allocations.  Extents are limited to WP_DST_NOALLOC_MAX_EXTENT per axis and
// WP_DST_NOALLOC_MAX_CELLS cells in total.
namespace {

constexpr int kNoAllocMaxN = WP_DST_NOALLOC_MAX_EXTENT;
constexpr long kNoAllocMaxCells = WP_DST_NOALLOC_MAX_CELLS;
constexpr long kNoAllocWords = 3L * kNoAllocMaxN * kNoAllocMaxN;

// [M_x | M_y | M_z], kNoAllocMaxN^2 doubles each (a folded matrix takes half of that)
static __device__ __align__(256) double g_dst_scratch[kNoAllocWords];

double* g_dst_scratch_ptr[64] = {nullptr};
std::mutex g_dst_scratch_mu;

// Resolves the scratch address on the current device once (cudaGetSymbolAddress, checked).  The
// address stays valid for the life of the device's primary context: after cudaDeviceReset (or any
// teardown of that context) the cached value is stale, so the entry point is not to be called on
// that device again in the same process.
cudaError_t noalloc_scratch(double** out) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> lk(g_dst_scratch_mu);
    if (!g_dst_scratch_ptr[dev]) {
        double* p = nullptr;
        e = cudaGetSymbolAddress((void**)&p, g_dst_scratch);
        if (e != cudaSuccess) return e;
        g_dst_scratch_ptr[dev] = p;
    }
    *out = g_dst_scratch_ptr[dev];
    return cudaSuccess;
}

}  // namespace

extern "C" CUWHHD_API wp_status wp_dst3d_solve_noalloc(double* dst, const double* f, int nx, int ny, int nz, double dx,
                                                       double dy, double dz, void* stream) {
    if (!dst || !f) { wp_set_error_msg("wp_dst3d_solve_noalloc: null pointer"); return WP_ERR_INVALID_ARG; }
    if (nx < 1 || ny < 1 || nz < 1 || !(dx > 0) || !(dy > 0) || !(dz > 0)) {
        wp_set_error_msg("wp_dst3d_solve_noalloc: extents must be >= 1 and spacings > 0");
        return WP_ERR_INVALID_ARG;
    }
    if (nx > kNoAllocMaxN || ny > kNoAllocMaxN || nz > kNoAllocMaxN || (long)nx * ny * nz > kNoAllocMaxCells) {
        wp_set_error_msg("wp_dst3d_solve_noalloc: grid exceeds the static scratch (at most 64 per axis and 64^3 "
                         "cells); use wp_dst3d_create/wp_dst3d_solve");
        return WP_ERR_INVALID_ARG;
    }
    double* scratch = nullptr;
    cudaError_t e = noalloc_scratch(&scratch);
    if (e != cudaSuccess) { wp_set_cuda_error(e, "dst3d noalloc scratch address", __FILE__, __LINE__); return WP_ERR_CUDA; }
    cudaStream_t s = (cudaStream_t)stream;
    double* M[3] = {scratch, scratch + (long)kNoAllocMaxN * kNoAllocMaxN, scratch + 2L * kNoAllocMaxN * kNoAllocMaxN};
    const int n[3] = {nx, ny, nz};
    for (int a = 0; a < 3 && e == cudaSuccess; ++a) e = make_matrix(M[a], n[a], s);
    if (e == cudaSuccess) e = solve_all(f, dst, M, nx, ny, nz, dx * dy, s);
    if (e != cudaSuccess) { wp_set_cuda_error(e, "dst3d noalloc solve", __FILE__, __LINE__); return WP_ERR_CUDA; }
    return WP_OK;
}
