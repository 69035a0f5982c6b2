// Per-wavelength set-up on the device that is not the hot loop: the Green's
// function spectrum (build_G, src/build_G.f90) and the T-matrix assembly
// T(:, c) = mat^H x_c (src/T_matrix.f90:260).
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <vector>

#include "ctx.h"

namespace {

constexpr double PI = 3.141592653589793;   // src/common.f90:20

// The zero-padded Green's function of build_G is even in every axis
// (A(P-k) = A(k), src/build_G.f90:34-54), so its DFT is even as well and is
// fully described by the octant 0 <= j <= P/2.  The octant is computed as a
// separable DCT-I of the spatial octant: F(j) = sum_k w_k A(k) cos(2 pi jk/P),
// w_0 = w_{P/2} = 1, otherwise 2.
__global__ void k_green_spatial(cd *A, int Hx, int Hy, int Hz, int Nx, int Ny, int Nz, double delta,
                                double mx, double my, double mz, double k) {
    const long long tot = (long long)Hx * Hy * Hz;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < tot; i += (long long)gridDim.x * blockDim.x) {
        const int x = (int)(i % Hx), y = (int)((i / Hx) % Hy), z = (int)(i / ((long long)Hx * Hy));
        cd v = cmk(0, 0);
        if (x < Nx && y < Ny && z < Nz && (x | y | z)) {
            // R = norm(nodes(:,1), nodes(:,las)) with nodes = min + delta*(k-1)
            const double dx = mx - (mx + delta * (double)x);
            const double dy = my - (my + delta * (double)y);
            const double dz = mz - (mz + delta * (double)z);
            const double R = sqrt(dx * dx + dy * dy + dz * dz);
            if (R > 0.0) {
                const double d = 4 * PI * R;
                double s, c;
                sincos(k * R, &s, &c);
                v = cmk(c / d, s / d);
            }
        }
        A[i] = v;
    }
}

// one DCT-I pass along axis `ax` (0: x, 1: y, 2: z) of an Hx*Hy*Hz octant
__global__ void k_dct1_axis(const cd *in, cd *out, int Hx, int Hy, int Hz, int ax, int P, double scale) {
    const long long tot = (long long)Hx * Hy * Hz;
    const int H = ax == 0 ? Hx : (ax == 1 ? Hy : Hz);
    const long long st = ax == 0 ? 1 : (ax == 1 ? Hx : (long long)Hx * Hy);
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < tot; i += (long long)gridDim.x * blockDim.x) {
        const int x = (int)(i % Hx), y = (int)((i / Hx) % Hy), z = (int)(i / ((long long)Hx * Hy));
        const int j = ax == 0 ? x : (ax == 1 ? y : z);
        const long long base = i - (long long)j * st;
        double re = 0, im = 0;
        for (int kk = 0; kk < H; ++kk) {
            const double w = (kk == 0 || kk == H - 1) ? 1.0 : 2.0;
            const long long m = ((long long)j * kk) % P;
            const double cs = cospi(2.0 * (double)m / (double)P) * w;
            const cd a = in[base + (long long)kk * st];
            re += cs * a.x;
            im += cs * a.y;
        }
        out[i] = cmk(re * scale, im * scale);
    }
}

// Tcols(r, c) = sum_i conj(mat(i, r)) X(i, c): 16x16 output tiles, split over
// K into partial sums that are added in order.  Bound by shared memory (two
// reads per complex multiply-add, 9 TFLOP/s); each step's elements are read
// while the one before is summed: 256 x 256 outputs over 38,592 unknowns take
// 2.26 ms, 2.52 without that, 48 x 48 89 us and 95.
constexpr int TB = 16;
// one output's sum over k0 <= i < k1 (every thread of the tile's CTA calls it)
__device__ __forceinline__ cd tile_sum(cd (&As)[TB][TB + 1], cd (&Bs)[TB][TB + 1], const cd *__restrict__ mat, long long n,
                                       int ncol, const cd *__restrict__ X, int ncb, int row0, int col0, long long k0,
                                       long long k1) {
    const int tr = threadIdx.y, tc = threadIdx.x;
    const int rr = row0 + tr, c2 = col0 + tr;
    const cd *m = rr < ncol ? mat + (long long)rr * n : nullptr, *x = c2 < ncb ? X + (long long)c2 * n : nullptr;
    // mat(kb + tc, row0 + tr) and X(kb + tc, col0 + tr), read a step ahead
    cd am, bx;
    auto load = [&](long long kb) {
        const long long kk = kb + tc;
        am = m && kk < k1 ? m[kk] : cmk(0, 0);
        bx = x && kk < k1 ? x[kk] : cmk(0, 0);
    };
    cd acc = cmk(0, 0);
    load(k0);
    for (long long kb = k0; kb < k1; kb += TB) {
        As[tc][tr] = am;
        Bs[tc][tr] = bx;
        __syncthreads();
        load(kb + TB);
#pragma unroll
        for (int kk = 0; kk < TB; ++kk) cfma_conj(acc, As[kk][tr], Bs[kk][tc]);
        __syncthreads();
    }
    return acc;
}
// splits p0, p0 + 1, ... (blockIdx.x)
__global__ void k_tgemm_partial(const cd *__restrict__ mat, long long n, int ncol, const cd *__restrict__ X,
                                int ncb, long long kchunk, int p0, cd *__restrict__ part) {
    __shared__ cd As[TB][TB + 1];
    __shared__ cd Bs[TB][TB + 1];
    const int row0 = blockIdx.y * TB, col0 = blockIdx.z * TB, r = row0 + threadIdx.y, cc = col0 + threadIdx.x;
    const long long k0 = (p0 + (long long)blockIdx.x) * kchunk;
    const cd acc = tile_sum(As, Bs, mat, n, ncol, X, ncb, row0, col0, k0, min(n, k0 + kchunk));
    if (r < ncol && cc < ncb) part[((long long)blockIdx.x * ncb + cc) * ncol + r] = acc;
}
// T = (first ? 0 : T) + the partial sums in order
__global__ void k_tgemm_reduce(const cd *part, int nsplit, int nout, bool first, cd *T) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nout) return;
    cd s = first ? cmk(0, 0) : T[i];
    for (int p = 0; p < nsplit; ++p) s = cadd(s, part[(long long)p * nout + i]);
    T[i] = s;
}
// every split of a tile in one CTA, the sums of k_tgemm_reduce in registers
__global__ void k_tgemm_whole(const cd *__restrict__ mat, long long n, int ncol, const cd *__restrict__ X, int ncb,
                              long long kchunk, cd *__restrict__ T) {
    __shared__ cd As[TB][TB + 1];
    __shared__ cd Bs[TB][TB + 1];
    const int row0 = blockIdx.x * TB, col0 = blockIdx.y * TB, r = row0 + threadIdx.y, cc = col0 + threadIdx.x;
    cd s = cmk(0, 0);
    for (long long k0 = 0; k0 < n; k0 += kchunk)
        s = cadd(s, tile_sum(As, Bs, mat, n, ncol, X, ncb, row0, col0, k0, min(n, k0 + kchunk)));
    if (r < ncol && cc < ncb) T[(long long)cc * ncol + r] = s;
}

// The split of the sums over n unknowns, a rule on n alone, so that an entry
// of T has the same bits in whatever block of rows and columns it is formed.
// 16 x 16 outputs per CTA leave a small T a few CTAs wide, so the splits go
// down to 512 unknowns: 48 x 48 outputs over 38,592 unknowns take 90 us (295
// with 4,096).
struct TSplit {
    int n;
    long long chunk;
    explicit TSplit(long long unknowns) {
        const long long want = std::min<long long>(64, std::max<long long>(1, unknowns / 512));
        chunk = ((unknowns + want - 1) / want + TB - 1) / TB * TB;
        n = (int)((unknowns + chunk - 1) / chunk);
    }
};

}  // namespace

int setup_green(scd_ctx *c, const scd_c128 *Fg) {
    NvtxRange range("Green octant");
    const long long oct = (long long)c->Hx * c->Hy * c->Hz;
    auto octant = [&](cd **p) -> int {
        if (*p || cudaMalloc(p, sizeof(cd) * oct) == cudaSuccess) return SCD_OK;
        cudaGetLastError();
        *p = nullptr;
        return set_error(c, SCD_OOM, "Green octant");
    };
    int rc = octant(&c->d_Fo);
    if (rc) return rc;
    const double scale = 1.0 / ((double)c->Px * (double)c->Py * (double)c->Pz);
    if (Fg) {
        // host Fg(2Nx,2Ny,2Nz) == (Px,Py,Pz): keep the octant, fold in the
        // 1/(8 Nx Ny Nz) of arr2vec (src/common.f90:436)
        std::vector<cd> h((size_t)oct);
        for (int z = 0; z < c->Hz; ++z)
            for (int y = 0; y < c->Hy; ++y)
                for (int x = 0; x < c->Hx; ++x) {
                    const scd_c128 v = Fg[(size_t)x + (size_t)c->Px * ((size_t)y + (size_t)c->Py * z)];
                    h[(size_t)x + (size_t)c->Hx * ((size_t)y + (size_t)c->Hy * z)] = cmk(v.re * scale, v.im * scale);
                }
        rc = check_cuda(c, cudaMemcpyAsync(c->d_Fo, h.data(), sizeof(cd) * oct, cudaMemcpyHostToDevice, c->st), "Green octant");
        if (!rc) prepare_green_yz(c);
        return rc;
    }
    // the axes' transforms go to and fro between the octant and the buffer that
    // holds it transposed in the end (fft_yz.cuh), so that the first matvec
    // neither allocates nor fills one
    if ((rc = octant(&c->d_Fyz))) return rc;
    cd *const tmp = c->d_Fyz;
    const int blocks = (int)std::min<long long>((oct + 255) / 256, 65535);
    k_green_spatial<<<blocks, 256, 0, c->st>>>(c->d_Fo, c->Hx, c->Hy, c->Hz, c->Nx, c->Ny, c->Nz, c->d.delta,
                                               c->d.min_coord[0], c->d.min_coord[1], c->d.min_coord[2], c->k);
    k_dct1_axis<<<blocks, 256, 0, c->st>>>(c->d_Fo, tmp, c->Hx, c->Hy, c->Hz, 0, c->Px, 1.0);
    k_dct1_axis<<<blocks, 256, 0, c->st>>>(tmp, c->d_Fo, c->Hx, c->Hy, c->Hz, 1, c->Py, 1.0);
    k_dct1_axis<<<blocks, 256, 0, c->st>>>(c->d_Fo, tmp, c->Hx, c->Hy, c->Hz, 2, c->Pz, scale);
    rc = check_cuda(c, cudaMemcpyAsync(c->d_Fo, tmp, sizeof(cd) * oct, cudaMemcpyDeviceToDevice, c->st), "Green");
    const bool kept = !rc && prepare_green_yz(c);
    if (!rc) rc = check_cuda(c, cudaStreamSynchronize(c->st), "Green");
    if (!kept) { cudaFree(c->d_Fyz); c->d_Fyz = nullptr; }
    return rc;
}

int launch_T_assemble(scd_ctx *c, const cd *d_mat, int ncol, int col0, int ncb, const cd *d_X, cd *d_T) {
    const long long n = c->n;
    const TSplit split(n);
    // the partial sums of as many columns at a time as there is memory for (64
    // splits of 1,350 x 1,350 outputs are 1.9 GB)
    cd *part = nullptr;
    int nb = ncb;
    while (cudaMallocAsync(&part, sizeof(cd) * (size_t)split.n * ncol * nb, c->st) != cudaSuccess) {
        cudaGetLastError();
        if (nb <= 1) return set_error(c, SCD_OOM, "partial sums of T");
        nb = (nb + 1) / 2;
    }
    for (int c0 = col0; c0 < col0 + ncb; c0 += nb) {
        const int bc = std::min(nb, col0 + ncb - c0);
        dim3 grid(split.n, (ncol + TB - 1) / TB, (bc + TB - 1) / TB);
        k_tgemm_partial<<<grid, dim3(TB, TB), 0, c->st>>>(d_mat, n, ncol, d_X + (size_t)c0 * n, bc, split.chunk, 0, part);
        k_tgemm_reduce<<<(ncol * bc + 255) / 256, 256, 0, c->st>>>(part, split.n, ncol * bc, true, d_T + (size_t)c0 * ncol);
        c->launches += 2;
    }
    cudaFreeAsync(part, c->st);
    return SCD_OK;
}


// ------------------------------------------------------------ no allocation
// scd_T_assemble_noalloc: the same split-K assembly T = mat^H X for callers
// that must not allocate device memory -- e.g. a Fortran host whose device
// arrays all come from its own allocator (CUDA Fortran `device` arrays,
// OpenACC data regions), where a cudaMalloc inside the library would hold
// memory outside that allocator's accounting and synchronise the device.
// The split-K partial sums live in this fixed file-scope array instead of a
// cudaMallocAsync buffer; where it does not hold all splits, they are summed a
// few at a time, with the bits of launch_T_assemble.
#define SCD_NOALLOC_SCRATCH (1 << 18)   // complex doubles: 4 MiB per device
static __device__ __align__(256) cd g_noalloc_scratch[SCD_NOALLOC_SCRATCH];

// device address of g_noalloc_scratch per device; the symbol name in host
// code is only a host-side stand-in, so the address is looked up once per
// device with that device current (first call on the device).  Atomic, as
// host threads may make their first calls at the same time; both store the
// same address.
static std::atomic<cd *> g_noalloc_ptr[128];

extern "C" SCD_API int scd_T_assemble_noalloc(const scd_c128 *mat, int64_t n, int32_t ncol, const scd_c128 *X,
                                              int32_t ncb, scd_c128 *T, void *stream) {
    if (!mat || !X || !T || n < 1 || ncol < 1 || ncb < 1) return SCD_BAD_ARG;
    if ((int64_t)ncol * ncb > SCD_NOALLOC_SCRATCH) return SCD_BAD_ARG;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 128) return SCD_NO_DEVICE;
    // an error left pending by an earlier call of the caller's is not this
    // call's: report it without launching and leave it for the caller to read
    if (cudaPeekAtLastError() != cudaSuccess) return SCD_CUDA_ERROR;
    cd *part = g_noalloc_ptr[dev].load(std::memory_order_acquire);
    if (!part) {
        if (cudaGetSymbolAddress((void **)&part, g_noalloc_scratch) != cudaSuccess || !part) {
            cudaGetLastError();   // this lookup's own error
            return SCD_CUDA_ERROR;
        }
        g_noalloc_ptr[dev].store(part, std::memory_order_release);
    }
    cudaStream_t st = (cudaStream_t)stream;
    // as many splits at a time as the scratch holds, shared evenly over the
    // passes (a full scratch is 1,024 CTAs' tiles, one wave); every partial entry
    // is written before it is read, so nothing needs clearing between calls.
    // Where the scratch holds one split, the 513 tiles or more fill the SMs by
    // themselves: 500 x 500 over 9,000 unknowns take 1.88 ms (2.36 in a pass per
    // split, without the reads ahead; 1.91 so in one pass); 300 x 300, two splits
    // a pass, 759 us against 828 in one CTA a tile.
    const TSplit split(n);
    const int nout = ncol * ncb, most = SCD_NOALLOC_SCRATCH / nout;
    const int passes = (split.n + most - 1) / most, per = (split.n + passes - 1) / passes;
    const dim3 tiles((ncol + TB - 1) / TB, (ncb + TB - 1) / TB);
    auto refused = [] {
        if (cudaPeekAtLastError() == cudaSuccess) return false;
        cudaGetLastError();   // this launch's own error
        return true;
    };
    if (most == 1 && split.n > 1) {
        k_tgemm_whole<<<tiles, dim3(TB, TB), 0, st>>>((const cd *)mat, n, ncol, (const cd *)X, ncb, split.chunk, (cd *)T);
        return refused() ? SCD_CUDA_ERROR : SCD_OK;
    }
    for (int p0 = 0; p0 < split.n; p0 += per) {
        const int np = std::min(per, split.n - p0);
        k_tgemm_partial<<<dim3(np, tiles.x, tiles.y), dim3(TB, TB), 0, st>>>((const cd *)mat, n, ncol, (const cd *)X, ncb,
                                                                            split.chunk, p0, part);
        if (refused()) return SCD_CUDA_ERROR;
        k_tgemm_reduce<<<(nout + 255) / 256, 256, 0, st>>>(part, np, nout, p0 == 0, (cd *)T);
        if (refused()) return SCD_CUDA_ERROR;
    }
    return SCD_OK;
}
