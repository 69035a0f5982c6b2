// The y and z passes of the pruned FFT convolution fused into one kernel,
// one CTA per (x column, grid): the (y, z) plane of an x-transformed grid is
// transformed along y (length PY, zero padded from Ny) into shared memory,
// then along z (length PZ, zero padded from Nz), multiplied by the Green
// spectrum, transformed back along z and y, and its Ny x Nz corner is written
// back in place.  Replaces the three passes y forward, z (forward, x Fg,
// inverse), y inverse (FFT3d_2 / IFFT3d_2, src/possu.f90:140-289, with the
// product of src/gmres_module.f90:104...): the plane crosses HBM once each way
// instead of six times, and the z lines are never strided in global memory.
//
// Global layout of an x-transformed grid (rg = 4 r + g): Wt[rg][x][z][y],
// x < Px, z < Nz, y < Ny (y fastest), written by the x forward pass and read
// by the x inverse pass.  The Green spectrum is the octant of Fg (even in
// every axis) pre-scaled by 1/(Px Py Pz), transposed for this pass to
// Fyz[(fx Hy + fy) Hz + fz], H = P/2 + 1.
//
// Shared memory (elements of C): twiddles twy[PY], twz[PZ]; the plane
// A[Nz][LSY], whose column c = (p + PER b) T + t of row z holds ky = t PER + p
// + N1 b (so that a line's threads store consecutive columns); one exchange
// buffer per warp.  Lines are transformed in registers (fft_line.cuh): a y
// line goes from global memory to the plane, a z line from a column of the
// plane through the Green product and back, a y line from the plane to global
// memory, each with one exchange per transform.  A z line reads and writes its
// own column only, so the CTA synchronises twice in all.
//
// Bound by shared memory and instruction issue about equally.  Before, the
// lines lived in shared memory between their phases (14 accesses an element
// where 5 remain) and only 64, 80, 96, 128 and 192 had a transform, so that a
// 22-node axis ran at 64 instead of 48.  32 complex64 right-hand sides: grid
// 22 x 20 x 18 156 -> 51 us, 46 x 40 x 28 585 -> 294; 16 in FP64, 24 x 24 x 24
// 242 -> 83; one in FP64, 64 x 54 x 40 126 -> 73.
//
// The phases are host-callable so that a host program can run the whole pass
// line by line and check it (tests/fft_yz_check.cu).
#pragma once
#include <algorithm>

#include "common.cuh"
#include "fft_line.cuh"

constexpr int YZ_THREADS = 256;   // most threads of a CTA

// plane row stride: 4 mod 8, so that four threads of four lines fall in
// distinct banks along the rows (y) and across them (z)
constexpr int yz_row(int PY) { return (PY + 7) / 8 * 8 + 4; }
template <int P> struct YzLine {
    static constexpr int LS = yz_row(P);
};

struct YzDims {
    int Nx, Ny, Nz, NzR;   // grid nodes, Nz rounded up to a multiple of 8
    int Px;                // x FFT length
    int Hx, Hy, Hz;        // octant sizes P/2 + 1
};

SCD_HD int yz_fold(int u, int P) { return u <= P - u ? u : P - u; }
SCD_HD int yz_round8(int n) { return (n + 7) & ~7; }

// exchange elements of a warp
constexpr int yz_exchange(int PY, int PZ) { return half_ew(PY) > half_ew(PZ) ? half_ew(PY) : half_ew(PZ); }
template <int PY, int PZ> constexpr int yz_ex() { return yz_exchange(PY, PZ); }
// shared-memory elements of a CTA of `threads` for planes of nz rows; the host
// pass (yz_plane_host) is one warp's
constexpr long long yz_elems(int PY, int PZ, int nz, int threads) {
    return (long long)PY + PZ + (long long)nz * yz_row(PY) + (long long)(threads / 32) * yz_exchange(PY, PZ);
}
template <int PY, int PZ>
SCD_HD long long yz_smem_elems(int nz, int threads = 32) { return yz_elems(PY, PZ, nz, threads); }

// ky of plane column c
template <int PY> SCD_HD int yz_ky(int c) {
    using H = HalfLine<PY>;
    const int t = c % H::T, q = c / H::T;
    return t * H::PER + q % H::PER + H::N1 * (q / H::PER);
}

// thread t of the y line of row z: global row -> x
template <int PY, typename C>
SCD_HD void yz_y_load(C (&x)[HalfLine<PY>::M], const C *Wp, int z, int t, bool live, const YzDims &D) {
    using H = HalfLine<PY>;
    ct_for<H::M>([&](auto k) {
        const int y = t + H::T * k;
        x[k] = live && y < D.Ny ? Wp[(long long)z * D.Ny + y] : czero<C>();
    });
}
template <int PY, typename C>
SCD_HD void yz_y_put(const C (&u)[HalfLine<PY>::PER][HalfLine<PY>::T], C *A, int z, int t) {
    using H = HalfLine<PY>;
    ct_for<H::PER>([&](auto p) {
        ct_for<H::T>([&](auto b) { A[z * YzLine<PY>::LS + (p + H::PER * b) * H::T + t] = u[p][b]; });
    });
}
template <int PY, typename C>
SCD_HD void yz_y_get(C (&u)[HalfLine<PY>::PER][HalfLine<PY>::T], const C *A, int z, int t, bool live) {
    using H = HalfLine<PY>;
    ct_for<H::PER>([&](auto p) {
        ct_for<H::T>([&](auto b) { u[p][b] = live ? A[z * YzLine<PY>::LS + (p + H::PER * b) * H::T + t] : czero<C>(); });
    });
}
template <int PY, typename C>
SCD_HD void yz_y_store(const C (&x)[HalfLine<PY>::M], C *Wp, int z, int t, const YzDims &D) {
    using H = HalfLine<PY>;
    ct_for<H::M>([&](auto k) {
        const int y = t + H::T * k;
        if (y < D.Ny) Wp[(long long)z * D.Ny + y] = x[k];
    });
}
// thread t of the z line of plane column c
template <int PY, int PZ, typename C>
SCD_HD void yz_z_load(C (&x)[HalfLine<PZ>::M], const C *A, int c, int t, bool live, const YzDims &D) {
    using H = HalfLine<PZ>;
    ct_for<H::M>([&](auto k) {
        const int z = t + H::T * k;
        x[k] = live && z < D.Nz ? A[z * YzLine<PY>::LS + c] : czero<C>();
    });
}
template <int PY, int PZ, typename C>
SCD_HD void yz_z_store(const C (&x)[HalfLine<PZ>::M], C *A, int c, int t, const YzDims &D) {
    using H = HalfLine<PZ>;
    ct_for<H::M>([&](auto k) {
        const int z = t + H::T * k;
        if (z < D.Nz) A[z * YzLine<PY>::LS + c] = x[k];
    });
}
// the Green values of thread t's part of a z line, Fr = the line's octant row
template <int PZ, typename C>
SCD_HD void yz_green_load(C (&f)[HalfLine<PZ>::PER][HalfLine<PZ>::T], const C *Fr, int t) {
    using H = HalfLine<PZ>;
    ct_for<H::PER>([&](auto p) { ct_for<H::T>([&](auto b) { f[p][b] = Fr[yz_fold(t * H::PER + p + H::N1 * b, PZ)]; }); });
}
template <int PZ, typename C>
SCD_HD void yz_green_mul(C (&u)[HalfLine<PZ>::PER][HalfLine<PZ>::T], const C (&f)[HalfLine<PZ>::PER][HalfLine<PZ>::T]) {
    using H = HalfLine<PZ>;
    ct_for<H::PER>([&](auto p) { ct_for<H::T>([&](auto b) { u[p][b] = cmul(f[p][b], u[p][b]); }); });
}

// the whole fused pass of one plane on the host (x column x, grid rg): the
// same steps, line after line, the threads of a line in turn
template <int PY, int PZ, typename C>
void yz_plane_host(C *Wp, const C *Fyz, const C *twy, const C *twz, int x, const YzDims &D, C *smem) {
    using HY = HalfLine<PY>;
    using HZ = HalfLine<PZ>;
    C *A = smem + PY + PZ, *E = A + (long long)D.Nz * YzLine<PY>::LS;
    for (int z = 0; z < D.Nz; ++z) {
        C *e = E + (z % HY::LW) * HY::ES;
        for (int t = 0; t < HY::T; ++t) {
            C v[HY::M];
            yz_y_load<PY>(v, Wp, z, t, true, D);
            half_fwd_a<PY>(v, e, twy, t);
        }
        for (int t = 0; t < HY::T; ++t) {
            C u[HY::PER][HY::T];
            half_fwd_b<PY>(e, u, t);
            yz_y_put<PY>(u, A, z, t);
        }
    }
    const int fx = yz_fold(x, D.Px);
    for (int c = 0; c < PY; ++c) {
        C *e = E + (c % HZ::LW) * HZ::ES;
        static C u[HZ::T][HZ::PER][HZ::T];
        for (int t = 0; t < HZ::T; ++t) {
            C v[HZ::M];
            yz_z_load<PY, PZ>(v, A, c, t, true, D);
            half_fwd_a<PZ>(v, e, twz, t);
        }
        for (int t = 0; t < HZ::T; ++t) {
            C f[HZ::PER][HZ::T];
            half_fwd_b<PZ>(e, u[t], t);
            yz_green_load<PZ>(f, Fyz + ((long long)fx * D.Hy + yz_fold(yz_ky<PY>(c), PY)) * D.Hz, t);
            yz_green_mul<PZ>(u[t], f);
        }
        for (int t = 0; t < HZ::T; ++t) half_inv_b<PZ>(u[t], e, t);
        for (int t = 0; t < HZ::T; ++t) {
            C v[HZ::M];
            half_inv_a<PZ>(e, twz, v, t);
            yz_z_store<PY, PZ>(v, A, c, t, D);
        }
    }
    for (int z = 0; z < D.Nz; ++z) {
        C *e = E + (z % HY::LW) * HY::ES;
        for (int t = 0; t < HY::T; ++t) {
            C u[HY::PER][HY::T];
            yz_y_get<PY>(u, A, z, t, true);
            half_inv_b<PY>(u, e, t);
        }
        for (int t = 0; t < HY::T; ++t) {
            C v[HY::M];
            half_inv_a<PY>(e, twy, v, t);
            yz_y_store<PY>(v, Wp, z, t, D);
        }
    }
}

// one launch of the fused pass (fft_yz_*.cu): nrg grids
template <typename C> struct YzLaunch {
    C *W;
    const C *Fyz, *twy, *twz;
    YzDims D;
    const int *done;
    int nrg;
    cudaStream_t st;
};
template <int PY, typename C> cudaError_t yz_launch(const YzLaunch<C> &l, int Pz);

#ifdef __CUDACC__
// one CTA per (x, rg): grid (Px, 4 nrhs); dynamic shared memory
// yz_smem_elems<PY, PZ>(Nz, threads) elements of C
template <int PY, int PZ, typename C>
__global__ void __launch_bounds__(YZ_THREADS, sizeof(C) == 8 ? 2 : 1)
k_fft_yz(C *__restrict__ Wt, const C *__restrict__ Fyz, const C *__restrict__ twy_g, const C *__restrict__ twz_g,
         YzDims D, const int *done) {
    const int x = blockIdx.x, rg = blockIdx.y;
    if (done && done[rg >> 2]) return;
    using HY = HalfLine<PY>;
    using HZ = HalfLine<PZ>;
    extern __shared__ __align__(16) unsigned char yz_raw[];
    C *twy = reinterpret_cast<C *>(yz_raw), *twz = twy + PY, *A = twz + PZ;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    C *E = A + D.Nz * YzLine<PY>::LS + warp * yz_ex<PY, PZ>();
    for (int i = threadIdx.x; i < PY; i += blockDim.x) twy[i] = twy_g[i];
    for (int i = threadIdx.x; i < PZ; i += blockDim.x) twz[i] = twz_g[i];
    C *Wp = Wt + ((long long)rg * D.Px + x) * D.Nz * D.Ny;
    const int ty = half_t<PY>(lane), ly = half_l<PY>(lane), tz = half_t<PZ>(lane), lz = half_l<PZ>(lane);
    __syncthreads();
    for (int z0 = warp * HY::LW; z0 < D.Nz; z0 += nw * HY::LW) {
        const int z = z0 + ly;
        const bool live = z < D.Nz;
        C *e = E + ly * HY::ES;
        {
            C v[HY::M];
            yz_y_load<PY>(v, Wp, z, ty, live, D);
            half_fwd_a<PY>(v, e, twy, ty);
        }
        __syncwarp();
        C u[HY::PER][HY::T];
        half_fwd_b<PY>(e, u, ty);
        if (live) yz_y_put<PY>(u, A, z, ty);
        __syncwarp();
    }
    __syncthreads();
    const C *Fx = Fyz + (long long)yz_fold(x, D.Px) * D.Hy * D.Hz;
    for (int c0 = warp * HZ::LW; c0 < PY; c0 += nw * HZ::LW) {
        const bool live = c0 + lz < PY;
        const int c = min(c0 + lz, PY - 1);
        C *e = E + lz * HZ::ES;
        {
            C v[HZ::M];
            yz_z_load<PY, PZ>(v, A, c, tz, live, D);
            half_fwd_a<PZ>(v, e, twz, tz);
        }
        C u[HZ::PER][HZ::T], f[HZ::PER][HZ::T];
        yz_green_load<PZ>(f, Fx + yz_fold(yz_ky<PY>(c), PY) * D.Hz, tz);
        __syncwarp();
        half_fwd_b<PZ>(e, u, tz);
        yz_green_mul<PZ>(u, f);
        __syncwarp();
        half_inv_b<PZ>(u, e, tz);
        __syncwarp();
        C v[HZ::M];
        half_inv_a<PZ>(e, twz, v, tz);
        if (live) yz_z_store<PY, PZ>(v, A, c, tz, D);
        __syncwarp();
    }
    __syncthreads();
    for (int z0 = warp * HY::LW; z0 < D.Nz; z0 += nw * HY::LW) {
        const int z = z0 + ly;
        const bool live = z < D.Nz;
        C *e = E + ly * HY::ES;
        {
            C u[HY::PER][HY::T];
            yz_y_get<PY>(u, A, z, ty, live);
            half_inv_b<PY>(u, e, ty);
        }
        __syncwarp();
        C v[HY::M];
        half_inv_a<PY>(e, twy, v, ty);
        if (live) yz_y_store<PY>(v, Wp, z, ty, D);
        __syncwarp();
    }
}

// Threads of a CTA: the count (128 or 256) that keeps more warps on an SM for
// the plane's size, 128 if both do (its lines fill the warps better on small
// planes).
template <int PY, int PZ, typename C>
cudaError_t yz_launch_t(const YzLaunch<C> &l) {
    auto bytes = [&](int threads) { return sizeof(C) * (size_t)yz_smem_elems<PY, PZ>(l.D.Nz, threads); };
    auto warps = [&](int threads) { return (int)std::min<size_t>((size_t)227 * 1024 / (bytes(threads) + 1024), 512 / threads) * threads; };
    const int threads = warps(256) > warps(128) ? 256 : 128;
    const size_t sh = bytes(threads);
    return launch_dyn<SMEM_CTA>(k_fft_yz<PY, PZ, C>, dim3(l.D.Px, l.nrg), threads, sh, l.st, l.W, l.Fyz, l.twy, l.twz, l.D, l.done);
}

// Fyz[(fx Hy + fy) Hz + fz] = Fo[(fz Hy + fy) Hx + fx]
template <typename C>
__global__ void k_green_yz(const C *__restrict__ Fo, C *__restrict__ Fyz, int Hx, int Hy, int Hz) {
    const long long n = (long long)Hx * Hy * Hz;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const int fz = (int)(i % Hz);
        const long long r = i / Hz;
        const int fy = (int)(r % Hy), fx = (int)(r / Hy);
        Fyz[i] = Fo[((long long)fz * Hy + fy) * Hx + fx];
    }
}
#endif
