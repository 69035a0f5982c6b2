// The pFFT matvec on the device: anterpolation onto the grid, the pruned
// FFT convolution with the Green's function, interpolation back to the tets,
// and the near-zone correction.  Restates compute_Ax2
// (src/gmres_module.f90:57-176) for the constant basis with the three
// cross-component convolutions (:122-144) merged into one by linearity:
//   Y_dd  = S  . G*(S^T x_d)                 d = x, y, z
//   Y2_e  = S_e . G*(Sx^T x_x + Sy^T x_y + Sz^T x_z)
//   Ax    = A_near x + (Y2 - k^2 Y)
// All vectors are slot ordered (tets sorted by cube); see ctx.h.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include <type_traits>

#include "ctx.h"
#include "fft_reg.cuh"
#include "fft_yz.cuh"
#include "linear_basis.h"

namespace {

constexpr int WARPS_PER_CTA = 4;
// resident CTAs per SM the complex64 interpolation of up to eight right-hand
// sides is compiled for (its register cap)
#ifndef SCD_GATHER_MINB
#define SCD_GATHER_MINB 3
#endif
// interpolation warps per SM that the spans of up to eight right-hand sides
// aim at
#ifndef SCD_GATHER_WARPS
#define SCD_GATHER_WARPS 24
#endif
// resident CTAs per SM of the FP64 interpolation of more than eight
// (k_gather_cta), and what the spans aim at in both precisions
#ifndef SCD_GATHER_CTAS
#define SCD_GATHER_CTAS 4
#endif

// slot order <-> the reference's unknown order (nb basis functions per tet:
// 1, or 4 for the linear basis, see linear_basis.h)
__global__ void k_permute_in(const cd *__restrict__ xo, cd *__restrict__ xs, const int *__restrict__ perm,
                             int T, long long ld, int nb) {
    const int r = blockIdx.y;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < 3LL * T; i += (long long)gridDim.x * blockDim.x) {
        long long s = i / 3, d = i - 3 * s;
        xs[r * ld + i] = xo[r * ld + basis_unknown(nb, perm[s], (int)d)];
    }
}

__global__ void k_permute_out(const cd *__restrict__ xs, cd *__restrict__ xo, const int *__restrict__ perm,
                              int T, long long ld, int nb) {
    const int r = blockIdx.y;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < 3LL * T; i += (long long)gridDim.x * blockDim.x) {
        long long s = i / 3, d = i - 3 * s;
        xo[r * ld + basis_unknown(nb, perm[s], (int)d)] = xs[r * ld + i];
    }
}

// ---------------------------------------------------------------- scatter
// Anterpolation (sparse_T_matmul, src/sparse.f90:13-43): the four box-node
// sums of the 27 nodes of every cube, one CTA per (cube, span of right-hand
// sides).  Projectors are stored P[(g*27 + j)*T + slot]; the cube's 108 rows
// are contiguous runs of its tets and are staged in shared memory NTC tets
// at a time by asynchronous copies, 16 threads to a row, all in flight at
// once, with the right-hand sides' x segments beside them, so that the sums
// read shared memory only.  Each sum runs over the tets in ascending order
// (grid 3: x, y, z of a tet in turn) in every variant, so a column gives the
// same bits alone and in a batch.  The row stride NTC + 1 keeps the lanes'
// reads of one tet in distinct banks.  bpart[((r*ncubes + c)*4 + g)*27 + j].
constexpr int SCB = 128;
template <typename C, int NTC>
__device__ __forceinline__ void stage_projectors(C (*Ps)[NTC + 1], const C *__restrict__ P, int T, int s, int m) {
    for (int row = threadIdx.x >> 4; row < 108; row += SCB / 16)
        for (int t = threadIdx.x & 15; t < m; t += 16)
            cp_async_el<(int)sizeof(C)>(&Ps[row][t], P + (size_t)row * T + s + t, true);
}

// Eight or more right-hand sides: the four warps take SR of them each per
// round, lane j < 27 sums node j.  Bound by latency, so everything a round
// reads is in flight before the sums start: 16 FP64 right-hand sides of a
// 12,864-tet sphere take 29 us (68 with x read from global memory tet by tet
// and rows staged through registers), 32 complex64 ones of 60k tets 106 us
// (178).
template <typename C, int NTC, int SR>
__global__ void __launch_bounds__(SCB)
k_scatter_cta(const C *__restrict__ x, long long ld, const C *__restrict__ P, int T, const int *__restrict__ cube_off,
              int ncubes, C *__restrict__ bpart, const int *skip, int nrhs, int rspan) {
    __shared__ C Ps[108][NTC + 1];
    __shared__ C xs[4][SR][3 * NTC];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int c = blockIdx.x;
    const int s0 = cube_off[c], nt = cube_off[c + 1] - s0;
    const int rlo = blockIdx.y * rspan, rhi = min(nrhs, rlo + rspan);
    const int nround = (rhi - rlo + 4 * SR - 1) / (4 * SR);
    const bool one = nt <= NTC;
    if (one) stage_projectors<C, NTC>(Ps, P, T, s0, nt);
    for (int rd = 0; rd < nround; ++rd) {
        const int rb = rlo + (rd * 4 + warp) * SR;
        C acc[SR][4];
#pragma unroll
        for (int q = 0; q < SR; ++q) acc[q][0] = acc[q][1] = acc[q][2] = acc[q][3] = czero<C>();
        for (int t0 = 0; t0 < nt; t0 += NTC) {
            const int m = min(NTC, nt - t0);
            if (!one) {
                __syncthreads();
                stage_projectors<C, NTC>(Ps, P, T, s0 + t0, m);
            }
            __syncwarp();
#pragma unroll
            for (int q = 0; q < SR; ++q) {
                const C *xr = x + (rb + q) * ld + 3LL * (s0 + t0);
                for (int e = lane; e < 3 * m; e += 32)
                    if (rb + q < rhi) cp_async_el<(int)sizeof(C)>(&xs[warp][q][e], xr + e, true);
            }
            cp_async_wait_all();
            if (!one || rd == 0) __syncthreads();
            else __syncwarp();
            if (lane < 27) {
                for (int t = 0; t < m; ++t) {
                    const C p0 = Ps[lane][t], px = Ps[27 + lane][t], py = Ps[54 + lane][t], pz = Ps[81 + lane][t];
#pragma unroll
                    for (int q = 0; q < SR; ++q) {
                        const C x0 = xs[warp][q][3 * t], x1 = xs[warp][q][3 * t + 1], x2 = xs[warp][q][3 * t + 2];
                        cfma(acc[q][0], p0, x0);
                        cfma(acc[q][1], p0, x1);
                        cfma(acc[q][2], p0, x2);
                        cfma(acc[q][3], px, x0);
                        cfma(acc[q][3], py, x1);
                        cfma(acc[q][3], pz, x2);
                    }
                }
            }
        }
        if (lane < 27) {
#pragma unroll
            for (int q = 0; q < SR; ++q) {
                const int r = rb + q;
                if (r < rhi && !(skip && skip[r])) {
                    C *o = bpart + ((long long)r * ncubes + c) * 4 * 27 + lane;
                    o[0] = acc[q][0];
                    o[27] = acc[q][1];
                    o[54] = acc[q][2];
                    o[81] = acc[q][3];
                }
            }
        }
    }
}

// Fewer than eight right-hand sides: warp g sums grid g for SR of them at a
// time, so that all four warps work on a single one.  Bound by the projector
// rows (4*27*T values, read once): one FP64 right-hand side takes 69 us at
// 150,720 tets, 3.8 TB/s of them, and 8 us at 1,680 (157 and 24 with one
// warp per cube reading its rows a tet at a time).
template <typename C, int NTC, int SR>
__global__ void __launch_bounds__(SCB)
k_scatter_few(const C *__restrict__ x, long long ld, const C *__restrict__ P, int T, const int *__restrict__ cube_off,
              int ncubes, C *__restrict__ bpart, const int *skip, int nrhs) {
    __shared__ C Ps[108][NTC + 1];
    __shared__ C xs[SR][3 * NTC];
    const int g = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int c = blockIdx.x;
    const int s0 = cube_off[c], nt = cube_off[c + 1] - s0;
    for (int r0 = 0; r0 < nrhs; r0 += SR) {
        C acc[SR];
#pragma unroll
        for (int q = 0; q < SR; ++q) acc[q] = czero<C>();
        for (int t0 = 0; t0 < nt; t0 += NTC) {
            const int m = min(NTC, nt - t0);
            __syncthreads();
            if (r0 == 0 || nt > NTC) stage_projectors<C, NTC>(Ps, P, T, s0 + t0, m);
#pragma unroll
            for (int q = 0; q < SR; ++q)
                if (r0 + q < nrhs)
                    for (int e = threadIdx.x; e < 3 * m; e += SCB)
                        cp_async_el<(int)sizeof(C)>(&xs[q][e], x + (r0 + q) * ld + 3LL * (s0 + t0) + e, true);
            cp_async_wait_all();
            __syncthreads();
            if (lane >= 27) continue;
            if (g < 3) {
                for (int t = 0; t < m; ++t) {
                    const C p0 = Ps[lane][t];
#pragma unroll
                    for (int q = 0; q < SR; ++q) cfma(acc[q], p0, xs[q][3 * t + g]);
                }
            } else {
                for (int t = 0; t < m; ++t) {
                    const C px = Ps[27 + lane][t], py = Ps[54 + lane][t], pz = Ps[81 + lane][t];
#pragma unroll
                    for (int q = 0; q < SR; ++q) {
                        cfma(acc[q], px, xs[q][3 * t]);
                        cfma(acc[q], py, xs[q][3 * t + 1]);
                        cfma(acc[q], pz, xs[q][3 * t + 2]);
                    }
                }
            }
        }
        if (lane < 27) {
#pragma unroll
            for (int q = 0; q < SR; ++q) {
                const int r = r0 + q;
                if (r < nrhs && !(skip && skip[r])) bpart[((long long)r * ncubes + c) * 4 * 27 + 27 * g + lane] = acc[q];
            }
        }
    }
}

// -------------------------------------------------------------------- FFT
// Radix-4 Stockham (with a final radix-2 stage for odd log2 P) on lines held
// in shared memory, FFTW sign convention (forward exp(-i)), unnormalised.
// TPL = P/4 threads cooperate on a line; all lines of a CTA advance together.
template <int P> struct Log2 { static constexpr int v = 1 + Log2<P / 2>::v; };
template <> struct Log2<1> { static constexpr int v = 0; };

template <bool INV, typename C>
__device__ __forceinline__ void radix4(C &v0, C &v1, C &v2, C &v3) {
    C a0 = cadd(v0, v2), a1 = csub(v0, v2), a2 = cadd(v1, v3), a3 = csub(v1, v3);
    // forward: X1 = a1 - i a3 ; X3 = a1 + i a3
    C ia3;                                                 // (+i or -i) * a3
    ia3.x = INV ? -a3.y : a3.y;
    ia3.y = INV ? a3.x : -a3.x;
    v0 = cadd(a0, a2);
    v2 = csub(a0, a2);
    v1 = cadd(a1, ia3);
    v3 = csub(a1, ia3);
}

// in-line padding pidx(i) = i + (i >> 4) (fft_reg.cuh): one spare slot per
// 16 complex values spreads the strided Stockham writes over the banks

template <bool INV, typename C>
__device__ __forceinline__ C twid(const C *tw, int i) {
    C w = tw[i];
    return INV ? cconj(w) : w;
}

template <int P, bool INV, typename C>
__device__ __forceinline__ void fft_line(C *s, const C *tw, int t) {
    constexpr int L = Log2<P>::v;
    constexpr int NB = P / 4;
    int Ns = 1;
#pragma unroll
    for (int st = 0; st < L / 2; ++st) {
        const int j = t;
        C v0 = s[pidx(j)], v1 = s[pidx(j + NB)], v2 = s[pidx(j + 2 * NB)], v3 = s[pidx(j + 3 * NB)];
        const int kk = j & (Ns - 1);
        if (Ns > 1) {
            const int step = P / (Ns * 4);
            v1 = cmul(v1, twid<INV, C>(tw, kk * step));
            v2 = cmul(v2, twid<INV, C>(tw, 2 * kk * step));
            v3 = cmul(v3, twid<INV, C>(tw, 3 * kk * step));
        }
        radix4<INV, C>(v0, v1, v2, v3);
        __syncthreads();
        const int idx = (j / Ns) * Ns * 4 + kk;
        s[pidx(idx)] = v0;
        s[pidx(idx + Ns)] = v1;
        s[pidx(idx + 2 * Ns)] = v2;
        s[pidx(idx + 3 * Ns)] = v3;
        __syncthreads();
        Ns *= 4;
    }
    if (L & 1) {   // radix-2 stage, Ns = P/2: butterflies j = t, t + NB
        C a[2], b[2];
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const int j = t + q * NB;
            a[q] = s[pidx(j)];
            b[q] = cmul(s[pidx(j + P / 2)], twid<INV, C>(tw, j));
        }
        __syncthreads();
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const int j = t + q * NB;
            s[pidx(j)] = cadd(a[q], b[q]);
            s[pidx(j + P / 2)] = csub(a[q], b[q]);
        }
        __syncthreads();
    }
}

// Lines per CTA of the shared-memory radix-4 transform, for the powers of two
// without a half-full line transform (fft_line.cuh): 8, 256 and 512.
template <int P, typename Cx> struct FftCfg {
    static constexpr int LS = P + (P >> 4) + 1;              // padded line stride (bank spread)
    static constexpr int TPL = P / 4;                        // threads per line
    static constexpr int LPB = 256 / TPL > 0 ? 256 / TPL : 1;
    static constexpr int THREADS = TPL * LPB;
};

struct GridDims {
    int Nx, Ny, Nz, Px, Py, Pz, Hx, Hy, Hz, ncx, ncy, ncz, ncubes;
};

__device__ __forceinline__ int fold(int u, int P) { return u <= P - u ? u : P - u; }

// node value of grid g at node (x,y,z) from the box partial sums: every box
// whose 3x3x3 node block contains the node contributes its local sum
template <typename C>
__device__ __forceinline__ C node_value(const C *__restrict__ bp, const GridDims &G, int g, int x, int y, int z) {
    int bxs[2], axs[2], nbx = 0, bys[2], ays[2], nby = 0, bzs[2], azs[2], nbz = 0;
    int b = x >> 1;
    if (b < G.ncx) { bxs[nbx] = b; axs[nbx++] = x - 2 * b; }
    if (!(x & 1) && x >= 2 && b - 1 < G.ncx) { bxs[nbx] = b - 1; axs[nbx++] = 2; }
    b = y >> 1;
    if (b < G.ncy) { bys[nby] = b; ays[nby++] = y - 2 * b; }
    if (!(y & 1) && y >= 2 && b - 1 < G.ncy) { bys[nby] = b - 1; ays[nby++] = 2; }
    b = z >> 1;
    if (b < G.ncz) { bzs[nbz] = b; azs[nbz++] = z - 2 * b; }
    if (!(z & 1) && z >= 2 && b - 1 < G.ncz) { bzs[nbz] = b - 1; azs[nbz++] = 2; }
    C v = czero<C>();
    for (int iz = 0; iz < nbz; ++iz)
        for (int iy = 0; iy < nby; ++iy)
            for (int ix = 0; ix < nbx; ++ix) {
                const int box = bxs[ix] + G.ncx * (bys[iy] + G.ncy * bzs[iz]);
                const int j = axs[ix] + 3 * ays[iy] + 9 * azs[iz];
                v = cadd(v, bp[((long long)box * 4 + g) * 27 + j]);
            }
    return v;
}

// X forward: lines (y < Ny, z < Nz) of grid (g, r); node assembly on load,
// zero padding x >= Nx.  W[(rg)][(z*Py + y)*Px + x] for the three-pass
// y/z chain, or (TL) the fused y-z pass's layout Wt[rg][x][z][y] (fft_yz.cuh):
// a CTA's lines are consecutive (z, y), so for every x its outputs are one
// contiguous run.
template <int P, typename Cx, bool TL>
__global__ void __launch_bounds__(FftCfg<P, Cx>::THREADS)
k_fft_x_fwd(const Cx *__restrict__ bpart, Cx *__restrict__ W, const Cx *__restrict__ twg, GridDims G, const int *done) {
    if (done && done[blockIdx.y >> 2]) return;
    using Cf = FftCfg<P, Cx>;
    __shared__ Cx sh[Cf::LPB * Cf::LS];
    __shared__ Cx tw[P];
    const int rg = blockIdx.y;                 // r*4 + g
    const int g = rg & 3, r = rg >> 2;
    const Cx *bp = bpart + (long long)r * G.ncubes * 4 * 27;
    for (int i = threadIdx.x; i < P; i += blockDim.x) tw[i] = twg[i];
    const int nlines = G.Ny * G.Nz;
    const int line0 = blockIdx.x * Cf::LPB;
    for (int e = threadIdx.x; e < Cf::LPB * P; e += blockDim.x) {
        const int l = e / P, x = e - l * P, line = line0 + l;
        Cx v = czero<Cx>();
        if (line < nlines && x < G.Nx) {
            const int y = line % G.Ny, z = line / G.Ny;
            v = node_value<Cx>(bp, G, g, x, y, z);
        }
        sh[l * Cf::LS + pidx(x)] = v;
    }
    __syncthreads();
    const int l = threadIdx.x / Cf::TPL, t = threadIdx.x - l * Cf::TPL;
    fft_line<P, false, Cx>(sh + l * Cf::LS, tw, t);
    if constexpr (TL) {
        Cx *Wr = W + (long long)rg * P * nlines;
        for (int e = threadIdx.x; e < Cf::LPB * P; e += blockDim.x) {
            const int x = e / Cf::LPB, ll = e - x * Cf::LPB, line = line0 + ll;
            if (line < nlines) Wr[(long long)x * nlines + line] = sh[ll * Cf::LS + pidx(x)];
        }
    } else {
        Cx *Wr = W + (long long)rg * G.Px * G.Py * G.Nz;
        for (int e = threadIdx.x; e < Cf::LPB * P; e += blockDim.x) {
            const int ll = e / P, x = e - ll * P, line = line0 + ll;
            if (line < nlines) {
                const int y = line % G.Ny, z = line / G.Ny;
                Wr[((long long)z * G.Py + y) * G.Px + x] = sh[ll * Cf::LS + pidx(x)];
            }
        }
    }
}

// The passes for the lengths of fft_line.cuh, 128 threads (64 where four warps'
// exchange buffers exceed static shared memory), lines in registers; the
// three-pass chain forms its lines as the fused pass does (the same bits).  X
// forward: thread t of line (y, z) assembles its nodes x = t + T k < Nx from
// the box partial sums -- the up to four boxes of (y, z) once per line, the
// one or two of x per node, in node_value's order -- and writes the layouts of
// k_fft_x_fwd.  Bound by the latency of the box reads: 32
// complex64 right-hand sides of a 46 x 40 x 28 grid take 107 us (166 with each
// node's boxes found by itself and lines in shared memory).
template <int P, typename Cx>
constexpr int XP_THREADS = (P + 4 * HalfLine<P>::EW) * sizeof(Cx) <= 48 * 1024 ? 128 : 64;
template <int P, typename Cx, bool TL>
__global__ void __launch_bounds__(XP_THREADS<P, Cx>)
k_fft_x_fwd_line(const Cx *__restrict__ bpart, Cx *__restrict__ W, const Cx *__restrict__ twg, GridDims G, const int *done) {
    if (done && done[blockIdx.y >> 2]) return;
    using H = HalfLine<P>;
    __shared__ Cx tw[P], ex[(XP_THREADS<P, Cx> / 32) * H::EW];
    const int rg = blockIdx.y, g = rg & 3, r = rg >> 2, nlines = G.Ny * G.Nz;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, t = half_t<P>(lane), l = half_l<P>(lane);
    for (int i = threadIdx.x; i < P; i += XP_THREADS<P, Cx>) tw[i] = twg[i];
    const int line = (blockIdx.x * (XP_THREADS<P, Cx> / 32) + warp) * H::LW + l;
    const bool live = line < nlines;
    const int y = live ? line % G.Ny : 0, z = live ? line / G.Ny : 0;
    const Cx *bp = bpart + (long long)r * G.ncubes * 108 + g * 27;
    // offsets of the (y, z) boxes' node rows, z the slower: box b of an axis
    // holds node b 2 + a; even nodes also belong to box b - 1 as its node 2
    int row[4];
    bool in[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int dz = q >> 1, dy = q & 1, bz = (z >> 1) - dz, by = (y >> 1) - dy;
        const int az = dz ? 2 : z & 1, ay = dy ? 2 : y & 1;
        in[q] = live && bz >= 0 && bz < G.ncz && by >= 0 && by < G.ncy && !(dz && (z & 1)) && !(dy && (y & 1));
        row[q] = in[q] ? G.ncx * (by + G.ncy * bz) * 108 + 3 * ay + 9 * az : 0;
    }
    __syncthreads();
    Cx *e = ex + warp * H::EW + l * H::ES;
    {
        Cx v[H::M];
        ct_for<H::M>([&](auto k) {
            const int x = t + H::T * k, b = x >> 1;
            const bool lo = x < G.Nx && b < G.ncx, hi = x < G.Nx && !(x & 1) && b >= 1 && b - 1 < G.ncx;
            Cx s = czero<Cx>();
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                if (in[q] && lo) s = cadd(s, bp[row[q] + 108 * b + (x & 1)]);
                if (in[q] && hi) s = cadd(s, bp[row[q] + 108 * (b - 1) + 2]);
            }
            v[k] = s;
        });
        half_fwd_a<P>(v, e, tw, t);
    }
    __syncwarp();
    Cx u[H::PER][H::T];
    half_fwd_b<P>(e, u, t);
    Cx *Wr = TL ? W + (long long)rg * P * nlines + line : W + ((long long)rg * G.Nz + z) * G.Py * P + (long long)y * P;
    const long long step = TL ? nlines : 1;
    if (live)
        ct_for<H::PER>([&](auto p) {
            ct_for<H::T>([&](auto b) { Wr[(t * H::PER + p + H::N1 * b) * step] = u[p][b]; });
        });
}
// inverse: R[(rg)][(z*Ny + y)*Nx + x], x < Nx
template <int P, typename Cx, bool TL>
__global__ void __launch_bounds__(XP_THREADS<P, Cx>)
k_fft_x_inv_line(const Cx *__restrict__ W, Cx *__restrict__ R, const Cx *__restrict__ twg, GridDims G, const int *done) {
    if (done && done[blockIdx.y >> 2]) return;
    using H = HalfLine<P>;
    __shared__ Cx tw[P], ex[(XP_THREADS<P, Cx> / 32) * H::EW];
    const int rg = blockIdx.y, nlines = G.Ny * G.Nz;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, t = half_t<P>(lane), l = half_l<P>(lane);
    for (int i = threadIdx.x; i < P; i += XP_THREADS<P, Cx>) tw[i] = twg[i];
    const int line = (blockIdx.x * (XP_THREADS<P, Cx> / 32) + warp) * H::LW + l;
    const bool live = line < nlines;
    Cx *e = ex + warp * H::EW + l * H::ES;
    {
        Cx u[H::PER][H::T];
        const int y = line % G.Ny, z = line / G.Ny;
        const Cx *Wr = TL ? W + (long long)rg * P * nlines + line : W + ((long long)rg * G.Nz + z) * G.Py * P + (long long)y * P;
        const long long step = TL ? nlines : 1;
        ct_for<H::PER>([&](auto p) {
            ct_for<H::T>([&](auto b) { u[p][b] = live ? Wr[(t * H::PER + p + H::N1 * b) * step] : czero<Cx>(); });
        });
        half_inv_b<P>(u, e, t);
    }
    __syncthreads();
    Cx v[H::M];
    half_inv_a<P>(e, tw, v, t);
    Cx *Rr = R + ((long long)rg * nlines + line) * G.Nx;
    if (live)
        ct_for<H::M>([&](auto k) {
            const int x = t + H::T * k;
            if (x < G.Nx) Rr[x] = v[k];
        });
}

// y and z passes of the three-pass chain on W[rg][z][y][x], lines of
// consecutive x.  A line is read whole before it is written.
template <int P, bool INV, typename Cx>
__global__ void __launch_bounds__(XP_THREADS<P, Cx>)
k_fft_y_line(Cx *__restrict__ W, const Cx *__restrict__ twg, GridDims G, const int *done) {
    if (done && done[blockIdx.y >> 2]) return;
    using H = HalfLine<P>;
    __shared__ Cx tw[P], ex[(XP_THREADS<P, Cx> / 32) * H::EW];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, t = half_t<P>(lane), l = half_l<P>(lane);
    for (int i = threadIdx.x; i < P; i += XP_THREADS<P, Cx>) tw[i] = twg[i];
    const int line = (blockIdx.x * (XP_THREADS<P, Cx> / 32) + warp) * H::LW + l;
    const bool live = line < G.Px * G.Nz;
    const int z = live ? line / G.Px : 0, x = live ? line - z * G.Px : 0;
    Cx *Wr = W + (((long long)blockIdx.y * G.Nz + z) * P) * G.Px + x;
    Cx *e = ex + warp * H::EW + l * H::ES;
    __syncthreads();
    if constexpr (!INV) {
        Cx v[H::M], u[H::PER][H::T];
        ct_for<H::M>([&](auto k) {
            const int y = t + H::T * k;
            v[k] = live && y < G.Ny ? Wr[(long long)y * G.Px] : czero<Cx>();
        });
        half_fwd_a<P>(v, e, tw, t);
        __syncwarp();
        half_fwd_b<P>(e, u, t);
        if (live)
            ct_for<H::PER>([&](auto p) {
                ct_for<H::T>([&](auto b) { Wr[(long long)(t * H::PER + p + H::N1 * b) * G.Px] = u[p][b]; });
            });
    } else {
        Cx v[H::M], u[H::PER][H::T];
        ct_for<H::PER>([&](auto p) {
            ct_for<H::T>([&](auto b) { u[p][b] = live ? Wr[(long long)(t * H::PER + p + H::N1 * b) * G.Px] : czero<Cx>(); });
        });
        half_inv_b<P>(u, e, t);
        __syncwarp();
        half_inv_a<P>(e, tw, v, t);
        if (live)
            ct_for<H::M>([&](auto k) {
                const int y = t + H::T * k;
                if (y < G.Ny) Wr[(long long)y * G.Px] = v[k];
            });
    }
}
template <int P, typename Cx>
__global__ void __launch_bounds__(XP_THREADS<P, Cx>)
k_fft_z_line(Cx *__restrict__ W, const Cx *__restrict__ Fo, const Cx *__restrict__ twg, GridDims G, const int *done) {
    if (done && done[blockIdx.y >> 2]) return;
    using H = HalfLine<P>;
    __shared__ Cx tw[P], ex[(XP_THREADS<P, Cx> / 32) * H::EW];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, t = half_t<P>(lane), l = half_l<P>(lane);
    for (int i = threadIdx.x; i < P; i += XP_THREADS<P, Cx>) tw[i] = twg[i];
    const int line = (blockIdx.x * (XP_THREADS<P, Cx> / 32) + warp) * H::LW + l;
    const bool live = line < G.Px * G.Py;
    const int y = live ? line / G.Px : 0, x = live ? line - y * G.Px : 0;
    const long long plane = (long long)G.Px * G.Py;
    Cx *Wr = W + (long long)blockIdx.y * plane * G.Nz + (long long)y * G.Px + x;
    const Cx *Fr = Fo + (long long)fold(y, G.Py) * G.Hx + fold(x, G.Px);
    Cx *e = ex + warp * H::EW + l * H::ES;
    Cx v[H::M], u[H::PER][H::T];
    __syncthreads();
    ct_for<H::M>([&](auto k) {
        const int z = t + H::T * k;
        v[k] = live && z < G.Nz ? Wr[z * plane] : czero<Cx>();
    });
    half_fwd_a<P>(v, e, tw, t);
    __syncwarp();
    half_fwd_b<P>(e, u, t);
    ct_for<H::PER>([&](auto p) {
        ct_for<H::T>([&](auto b) {
            u[p][b] = cmul(__ldg(&Fr[(long long)fold(t * H::PER + p + H::N1 * b, P) * G.Hy * G.Hx]), u[p][b]);
        });
    });
    __syncwarp();
    half_inv_b<P>(u, e, t);
    __syncwarp();
    half_inv_a<P>(e, tw, v, t);
    if (live)
        ct_for<H::M>([&](auto k) {
            const int z = t + H::T * k;
            if (z < G.Nz) Wr[z * plane] = v[k];
        });
}

// Y pass: lines (x < Px, z < Nz); forward reads y < Ny and writes y < Py,
// inverse reads y < Py and writes y < Ny.  A CTA takes LPB consecutive x.
template <int P, bool INV, typename Cx>
__global__ void __launch_bounds__(FftCfg<P, Cx>::THREADS)
k_fft_y(Cx *__restrict__ W, const Cx *__restrict__ twg, GridDims G, const int *done) {
    if (done && done[blockIdx.y >> 2]) return;
    using Cf = FftCfg<P, Cx>;
    __shared__ Cx sh[Cf::LPB * Cf::LS];
    __shared__ Cx tw[P];
    const int rg = blockIdx.y;
    for (int i = threadIdx.x; i < P; i += blockDim.x) tw[i] = twg[i];
    const int xblocks = (G.Px + Cf::LPB - 1) / Cf::LPB;
    const int z = blockIdx.x / xblocks, x0 = (blockIdx.x - z * xblocks) * Cf::LPB;
    Cx *Wr = W + (long long)rg * G.Px * G.Py * G.Nz + (long long)z * G.Py * G.Px;
    const int nin = INV ? G.Py : G.Ny, nout = INV ? G.Ny : G.Py;
    // sh layout [line][y]
    for (int e = threadIdx.x; e < Cf::LPB * P; e += blockDim.x) {
        const int y = e / Cf::LPB, l = e - y * Cf::LPB, x = x0 + l;
        Cx v = czero<Cx>();
        if (y < nin && x < G.Px) v = Wr[(long long)y * G.Px + x];
        sh[l * Cf::LS + pidx(y)] = v;
    }
    __syncthreads();
    const int l = threadIdx.x / Cf::TPL, t = threadIdx.x - l * Cf::TPL;
    fft_line<P, INV, Cx>(sh + l * Cf::LS, tw, t);
    for (int e = threadIdx.x; e < Cf::LPB * P; e += blockDim.x) {
        const int y = e / Cf::LPB, ll = e - y * Cf::LPB, x = x0 + ll;
        if (y < nout && x < G.Px) Wr[(long long)y * G.Px + x] = sh[ll * Cf::LS + pidx(y)];
    }
}

// Z pass: lines (x < Px, y < Py), forward FFT of z < Nz (zero padded), times
// the Green octant Fo (folded by evenness), inverse FFT, keep z < Nz.
template <int P, typename Cx>
__global__ void __launch_bounds__(FftCfg<P, Cx>::THREADS)
k_fft_z(Cx *__restrict__ W, const Cx *__restrict__ Fo, const Cx *__restrict__ twg, GridDims G, const int *done) {
    if (done && done[blockIdx.y >> 2]) return;
    using Cf = FftCfg<P, Cx>;
    __shared__ Cx sh[Cf::LPB * Cf::LS];
    __shared__ Cx tw[P];
    const int rg = blockIdx.y;
    for (int i = threadIdx.x; i < P; i += blockDim.x) tw[i] = twg[i];
    const int xblocks = (G.Px + Cf::LPB - 1) / Cf::LPB;
    const int y = blockIdx.x / xblocks, x0 = (blockIdx.x - y * xblocks) * Cf::LPB;
    const long long plane = (long long)G.Px * G.Py;
    Cx *Wr = W + (long long)rg * plane * G.Nz + (long long)y * G.Px;
    for (int e = threadIdx.x; e < Cf::LPB * P; e += blockDim.x) {
        const int z = e / Cf::LPB, l = e - z * Cf::LPB, x = x0 + l;
        Cx v = czero<Cx>();
        if (z < G.Nz && x < G.Px) v = Wr[(long long)z * plane + x];
        sh[l * Cf::LS + pidx(z)] = v;
    }
    __syncthreads();
    const int l = threadIdx.x / Cf::TPL, t = threadIdx.x - l * Cf::TPL;
    fft_line<P, false, Cx>(sh + l * Cf::LS, tw, t);
    const int fy = fold(y, G.Py);
    // consecutive threads take consecutive lines (x), so the octant reads of
    // one z plane are contiguous
    for (int e = threadIdx.x; e < Cf::LPB * P; e += blockDim.x) {
        const int z = e / Cf::LPB, ll = e - z * Cf::LPB, x = x0 + ll;
        if (x < G.Px) {
            const Cx f = __ldg(&Fo[((long long)fold(z, G.Pz) * G.Hy + fy) * G.Hx + fold(x, G.Px)]);
            sh[ll * Cf::LS + pidx(z)] = cmul(f, sh[ll * Cf::LS + pidx(z)]);
        }
    }
    __syncthreads();
    fft_line<P, true, Cx>(sh + l * Cf::LS, tw, t);
    for (int e = threadIdx.x; e < Cf::LPB * P; e += blockDim.x) {
        const int z = e / Cf::LPB, ll = e - z * Cf::LPB, x = x0 + ll;
        if (z < G.Nz && x < G.Px) Wr[(long long)z * plane + x] = sh[ll * Cf::LS + pidx(z)];
    }
}

// X inverse: lines (y < Ny, z < Nz), keep x < Nx, write the result grid
// R[(rg)][(z*Ny + y)*Nx + x]; the input in the three-pass layout or (TL) the
// fused y-z pass's Wt[rg][x][z][y]
template <int P, typename Cx, bool TL>
__global__ void __launch_bounds__(FftCfg<P, Cx>::THREADS)
k_fft_x_inv(const Cx *__restrict__ W, Cx *__restrict__ R, const Cx *__restrict__ twg, GridDims G, const int *done) {
    if (done && done[blockIdx.y >> 2]) return;
    using Cf = FftCfg<P, Cx>;
    __shared__ Cx sh[Cf::LPB * Cf::LS];
    __shared__ Cx tw[P];
    const int rg = blockIdx.y;
    for (int i = threadIdx.x; i < P; i += blockDim.x) tw[i] = twg[i];
    const int nlines = G.Ny * G.Nz;
    const int line0 = blockIdx.x * Cf::LPB;
    if constexpr (TL) {
        const Cx *Wr = W + (long long)rg * P * nlines;
        for (int e = threadIdx.x; e < Cf::LPB * P; e += blockDim.x) {
            const int x = e / Cf::LPB, l = e - x * Cf::LPB, line = line0 + l;
            sh[l * Cf::LS + pidx(x)] = line < nlines ? Wr[(long long)x * nlines + line] : czero<Cx>();
        }
    } else {
        const Cx *Wr = W + (long long)rg * G.Px * G.Py * G.Nz;
        for (int e = threadIdx.x; e < Cf::LPB * P; e += blockDim.x) {
            const int l = e / P, x = e - l * P, line = line0 + l;
            Cx v = czero<Cx>();
            if (line < nlines) {
                const int y = line % G.Ny, z = line / G.Ny;
                v = Wr[((long long)z * G.Py + y) * G.Px + x];
            }
            sh[l * Cf::LS + pidx(x)] = v;
        }
    }
    __syncthreads();
    const int l = threadIdx.x / Cf::TPL, t = threadIdx.x - l * Cf::TPL;
    fft_line<P, true, Cx>(sh + l * Cf::LS, tw, t);
    Cx *Rr = R + (long long)rg * G.Nx * G.Ny * G.Nz;
    for (int e = threadIdx.x; e < Cf::LPB * P; e += blockDim.x) {
        const int ll = e / P, x = e - ll * P, line = line0 + ll;
        if (line < nlines && x < G.Nx) {
            const int y = line % G.Ny, z = line / G.Ny;
            Rr[((long long)z * G.Ny + y) * G.Nx + x] = sh[ll * Cf::LS + pidx(x)];
        }
    }
}

// ------------------------------------------------------------ near zone
// Row sums y(g1) += M x(g2) and, for off-diagonal tiles, column sums
// y(g2) += M^T x(g1) (transpose, not conjugate: the operator is complex
// symmetric, src/sparse_mat.f90:113-116).  M(3i+a, 3j+b) is entry (a,b) of
// block (i,j), at tile_at(n1, i, j, a + 3b) (see NearTile).
//
// One CTA per group g: it walks the tiles (g, g2), g2 >= g, in tile order,
// keeping the group's row sums in registers across them, so every group has
// a single row slot; each off-diagonal tile's column sums go to that tile's
// partial slot of g2.  k_gather adds the slots in a fixed order.
//
// Tiles stream through a shared-memory ring filled by a producer thread: a
// tile's blocks and its x segment arrive by bulk copies (TMA engine,
// completion counted in bytes on the slot's "full" mbarrier) at the ring's
// head, so as many tiles are in flight as their sizes allow (up to NZ_SLOTS).
// The x segments come from xT, the right-hand sides interleaved per unknown
// (k_xpose), so a group's x is one contiguous run x[3j+b][r].  Consumer
// warps release a tile on its slot's "empty" barrier; there is no CTA-wide
// barrier in the tile loop.
//
// Every sum runs in one canonical order for any number of right-hand sides,
// so a column's result does not depend on the batch it is solved in: in FP64
// see k_near_dmma below; in complex64 row sums over tiles in order, then j =
// 0..n2-1, then b = 0..2, column sums over i = 0..n1-1, then a = 0..2.
constexpr int NZ_QMAX = 4;             // quads of right-hand sides per pass
constexpr int NZ_SLOTS = 8;                 // tiles in flight at most (mbarrier pairs)
constexpr int NZ_META = 272;                // bytes of barriers, ring offsets and the stop flag
constexpr size_t NZ_SMEM_2CTA = 113 * 1024; // dynamic shared memory per CTA that lets two CTAs share an SM
constexpr size_t NZ_SMEM_4CTA = 56 * 1024;  // ... four CTAs
// With one right-hand side a tile's sums are short dependent chains, so the
// kernel is latency-bound per tile: four CTAs per SM (registers and ring
// bounded to fit) keep four tiles in progress; 43,248 tets in FP64 take 276 us
// so, 319 with three CTAs whose rings hold two tiles.  With register tiles of
// four right-hand sides the compiler is left free (two CTAs fit).
template <int U> constexpr int NZ_MIN_CTAS = U == 1 ? 4 : 1;
template <int NS> constexpr int N1_THREADS = 32 * ((2 * SCD_GROUP_MAX * NS + 31) / 32) + 32;
constexpr size_t NZ_SMEM_MAX = SMEM_CTA;
constexpr int NZ_MAX_THREADS = 2 * 32 * ((SCD_GROUP_MAX * NZ_QMAX + 31) / 32) + 32;

struct NearPass {
    const NearTile *tiles;
    const int *grp_order;    // groups, most work first (a short last wave)
    const int *grp_tile, *grp_off;
    const long long *pslot_base;
    const void *data;
    const void *xT;          // [pass][3T][RG]
    long long n;             // 3T
    void *part;
    long long part_len;
    const int *skip;
    int nrhs, nq, half, rg_stride;   // rg_stride: right-hand sides per xT row (nq*U, or 2 for a lone complex64 one)
    uint32_t x1_bytes;       // x(g) buffer (multiple of 16)
    uint32_t ring_bytes;     // tile ring (multiple of 16, at least one tile with its x segment)
    int *err;
};

// x (nrhs columns of stride ld) -> xT[p][k][RG]: the RG right-hand sides of
// pass p interleaved per unknown k, zero beyond nrhs
template <typename C>
__global__ void k_xpose(const C *__restrict__ x, long long ld, long long n, int nrhs, int PS, int RG, C *__restrict__ xT) {
    const long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    const int p = blockIdx.y;
    if (k >= n) return;
    C *dst = xT + ((long long)p * n + k) * RG;
    for (int r = 0; r < RG; ++r) {
        const int rr = p * PS + r;
        dst[r] = (r < PS && rr < nrhs) ? x[(long long)rr * ld + k] : czero<C>();
    }
}

// U consecutive values of C from shared address addr (16-byte aligned when
// C is complex64 and U is even)
template <typename C, int U>
__device__ __forceinline__ void load_xu(uint32_t addr, C (&xu)[U]) {
    if constexpr (sizeof(C) == 8 && U % 2 == 0) {
#pragma unroll
        for (int u = 0; u < U; u += 2) lds_c2(addr + 8 * u, xu[u], xu[u + 1]);
    } else {
#pragma unroll
        for (int u = 0; u < U; ++u) xu[u] = lds_c(addr + (uint32_t)sizeof(C) * u, C{});
    }
}

// What the near-zone kernels share: the barriers and the ring at the front of
// dynamic shared memory, and the producer that fills the ring.
struct NearFrame {
    uint64_t *full, *empty;
    // per slot, written by the producer before the slot's arrive: ring offset,
    // n2 and column partial slot of the tile (consumers read no tile table)
    int *toff, *tn2;
    long long *tcol;
    // raised by the first wait that gives up: the producer issues no more
    // copies, the consumers skip the remaining tiles (still arriving on their
    // barriers), and the kernel returns with a.err set
    volatile int *stop;
    unsigned char *x1, *ring;
    __device__ NearFrame(unsigned char *sh, uint32_t x1_bytes) {
        full = reinterpret_cast<uint64_t *>(sh);
        empty = full + NZ_SLOTS;
        toff = reinterpret_cast<int *>(sh + 16 * NZ_SLOTS);
        tn2 = toff + NZ_SLOTS;
        tcol = reinterpret_cast<long long *>(sh + 24 * NZ_SLOTS);
        stop = reinterpret_cast<volatile int *>(sh + 32 * NZ_SLOTS);
        x1 = sh + NZ_META;
        ring = sh + NZ_META + x1_bytes;
    }
    // one thread of the CTA, before a __syncthreads
    __device__ void init(int consumer_warps) const {
        for (int k = 0; k < NZ_SLOTS; ++k) {
            mbar_init(&full[k], 1);              // the producer's arrive (with the tile's bytes)
            mbar_init(&empty[k], consumer_warps);
        }
        *stop = 0;
        mbar_fence_init();
    }
};

// The producer thread: tiles t0..t1-1 of group rows [s1, s1 + n1), once per
// pass of PS right-hand sides, each with its x segment (and the group's own x
// beside the first).  Ring accounting: `used` bytes are reserved by the
// `count` tiles in flight (a tile that wraps also reserves the unused end of
// the ring); tiles are released in order, oldest first.
template <typename ST, typename C>
__device__ __forceinline__ void near_produce(const NearPass &a, const NearFrame &f, int t0, int t1, int s1, int n1, int PS) {
    const ST *data = static_cast<const ST *>(a.data);
    const C *xT = static_cast<const C *>(a.xT);
    const int RG = a.rg_stride;     // xT row length
    const uint32_t R = a.ring_bytes;
    uint32_t head = 0, used = 0;
    uint32_t resv[NZ_SLOTS] = {};
    int oldest = 0, count = 0, ord = 0;
    int last[NZ_SLOTS];                  // latest tile issued into each slot
    for (int k = 0; k < NZ_SLOTS; ++k) last[k] = -1;
    bool halt = false;
    auto release_oldest = [&]() {
        const int k = oldest % NZ_SLOTS;
        if (!mbar_wait_or(&f.empty[k], (uint32_t)((oldest / NZ_SLOTS) & 1), a.err, f.stop)) halt = true;
        used -= resv[k];
        ++oldest;
        --count;
    };
    for (int r0 = 0; r0 < a.nrhs && !halt; r0 += PS) {
        const C *xp = xT + (long long)(r0 / PS) * a.n * RG;
        while (count > 0 && !halt) release_oldest();   // x1 is rewritten: the previous pass must be done
        for (int t = t0; t < t1 && !halt; ++t, ++ord) {
            const NearTile &tl = a.tiles[t];
            const uint32_t mb = (uint32_t)(tile_elems(tl.n1, tl.n2) * (long long)sizeof(ST));
            const uint32_t xb = (uint32_t)(3 * tl.n2 * RG * sizeof(C));
            const uint32_t x1b = t == t0 ? (uint32_t)(3 * n1 * RG * sizeof(C)) : 0u;
            const uint32_t S = mb + xb;
            bool fit = head + S <= R;
            uint32_t res = fit ? S : (R - head) + S;
            while (count > 0 && !halt && (count == NZ_SLOTS || used + res > R)) release_oldest();
            if (halt || *f.stop) { halt = true; break; }
            if (count == 0) { head = 0; used = 0; fit = true; res = S; }
            const uint32_t st = fit ? head : 0u;
            const int k = ord % NZ_SLOTS;
            f.toff[k] = (int)st;
            f.tn2[k] = tl.n2;
            f.tcol[k] = tl.col_off;
            mbar_expect_tx(&f.full[k], S + x1b);
            bulk_g2s(f.ring + st, data + tl.data_off, mb, &f.full[k]);
            bulk_g2s(f.ring + st + mb, xp + 3LL * tl.s2 * RG, xb, &f.full[k]);
            if (x1b) bulk_g2s(f.x1, xp + 3LL * s1 * RG, x1b, &f.full[k]);
            head = st + S;
            used += res;
            resv[k] = res;
            last[k] = ord;
            ++count;
        }
    }
    if (halt) {
        // a wait gave up: tell the consumers, then let every copy still
        // landing in the ring finish before the CTA exits
        *f.stop = 1;
        for (int k = 0; k < NZ_SLOTS; ++k)
            if (last[k] >= 0) mbar_wait(&f.full[k], (uint32_t)((last[k] / NZ_SLOTS) & 1), a.err);
    }
}

// a consumer warp waits for tile `ord`; false (and the slot released) if the
// pipeline has stopped -- the warp skips or computes as one
__device__ __forceinline__ bool near_wait_tile(const NearPass &a, const NearFrame &f, int ord, int lane) {
    const int k = ord % NZ_SLOTS;
    bool ok = !*f.stop && mbar_wait_or(&f.full[k], (uint32_t)((ord / NZ_SLOTS) & 1), a.err, f.stop);
    ok = __all_sync(0xffffffffu, ok);
    if (!ok) {
        *f.stop = 1;
        __syncwarp();
        if (lane == 0) mbar_arrive(&f.empty[k]);
    }
    return ok;
}

// The complex64 matvec on the CUDA cores (complex128 storage, or on request).
// Warps [0, HT) hold row items (quad q, block row i): a 3 x U register tile of
// row sums for right-hand sides Uq..Uq+U-1.  Warps [HT, 2HT) hold column items
// (q, block column j).  Lanes run over i (resp. j), so with the odd plane
// stride both sides read the tile without bank conflicts, and x is a
// broadcast.
template <typename ST, int U>
__global__ void __launch_bounds__(NZ_MAX_THREADS, NZ_MIN_CTAS<U>) k_near_groups(NearPass a) {
    typedef cf C;
    extern __shared__ __align__(128) unsigned char nz_sh[];
    const NearFrame f(nz_sh, a.x1_bytes);
    C *const X1 = reinterpret_cast<C *>(f.x1);                 // x(g)
    C *part = static_cast<C *>(a.part);

    const int g = a.grp_order[blockIdx.x];
    const int t0 = a.grp_tile[g], t1 = a.grp_tile[g + 1];
    const int s1 = a.grp_off[g], n1 = a.grp_off[g + 1] - s1;
    const int ld1 = n1 | 1;
    const int RG = a.rg_stride;     // xT row length
    const int PS = a.nq * U;        // right-hand sides per pass
    const int HT = a.half;
    const int ncw = 2 * HT / 32;                 // consumer warps
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    if (threadIdx.x == 0) f.init(ncw);
    __syncthreads();
    if (warp == ncw) {
        if (lane == 0) near_produce<ST, C>(a, f, t0, t1, s1, n1, PS);
        return;
    }

    // ---------------------------------------------------------- consumers
    const bool rowside = warp < HT / 32;
    const int it = rowside ? threadIdx.x : threadIdx.x - HT;
    const bool row_item = rowside && it < n1 * a.nq;
    const int rq = row_item ? it / n1 : 0, ri = row_item ? it - rq * n1 : 0;
    int ord = 0;
    for (int r0 = 0; r0 < a.nrhs; r0 += PS) {
        const int rg = min(PS, a.nrhs - r0);
        C acc[3][U];
#pragma unroll
        for (int q = 0; q < 3; ++q)
#pragma unroll
            for (int u = 0; u < U; ++u) acc[q][u] = czero<C>();
        for (int t = t0; t < t1; ++t, ++ord) {
            const int kslot = ord % NZ_SLOTS;
            if (!near_wait_tile(a, f, ord, lane)) continue;
            const int n2 = f.tn2[kslot];
            const long long tcoff = f.tcol[kslot];
            const uint32_t M = smem_addr(f.ring + f.toff[kslot]);
            const uint32_t X2 = M + (uint32_t)(tile_elems(n1, n2) * (long long)sizeof(ST));
            constexpr uint32_t SB = sizeof(ST), CB = sizeof(C);
            const uint32_t mrow = SB * ld1, xrow = CB * RG;   // bytes between planes / x rows
            if (rowside) {
                if (row_item) {
                    uint32_t mp = M + SB * ri;            // plane (9j + 3b), lane i
                    uint32_t xp = X2 + CB * U * rq;       // x row 3j + b
                    for (int j = 0; j < 3 * n2; ++j) {
                        C xu[U];
                        load_xu<C, U>(xp, xu);
                        const C mm[3] = {as_c<C>(lds_c(mp, ST{})), as_c<C>(lds_c(mp + mrow, ST{})),
                                         as_c<C>(lds_c(mp + 2 * mrow, ST{}))};
                        mac3<C, U>(acc, mm, xu);
                        mp += 3 * mrow;
                        xp += xrow;
                    }
                }
            } else if (tcoff >= 0 && it < n2 * a.nq) {
                const int q = it / n2, j = it - q * n2;
                C cacc[3][U];
#pragma unroll
                for (int b = 0; b < 3; ++b)
#pragma unroll
                    for (int u = 0; u < U; ++u) cacc[b][u] = czero<C>();
                const uint32_t mj = M + SB * 9 * j * ld1;
                uint32_t xp = smem_addr(X1) + CB * U * q;   // x row 3i + a
                for (int i = 0; i < n1; ++i) {
#pragma unroll
                    for (int aa = 0; aa < 3; ++aa) {
                        C xu[U];
                        load_xu<C, U>(xp, xu);
                        const uint32_t mp = mj + aa * mrow + SB * i;
                        const C mm[3] = {as_c<C>(lds_c(mp, ST{})), as_c<C>(lds_c(mp + 3 * mrow, ST{})),
                                         as_c<C>(lds_c(mp + 6 * mrow, ST{}))};
                        mac3<C, U>(cacc, mm, xu);
                        xp += xrow;
                    }
                }
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int r = U * q + u;
                    if (r < rg && !(a.skip && a.skip[r0 + r])) {
                        C *pc = part + (r0 + r) * a.part_len + tcoff + 3 * j;
                        pc[0] = cacc[0][u];
                        pc[1] = cacc[1][u];
                        pc[2] = cacc[2][u];
                    }
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&f.empty[kslot]);
        }
        if (row_item) {
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int r = U * rq + u;
                if (r < rg && !(a.skip && a.skip[r0 + r])) {
                    C *pr = part + (r0 + r) * a.part_len + a.pslot_base[g] + 3 * ri;
                    pr[0] = acc[0][u];
                    pr[1] = acc[1][u];
                    pr[2] = acc[2][u];
                }
            }
        }
    }
}

// ---- FP64
// Both FP64 kernels form a sum over unknowns k in blocks of four: per block
// the real part adds Ar(k) xr(k) for the four k in order, then -Ai(k) xi(k);
// the imaginary part Ar(k) xi(k), then Ai(k) xr(k).  That is what two
// m8n8k4 DMMAs per part compute (each output is a chain of four fused
// multiply-adds in k order, checked bit for bit over 128,000 random sums), so
// one right-hand side on the FMA units and many on the tensor cores give a
// column the same bits.  NS = 2 sums even and odd blocks of a tile separately,
// then adds the two.  A row sum adds its tiles' sums in order; k past the end
// contributes fma(0, 0, s).
__device__ __forceinline__ void dmma(double (&c)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};\n"
                 : "+d"(c[0]), "+d"(c[1])
                 : "d"(a), "d"(b));
}

// Two or more right-hand sides, 8 NT of them per pass (their rows of xT are
// 8 NT + 2 values apart: a quarter-warp's reads of four k and two
// right-hand sides then fall in distinct banks).  Consumer warp w forms the
// row sums of unknowns 8w .. 8w + 7 of the group, kept in registers across
// the tiles, and the column sums of unknowns 8w .. 8w + 7 of each tile's g2:
// one element read and converted per lane feeds 4 NT DMMAs.  Bound by the
// FP64 tensor pipe (37 TFLOP/s measured; 63 % active at 16 right-hand sides):
// 16 right-hand sides of a 12,864-tet sphere take 331 us (585 with register
// tiles of FMAs), 16 of 3,000 tets 130 (172).
constexpr int ND_WARPS = (3 * SCD_GROUP_MAX + 7) / 8;   // consumer warps, then the producer
template <int NT> constexpr int ND_PS = 8 * NT;
template <int NT> constexpr int ND_RG = 8 * NT + 2;

// a lane's operands of one block: its element and NT values of x, zero past the end
template <typename ST, int NT> struct DmmaOperands {
    ST m;
    cd x[NT];
    __device__ __forceinline__ void load(uint32_t ma, uint32_t xa, bool in, int nt) {
        m = in ? lds_c(ma, ST{}) : ST{};
#pragma unroll
        for (int t = 0; t < NT; ++t)
            if (t < nt) x[t] = in ? lds_c(xa + 128 * t, cd{}) : cmk(0, 0);
    }
};
template <typename ST, int NT>
__device__ __forceinline__ void dmma_block(double (&re)[NT][2], double (&im)[NT][2], const DmmaOperands<ST, NT> &o, int nt) {
    const cd m = as_c<cd>(o.m);
#pragma unroll
    for (int t = 0; t < NT; ++t)
        if (t < nt) { dmma(re[t], m.x, o.x[t].x); dmma(im[t], m.x, o.x[t].y); }
#pragma unroll
    for (int t = 0; t < NT; ++t)
        if (t < nt) { dmma(re[t], -m.y, o.x[t].y); dmma(im[t], m.y, o.x[t].x); }
}
// a tile's sums over K unknowns in blocks of four, the next block's operands
// read before the present one's DMMAs; at(kk) is the lane's element address
// for its unknown kk of a block
template <typename ST, int NT, int NS, typename At>
__device__ __forceinline__ void dmma_sum(double (&re)[NS][NT][2], double (&im)[NS][NT][2], uint32_t xa, int K, int k4, int nt, At at) {
#pragma unroll
    for (int p = 0; p < NS; ++p)
#pragma unroll
        for (int t = 0; t < NT; ++t) re[p][t][0] = re[p][t][1] = im[p][t][0] = im[p][t][1] = 0.0;
    constexpr uint32_t XB = 16 * 4 * ND_RG<NT>;                                // x rows of a block
    DmmaOperands<ST, NT> cur, nxt;
    cur.load(at(k4), xa, k4 < K, nt);
    for (int k = 0; k < K; k += 4 * NS) {
#pragma unroll
        for (int p = 0; p < NS; ++p) {
            const int kp = k + 4 * p;
            if (p > 0 && kp >= K) break;
            xa += XB;
            const int kk = kp + 4 + k4;
            nxt.load(at(kk), xa, kk < K, nt);
            dmma_block<ST, NT>(re[p], im[p], cur, nt);
            cur = nxt;
        }
    }
    if constexpr (NS == 2)
#pragma unroll
        for (int t = 0; t < NT; ++t)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                re[0][t][e] = SCD_ADD(re[0][t][e], re[1][t][e]);
                im[0][t][e] = SCD_ADD(im[0][t][e], im[1][t][e]);
            }
}
template <int NT>
__device__ __forceinline__ void dmma_store(cd *part, const NearPass &a, int r0, int rg, long long at, const double (&re)[NT][2],
                                           const double (&im)[NT][2], int lane) {
#pragma unroll
    for (int t = 0; t < NT; ++t)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int r = 8 * t + 2 * (lane & 3) + e;
            if (r < rg && !(a.skip && a.skip[r0 + r])) part[(r0 + r) * a.part_len + at] = cmk(re[t][e], im[t][e]);
        }
}

template <typename ST, int NT, int NS>
__global__ void __launch_bounds__(32 * ND_WARPS + 32, 2) k_near_dmma(NearPass a) {
    extern __shared__ __align__(128) unsigned char nz_sh[];
    const NearFrame f(nz_sh, a.x1_bytes);
    cd *part = static_cast<cd *>(a.part);
    const int g = a.grp_order[blockIdx.x];
    const int t0 = a.grp_tile[g], t1 = a.grp_tile[g + 1];
    const int s1 = a.grp_off[g], n1 = a.grp_off[g + 1] - s1;
    const int ld1 = n1 | 1, K1 = 3 * n1;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) f.init(ND_WARPS);
    __syncthreads();
    if (warp == ND_WARPS) {
        if (lane == 0) near_produce<ST, cd>(a, f, t0, t1, s1, n1, ND_PS<NT>);
        return;
    }
    constexpr uint32_t SB = sizeof(ST);
    const int m8 = 8 * warp + (lane >> 2), k4 = lane & 3;
    const int row = min(m8, K1 - 1);
    const uint32_t row_at = SB * ((row % 3) * ld1 + row / 3);                  // element (row, 0) of a tile
    const uint32_t x_at = 16 * (k4 * ND_RG<NT> + (lane >> 2));
    int ord = 0;
    for (int r0 = 0; r0 < a.nrhs; r0 += ND_PS<NT>) {
        const int rg = min(ND_PS<NT>, a.nrhs - r0), nt = (rg + 7) / 8;
        double rre[NT][2], rim[NT][2], re[NS][NT][2], im[NS][NT][2];
#pragma unroll
        for (int t = 0; t < NT; ++t) rre[t][0] = rre[t][1] = rim[t][0] = rim[t][1] = 0.0;
        for (int t = t0; t < t1; ++t, ++ord) {
            if (!near_wait_tile(a, f, ord, lane)) continue;
            const int kslot = ord % NZ_SLOTS;
            const int n2 = f.tn2[kslot], K2 = 3 * n2;
            const long long tcoff = f.tcol[kslot];
            const uint32_t M = smem_addr(f.ring + f.toff[kslot]);
            const uint32_t X2 = M + (uint32_t)(tile_elems(n1, n2) * (long long)sizeof(ST));
            if (8 * warp < K1) {
                dmma_sum<ST, NT, NS>(re, im, X2 + x_at, K2, k4, nt, [&](int kk) { return M + row_at + SB * 3 * ld1 * kk; });
#pragma unroll
                for (int q = 0; q < NT; ++q)
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        rre[q][e] = SCD_ADD(rre[q][e], re[0][q][e]);
                        rim[q][e] = SCD_ADD(rim[q][e], im[0][q][e]);
                    }
            }
            if (tcoff >= 0 && 8 * warp < K2) {
                const uint32_t mc = M + SB * 3 * min(m8, K2 - 1) * ld1;
                int aa = k4 % 3, i = k4 / 3;              // row kk = 3i + aa, in steps of four
                dmma_sum<ST, NT, NS>(re, im, smem_addr(f.x1) + x_at, K1, k4, nt, [&](int) {
                    const uint32_t at = mc + SB * (aa * ld1 + i);
                    ++i;
                    if (++aa == 3) { aa = 0; ++i; }
                    return at;
                });
                if (m8 < K2) dmma_store<NT>(part, a, r0, rg, tcoff + m8, re[0], im[0], lane);
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&f.empty[kslot]);
        }
        if (m8 < K1) dmma_store<NT>(part, a, r0, rg, a.pslot_base[g] + m8, rre, rim, lane);
    }
}

// One right-hand side: NS adjacent lanes form the three row sums of one tet of
// the group, or the three column sums of one tet of g2, lane p the blocks p,
// p + NS, ...: per block 12 elements and 4 values of x are read together for
// 48 FMAs.  Row and column items run the same code on other addresses and
// follow one another over the lanes, so that a tile of 20 x 20 tets fills 80
// of 96 lanes (40 + 40 of 64 + 64 with a side to each warp): the conversions
// of the stored complex64 elements, each made once for its row and once for
// its column, are what the kernel is bound by.  150,720 tets take 723 us,
// 4.1 TB/s of tiles (788 with a side to each warp), 43,248 take 276 (323),
// 1,680 take 45 (54).
template <typename ST> struct OneBlock {
    ST m[4][3];
    cd x[4];
    // element d of unknown q at ma[q] + d * md
    __device__ __forceinline__ void load(const uint32_t (&ma)[4], uint32_t md, uint32_t xa, int nk) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const bool in = q < nk;
            x[q] = in ? lds_c(xa + 16 * q, cd{}) : cmk(0, 0);
#pragma unroll
            for (int d = 0; d < 3; ++d) m[q][d] = in ? lds_c(ma[q] + d * md, ST{}) : ST{};
        }
    }
    __device__ __forceinline__ void add(cd (&acc)[3]) const {
#pragma unroll
        for (int q = 0; q < 4; ++q)
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                const cd v = as_c<cd>(m[q][d]);
                acc[d].x = SCD_FMA(v.x, x[q].x, acc[d].x);
                acc[d].y = SCD_FMA(v.x, x[q].y, acc[d].y);
            }
#pragma unroll
        for (int q = 0; q < 4; ++q)
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                const cd v = as_c<cd>(m[q][d]);
                acc[d].x = SCD_FMA(-v.y, x[q].y, acc[d].x);
                acc[d].y = SCD_FMA(v.y, x[q].x, acc[d].y);
            }
    }
};
// the NS lanes' sums added (every lane of the warp calls it)
template <int NS>
__device__ __forceinline__ void one_combine(cd (&acc)[3]) {
    if constexpr (NS == 2)
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const cd o = make_double2(__shfl_xor_sync(0xffffffffu, acc[d].x, 1), __shfl_xor_sync(0xffffffffu, acc[d].y, 1));
            acc[d] = cadd(acc[d], o);
        }
}

template <typename ST, int NS>
__global__ void __launch_bounds__(N1_THREADS<NS>, 4) k_near_one(NearPass a) {
    extern __shared__ __align__(128) unsigned char nz_sh[];
    const NearFrame f(nz_sh, a.x1_bytes);
    cd *part = static_cast<cd *>(a.part);
    const int g = a.grp_order[blockIdx.x];
    const int t0 = a.grp_tile[g], t1 = a.grp_tile[g + 1];
    const int s1 = a.grp_off[g], n1 = a.grp_off[g + 1] - s1;
    const int ld1 = n1 | 1, ncw = a.half / 32;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) f.init(ncw);
    __syncthreads();
    if (warp == ncw) {
        if (lane == 0) near_produce<ST, cd>(a, f, t0, t1, s1, n1, 1);
        return;
    }
    constexpr uint32_t SB = sizeof(ST);
    const bool on = !(a.skip && a.skip[0]);
    const int item = threadIdx.x / NS, p = threadIdx.x - NS * item;   // row tets, then column tets; partial
    const bool row = item < n1;
    const int col = item - n1;
    const uint32_t plane = SB * ld1;
    // element (d, k = 3i + aa) of the item: from one k to the next `inc`, from
    // aa = 2 to the next i `wrap`; d planes md apart
    const uint32_t md = row ? plane : 3 * plane;
    const uint32_t inc = row ? 3 * plane : plane, wrap = row ? 3 * plane : SB - 2 * plane;
    const uint32_t first = row ? SB * item + 12 * p * plane : 9 * col * plane + ((4 * p) % 3) * plane + SB * ((4 * p) / 3);
    cd sum[3] = {cmk(0, 0), cmk(0, 0), cmk(0, 0)};
    for (int t = t0, ord = 0; t < t1; ++t, ++ord) {
        if (!near_wait_tile(a, f, ord, lane)) continue;
        const int kslot = ord % NZ_SLOTS;
        const int n2 = f.tn2[kslot];
        const long long tcoff = f.tcol[kslot];
        const uint32_t M = smem_addr(f.ring + f.toff[kslot]);
        const uint32_t X2 = M + (uint32_t)(tile_elems(n1, n2) * (long long)sizeof(ST));
        cd acc[3] = {cmk(0, 0), cmk(0, 0), cmk(0, 0)};
        const bool cols = !row && tcoff >= 0 && col < n2;
        const int K = row ? 3 * n2 : cols ? 3 * n1 : 0;
        uint32_t ma = M + first, xa = (row ? X2 : smem_addr(f.x1)) + 64 * p;
        int aa = (4 * p) % 3;
        OneBlock<ST> o;
        for (int k = 4 * p; k < K; k += 4 * NS) {
            uint32_t m4[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                m4[q] = ma;
                ma += aa == 2 ? wrap : inc;
                aa = aa == 2 ? 0 : aa + 1;
            }
            o.load(m4, md, xa, K - k);
            o.add(acc);
            if constexpr (NS == 2) {       // the other lane's block
                ma += 3 * inc + (wrap - inc) + (aa == 2 ? wrap : inc);
                aa = aa == 2 ? 0 : aa + 1;
            }
            xa += 64 * NS;
        }
        __syncwarp();
        one_combine<NS>(acc);
        if (row) {
#pragma unroll
            for (int d = 0; d < 3; ++d) sum[d] = cadd(sum[d], acc[d]);
        } else if (cols && p == 0 && on) {
            cd *pc = part + tcoff + 3 * col;
            pc[0] = acc[0]; pc[1] = acc[1]; pc[2] = acc[2];
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&f.empty[kslot]);
    }
    if (row && p == 0 && on) {
        cd *pr = part + a.pslot_base[g] + 3 * item;
        pr[0] = sum[0]; pr[1] = sum[1]; pr[2] = sum[2];
    }
}

// ---------------------------------------------------------------- gather
// Interpolation (sparse_eps_matmul, src/sparse.f90:47-77) and final
// assembly (src/gmres_module.f90:148-170), one warp per (near-zone group,
// span of rspan right-hand sides), one lane per tet, GA_RG right-hand sides
// at a time: the 27 box-node values of the four result grids are staged in
// shared memory, each lane forms its tet's six 27-term sums from the
// projector rows P[(g*27 + j)*T + slot] (coalesced across lanes; they stay
// in L1 for the next group of the span), adds the group's near-zone partial
// slots in slot order and writes Ax = near + (Y2 - k^2 Y).  The spans are the
// grid's y index; rspan is a multiple of GA_RG.
template <typename C, int GA_RG>
__global__ void __launch_bounds__(32 * WARPS_PER_CTA, sizeof(C) == 8 ? SCD_GATHER_MINB : 1)
k_gather(const C *__restrict__ Rg, const C *__restrict__ P, int T, const int *__restrict__ grp_off,
         const int *__restrict__ grp_cube, int ngroups, GridDims G, typename CReal<C>::type k2,
         const C *__restrict__ part, long long part_len, const long long *__restrict__ pslot_base,
         const int *__restrict__ pslot_cnt, C *__restrict__ y, long long ld, const int *skip, int nrhs,
         int rspan) {
    __shared__ C Rs[WARPS_PER_CTA][GA_RG][4][27];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int gq = blockIdx.x * WARPS_PER_CTA + warp;
    if (gq >= ngroups) return;
    const int s0 = grp_off[gq], s1 = grp_off[gq + 1];
    const int nc = s1 - s0;
    const int c = grp_cube[gq];
    const int bx = c % G.ncx, by = (c / G.ncx) % G.ncy, bz = c / (G.ncx * G.ncy);
    const long long NN = (long long)G.Nx * G.Ny * G.Nz;
    const long long pbase = pslot_base[gq];
    const int nslot = pslot_cnt[gq];
    long long node = 0;
    if (lane < 27) {
        const int a = lane % 3, b = (lane / 3) % 3, cc = lane / 9;
        node = ((long long)(2 * bz + cc) * G.Ny + (2 * by + b)) * G.Nx + (2 * bx + a);
    }
    const int rend = min(nrhs, (int)(blockIdx.y + 1) * rspan);
    for (int r0 = blockIdx.y * rspan; r0 < rend; r0 += GA_RG) {
        __syncwarp();
        if (lane < 27) {
#pragma unroll
            for (int q = 0; q < GA_RG; ++q) {
                const int r = r0 + q;
                if (r < nrhs) {
                    const C *Rr = Rg + (long long)r * 4 * NN;
#pragma unroll
                    for (int g = 0; g < 4; ++g) Rs[warp][q][g][lane] = Rr[g * NN + node];
                }
            }
        }
        __syncwarp();
        for (int sl = lane; sl < nc; sl += 32) {
            const int s = s0 + sl;
            C acc[GA_RG][6];
#pragma unroll
            for (int q = 0; q < GA_RG; ++q)
#pragma unroll
                for (int v = 0; v < 6; ++v) acc[q][v] = czero<C>();
#pragma unroll 3
            for (int j = 0; j < 27; ++j) {
                const C p0 = P[(size_t)j * T + s], px = P[(size_t)(27 + j) * T + s];
                const C py = P[(size_t)(54 + j) * T + s], pz = P[(size_t)(81 + j) * T + s];
#pragma unroll
                for (int q = 0; q < GA_RG; ++q) {
                    cfma(acc[q][0], p0, Rs[warp][q][0][j]);
                    cfma(acc[q][1], p0, Rs[warp][q][1][j]);
                    cfma(acc[q][2], p0, Rs[warp][q][2][j]);
                    const C r3 = Rs[warp][q][3][j];
                    cfma(acc[q][3], px, r3);
                    cfma(acc[q][4], py, r3);
                    cfma(acc[q][5], pz, r3);
                }
            }
            // far field first (acc dies), then the partial slots of all
            // right-hand sides of the round in one sweep over the slots, so
            // that 3 GA_RG independent loads are in flight per slot; each sum
            // still runs over the slots in order
            C far[GA_RG][3], nz[GA_RG][3];
            bool on[GA_RG];
#pragma unroll
            for (int q = 0; q < GA_RG; ++q) {
                const int r = r0 + q;
                on[q] = r < nrhs && !(skip && skip[r]);
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    far[q][d] = csub_scaled(acc[q][3 + d], k2, acc[q][d]);
                    nz[q][d] = czero<C>();
                }
            }
            const C *pr0 = part + pbase + 3 * sl;
#pragma unroll 2
            for (int t = 0; t < nslot; ++t) {
                const C *pt = pr0 + (long long)t * 3 * nc;
#pragma unroll
                for (int q = 0; q < GA_RG; ++q) {
                    if (!on[q]) continue;
                    const C *pq = pt + (r0 + q) * part_len;
#pragma unroll
                    for (int d = 0; d < 3; ++d) nz[q][d] = cadd(nz[q][d], pq[d]);
                }
            }
#pragma unroll
            for (int q = 0; q < GA_RG; ++q) {
                if (!on[q]) continue;
                C *yr = y + (r0 + q) * ld + 3LL * s;
#pragma unroll
                for (int d = 0; d < 3; ++d) yr[d] = cadd(nz[q][d], far[q][d]);
            }
        }
    }
}

// The same interpolation for more than eight right-hand sides, one CTA per
// (group, span): the group's 108 projector rows are staged in shared memory by
// asynchronous copies, and the four warps take SR right-hand sides each per
// round, in k_gather's order of sums (the same bits).  Bound by the latency of
// the slot and node reads: 32 complex64 right-hand sides of 60k tets take 238 us
// (334 with a warp per group that reads the rows from L1 every round), 16 FP64
// ones of 12,864 tets 57 (67); five CTAs per SM (96 registers) take 266.
// Eight right-hand sides are two rounds of k_gather's four, which occupies more
// warps: 8 complex64 of 43,248 tets take 104 us there and 117 here, 8 FP64 of
// 12,864 tets 49 and 56; 9 take 130 and 124, 63 and 58.
constexpr int GCB = 128, GC_SR = 4, GC_MIN = 9;
template <typename C, int SR> struct GatherShared {
    C P[108][SCD_GROUP_MAX + 1];
    C R[GCB / 32][SR][4][27];
};
template <typename C, int SR>
__global__ void __launch_bounds__(GCB, sizeof(C) == 8 ? SCD_GATHER_CTAS : 2)
k_gather_cta(const C *__restrict__ Rg, const C *__restrict__ P, int T, const int *__restrict__ grp_off,
             const int *__restrict__ grp_cube, GridDims G, typename CReal<C>::type k2, const C *__restrict__ part,
             long long part_len, const long long *__restrict__ pslot_base, const int *__restrict__ pslot_cnt,
             C *__restrict__ y, long long ld, const int *skip, int nrhs, int rspan) {
    extern __shared__ __align__(16) unsigned char ga_raw[];
    GatherShared<C, SR> &sh = *reinterpret_cast<GatherShared<C, SR> *>(ga_raw);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gq = blockIdx.x;
    const int s0 = grp_off[gq], nc = grp_off[gq + 1] - s0, c = grp_cube[gq];
    for (int row = threadIdx.x >> 4; row < 108; row += GCB / 16)
        for (int t = threadIdx.x & 15; t < nc; t += 16)
            cp_async_el<(int)sizeof(C)>(&sh.P[row][t], P + (size_t)row * T + s0 + t, true);
    const int bx = c % G.ncx, by = (c / G.ncx) % G.ncy, bz = c / (G.ncx * G.ncy);
    const long long NN = (long long)G.Nx * G.Ny * G.Nz;
    const C *pr0 = part + pslot_base[gq] + 3 * lane;
    const int nslot = pslot_cnt[gq];
    const int a = lane % 3, b = (lane / 3) % 3, cc = lane / 9;
    const long long node = ((long long)(2 * bz + cc) * G.Ny + (2 * by + b)) * G.Nx + (2 * bx + a);
    const int rlo = blockIdx.y * rspan, rhi = min(nrhs, rlo + rspan);
    const int nround = (rhi - rlo + GCB / 32 * SR - 1) / (GCB / 32 * SR);
    for (int rd = 0; rd < nround; ++rd) {
        const int r0 = rlo + (rd * (GCB / 32) + warp) * SR;
        __syncwarp();
        if (lane < 27)
#pragma unroll
            for (int q = 0; q < SR; ++q)
                if (r0 + q < rhi)
#pragma unroll
                    for (int g = 0; g < 4; ++g)
                        cp_async_el<(int)sizeof(C)>(&sh.R[warp][q][g][lane], Rg + ((long long)(r0 + q) * 4 + g) * NN + node, true);
        cp_async_wait_all();
        if (rd == 0) __syncthreads();
        else __syncwarp();
        if (lane >= nc || r0 >= rhi) continue;
        C acc[SR][6];
#pragma unroll
        for (int q = 0; q < SR; ++q)
#pragma unroll
            for (int v = 0; v < 6; ++v) acc[q][v] = czero<C>();
        for (int j = 0; j < 27; ++j) {
            const C p0 = sh.P[j][lane], px = sh.P[27 + j][lane], py = sh.P[54 + j][lane], pz = sh.P[81 + j][lane];
#pragma unroll
            for (int q = 0; q < SR; ++q) {
                cfma(acc[q][0], p0, sh.R[warp][q][0][j]);
                cfma(acc[q][1], p0, sh.R[warp][q][1][j]);
                cfma(acc[q][2], p0, sh.R[warp][q][2][j]);
                const C r3 = sh.R[warp][q][3][j];
                cfma(acc[q][3], px, r3);
                cfma(acc[q][4], py, r3);
                cfma(acc[q][5], pz, r3);
            }
        }
        C far[SR][3], nz[SR][3];
        bool on[SR];
#pragma unroll
        for (int q = 0; q < SR; ++q) {
            on[q] = r0 + q < rhi && !(skip && skip[r0 + q]);
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                far[q][d] = csub_scaled(acc[q][3 + d], k2, acc[q][d]);
                nz[q][d] = czero<C>();
            }
        }
#pragma unroll 2
        for (int t = 0; t < nslot; ++t) {
            const C *pt = pr0 + (long long)t * 3 * nc;
#pragma unroll
            for (int q = 0; q < SR; ++q) {
                if (!on[q]) continue;
                const C *pq = pt + (r0 + q) * part_len;
#pragma unroll
                for (int d = 0; d < 3; ++d) nz[q][d] = cadd(nz[q][d], pq[d]);
            }
        }
#pragma unroll
        for (int q = 0; q < SR; ++q) {
            if (!on[q]) continue;
            C *yr = y + (r0 + q) * ld + 3LL * (s0 + lane);
#pragma unroll
            for (int d = 0; d < 3; ++d) yr[d] = cadd(nz[q][d], far[q][d]);
        }
    }
}

__global__ void k_twiddles(cd *tw, int P) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < P) {
        double s, c;
        sincospi(-2.0 * (double)i / (double)P, &s, &c);
        tw[i] = cmk(c, s);
    }
}

__global__ void k_narrow(const cd *in, cf *out, long long n) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        out[i] = make_float2((float)in[i].x, (float)in[i].y);
}

GridDims dims_of(const scd_ctx *c) {
    GridDims G;
    G.Nx = c->Nx; G.Ny = c->Ny; G.Nz = c->Nz;
    G.Px = c->Px; G.Py = c->Py; G.Pz = c->Pz;
    G.Hx = c->Hx; G.Hy = c->Hy; G.Hz = c->Hz;
    G.ncx = c->ncx; G.ncy = c->ncy; G.ncz = c->ncz; G.ncubes = c->ncubes;
    return G;
}

// operator copies and work buffers of one precision
template <typename C> struct Res;
template <> struct Res<cd> {
    static const cd *P(scd_ctx *c) { return c->d_P; }
    static const cd *Fo(scd_ctx *c) { return c->d_Fo; }
    static const cd *Fyz(scd_ctx *c) { return c->d_Fyz; }
    static const cd *tw(scd_ctx *c, int a) { return c->d_tw[a]; }
    static cd *bpart(scd_ctx *c) { return c->d_bpart; }
    static cd *W(scd_ctx *c) { return c->d_W; }
    static cd *R(scd_ctx *c) { return c->d_R; }
    static cd *part(scd_ctx *c) { return c->d_nzpart; }
    static cd *xT(scd_ctx *c) { return c->d_xT; }
};
template <> struct Res<cf> {
    static const cf *P(scd_ctx *c) { return c->f_P; }
    static const cf *Fo(scd_ctx *c) { return c->f_Fo; }
    static const cf *Fyz(scd_ctx *c) { return c->f_Fyz; }
    static const cf *tw(scd_ctx *c, int a) { return c->f_tw[a]; }
    static cf *bpart(scd_ctx *c) { return c->f_bpart; }
    static cf *W(scd_ctx *c) { return c->f_W; }
    static cf *R(scd_ctx *c) { return c->f_R; }
    static cf *part(scd_ctx *c) { return c->f_nzpart; }
    static cf *xT(scd_ctx *c) { return c->f_xT; }
};

// CTAs of a line kernel over n lines
template <int P, typename C> dim3 line_grid(int n, int nrg) {
    constexpr int per = XP_THREADS<P, C> / 32 * HalfLine<P>::LW;
    return dim3((n + per - 1) / per, nrg);
}
template <int P, typename C>
void fft_x_fwd_t(scd_ctx *c, const GridDims &G, int nrg, const int *done, const C *tw, bool tl) {
    if constexpr (half_len(P)) {
        const dim3 grid = line_grid<P, C>(G.Ny * G.Nz, nrg);
        if (tl) k_fft_x_fwd_line<P, C, true><<<grid, XP_THREADS<P, C>, 0, c->st>>>(Res<C>::bpart(c), Res<C>::W(c), tw, G, done);
        else k_fft_x_fwd_line<P, C, false><<<grid, XP_THREADS<P, C>, 0, c->st>>>(Res<C>::bpart(c), Res<C>::W(c), tw, G, done);
    } else {
        using Cf = FftCfg<P, C>;
        dim3 grid((G.Ny * G.Nz + Cf::LPB - 1) / Cf::LPB, nrg);
        if (tl) k_fft_x_fwd<P, C, true><<<grid, Cf::THREADS, 0, c->st>>>(Res<C>::bpart(c), Res<C>::W(c), tw, G, done);
        else k_fft_x_fwd<P, C, false><<<grid, Cf::THREADS, 0, c->st>>>(Res<C>::bpart(c), Res<C>::W(c), tw, G, done);
    }
}
template <int P, bool INV, typename C>
void fft_y_t(scd_ctx *c, const GridDims &G, int nrg, const int *done, const C *tw) {
    if constexpr (half_len(P)) {
        k_fft_y_line<P, INV, C><<<line_grid<P, C>(G.Px * G.Nz, nrg), XP_THREADS<P, C>, 0, c->st>>>(Res<C>::W(c), tw, G, done);
    } else {
        using Cf = FftCfg<P, C>;
        dim3 grid(((G.Px + Cf::LPB - 1) / Cf::LPB) * G.Nz, nrg);
        k_fft_y<P, INV, C><<<grid, Cf::THREADS, 0, c->st>>>(Res<C>::W(c), tw, G, done);
    }
}
template <int P, typename C>
void fft_z_t(scd_ctx *c, const GridDims &G, int nrg, const int *done, const C *tw) {
    if constexpr (half_len(P)) {
        k_fft_z_line<P, C><<<line_grid<P, C>(G.Px * G.Py, nrg), XP_THREADS<P, C>, 0, c->st>>>(Res<C>::W(c), Res<C>::Fo(c), tw, G, done);
    } else {
        using Cf = FftCfg<P, C>;
        dim3 grid(((G.Px + Cf::LPB - 1) / Cf::LPB) * G.Py, nrg);
        k_fft_z<P, C><<<grid, Cf::THREADS, 0, c->st>>>(Res<C>::W(c), Res<C>::Fo(c), tw, G, done);
    }
}
template <int P, typename C>
void fft_x_inv_t(scd_ctx *c, const GridDims &G, int nrg, const int *done, const C *tw, bool tl) {
    if constexpr (half_len(P)) {
        const dim3 grid = line_grid<P, C>(G.Ny * G.Nz, nrg);
        if (tl) k_fft_x_inv_line<P, C, true><<<grid, XP_THREADS<P, C>, 0, c->st>>>(Res<C>::W(c), Res<C>::R(c), tw, G, done);
        else k_fft_x_inv_line<P, C, false><<<grid, XP_THREADS<P, C>, 0, c->st>>>(Res<C>::W(c), Res<C>::R(c), tw, G, done);
    } else {
        using Cf = FftCfg<P, C>;
        dim3 grid((G.Ny * G.Nz + Cf::LPB - 1) / Cf::LPB, nrg);
        if (tl) k_fft_x_inv<P, C, true><<<grid, Cf::THREADS, 0, c->st>>>(Res<C>::W(c), Res<C>::R(c), tw, G, done);
        else k_fft_x_inv<P, C, false><<<grid, Cf::THREADS, 0, c->st>>>(Res<C>::W(c), Res<C>::R(c), tw, G, done);
    }
}

// the fused y-z pass (fft_yz.cuh)
template <typename C>
void fft_yz(scd_ctx *c, const GridDims &G, int nrg, const int *done) {
    YzLaunch<C> l;
    l.W = Res<C>::W(c); l.Fyz = Res<C>::Fyz(c); l.twy = Res<C>::tw(c, 1); l.twz = Res<C>::tw(c, 2);
    l.D.Nx = G.Nx; l.D.Ny = G.Ny; l.D.Nz = G.Nz; l.D.NzR = yz_round8(G.Nz);
    l.D.Px = G.Px; l.D.Hx = G.Hx; l.D.Hy = G.Hy; l.D.Hz = G.Hz;
    l.done = done; l.nrg = nrg; l.st = c->st;
    cudaError_t e = cudaErrorInvalidValue;
    switch (G.Py) {
        case 16: e = yz_launch<16>(l, G.Pz); break;
        case 32: e = yz_launch<32>(l, G.Pz); break;
        case 40: e = yz_launch<40>(l, G.Pz); break;
        case 48: e = yz_launch<48>(l, G.Pz); break;
        case 64: e = yz_launch<64>(l, G.Pz); break;
        case 80: e = yz_launch<80>(l, G.Pz); break;
        case 96: e = yz_launch<96>(l, G.Pz); break;
        case 112: e = yz_launch<112>(l, G.Pz); break;
        case 128: e = yz_launch<128>(l, G.Pz); break;
        case 192: e = yz_launch<192>(l, G.Pz); break;
        default: break;
    }
    if (e != cudaSuccess) c->launch_err = e;
}

// least shared memory of the fused y-z pass for the context's lengths (CTAs of
// 128 threads)
template <typename C>
size_t yz_smem_bytes(const scd_ctx *c) { return sizeof(C) * (size_t)yz_elems(c->Py, c->Pz, c->Nz, 128); }

// whether the complex64 (or FP64) chain takes the fused y-z pass: both lengths
// have warp-synchronous line transforms and the CTA fits shared memory
template <typename C>
bool use_yz(const scd_ctx *c) {
    if (!c->yz_on || !half_len(c->Py) || !half_len(c->Pz)) return false;
    return yz_smem_bytes<C>(c) <= SMEM_CTA;
}

// the transposed Green octant of the fused pass, built from Fo once per
// Green spectrum; false (three-pass chain) if it cannot be allocated
template <typename C>
bool ensure_fyz(scd_ctx *c) {
    constexpr bool single = std::is_same<C, cf>::value;
    bool &ready = single ? c->fyz_ready_f : c->fyz_ready;
    if (ready) return true;
    C *&buf = *reinterpret_cast<C **>(single ? (void *)&c->f_Fyz : (void *)&c->d_Fyz);
    const long long no = (long long)c->Hx * c->Hy * c->Hz;
    if (!buf && cudaMalloc((void **)&buf, sizeof(C) * (size_t)no) != cudaSuccess) {
        cudaGetLastError();
        buf = nullptr;
        return false;
    }
    k_green_yz<C><<<(unsigned)std::min<long long>((no + 255) / 256, 4096), 256, 0, c->st>>>(Res<C>::Fo(c), buf, c->Hx,
                                                                                          c->Hy, c->Hz);
    ready = true;
    return true;
}

// Right-hand sides that one block walks: a tuned span, or the most that still
// gives every SM `per_sm` of the `items` x spans blocks, rounded up to the
// `unit` of a round.  A longer span reads the projector rows fewer times, a
// shorter one keeps a small mesh from leaving SMs idle: 32 complex64
// right-hand sides of 6,144 tets (300 groups) interpolated in 32 us with spans
// of 4 per warp, in 91 with one span of 32; at 60k tets both took 335.
int rhs_span(const scd_ctx *c, int tuned, int nrhs, int items, int unit, int per_sm) {
    int sp = std::min(tuned, nrhs);
    if (sp <= 0) {
        const long long want = (long long)per_sm * c->nsm;
        const long long spans = std::min<long long>((nrhs + unit - 1) / unit, (want + items - 1) / std::max(items, 1));
        sp = (int)((nrhs + spans - 1) / std::max<long long>(spans, 1));
    }
    return (sp + unit - 1) / unit * unit;
}
}  // namespace

bool prepare_green_yz(scd_ctx *c) { return use_yz<cd>(c) && ensure_fyz<cd>(c); }

// the spans that a matvec of nrhs right-hand sides takes for a tuned value:
// the anterpolation walks 16 at a time in five resident CTAs per SM, and all
// of fewer than eight (k_scatter_few); the interpolation 16 above eight
// (k_gather_cta), up to eight two waves of twelve warps
int scatter_span_of(const scd_ctx *c, int nrhs, int tuned) {
    return nrhs >= 8 ? rhs_span(c, tuned, nrhs, c->ncubes, 16, 5) : nrhs;
}
int gather_span_of(const scd_ctx *c, int nrhs, int tuned) {
    return nrhs >= GC_MIN ? rhs_span(c, tuned, nrhs, c->ngroups, GCB / 32 * GC_SR, SCD_GATHER_CTAS)
                          : rhs_span(c, tuned, nrhs, c->ngroups, nrhs >= 4 ? 4 : 1, SCD_GATHER_WARPS);
}

namespace {
#define SCD_DISPATCH_P(PV, CALL)                     \
    switch (PV) {                                    \
        case 8: CALL(8); break;                      \
        case 16: CALL(16); break;                    \
        case 32: CALL(32); break;                    \
        case 64: CALL(64); break;                    \
        case 128: CALL(128); break;                  \
        case 40: CALL(40); break;                    \
        case 48: CALL(48); break;                    \
        case 80: CALL(80); break;                    \
        case 112: CALL(112); break;                  \
        case 96: CALL(96); break;                    \
        case 192: CALL(192); break;                  \
        case 256: CALL(256); break;                  \
        case 512: CALL(512); break;                  \
        default: break;                              \
    }

template <typename C>
void fft_chain_t(scd_ctx *c, const C *x, int nrhs, const int *done) {
    const GridDims G = dims_of(c);
    {
        const C *P = Res<C>::P(c);
        constexpr int NTC = sizeof(C) == 8 ? 32 : 16, NTF = sizeof(C) == 8 ? 32 : 24;   // static shared memory: 48 KB
        const dim3 gx((unsigned)c->ncubes);
        if (nrhs >= 8) {
            const int sp = scatter_span_of(c, nrhs, c->scatter_span);
            k_scatter_cta<C, NTC, 4><<<dim3((unsigned)c->ncubes, (nrhs + sp - 1) / sp), SCB, 0, c->st>>>(
                x, c->n, P, c->T, c->d_cube_off, c->ncubes, Res<C>::bpart(c), done, nrhs, sp);
        } else if (nrhs >= 2) {
            k_scatter_few<C, NTF, 4><<<gx, SCB, 0, c->st>>>(x, c->n, P, c->T, c->d_cube_off, c->ncubes,
                                                            Res<C>::bpart(c), done, nrhs);
        } else {
            k_scatter_few<C, NTF, 1><<<gx, SCB, 0, c->st>>>(x, c->n, P, c->T, c->d_cube_off, c->ncubes,
                                                            Res<C>::bpart(c), done, nrhs);
        }
    }
    const int nrg = 4 * nrhs;
    const bool tl = use_yz<C>(c) && ensure_fyz<C>(c);
#define XF(PP) fft_x_fwd_t<PP, C>(c, G, nrg, done, Res<C>::tw(c, 0), tl)
#define YF(PP) fft_y_t<PP, false, C>(c, G, nrg, done, Res<C>::tw(c, 1))
#define ZC(PP) fft_z_t<PP, C>(c, G, nrg, done, Res<C>::tw(c, 2))
#define YI(PP) fft_y_t<PP, true, C>(c, G, nrg, done, Res<C>::tw(c, 1))
#define XI(PP) fft_x_inv_t<PP, C>(c, G, nrg, done, Res<C>::tw(c, 0), tl)
    SCD_DISPATCH_P(c->Px, XF)
    if (tl) {
        fft_yz<C>(c, G, nrg, done);
    } else {
        SCD_DISPATCH_P(c->Py, YF)
        SCD_DISPATCH_P(c->Pz, ZC)
        SCD_DISPATCH_P(c->Py, YI)
    }
    SCD_DISPATCH_P(c->Px, XI)
#undef XF
#undef YF
#undef ZC
#undef YI
#undef XI
    c->launches += tl ? 4 : 6;
}

// One near-zone launch: `passes` of PS right-hand sides whose rows of xT are
// rg values apart, ncw consumer warps per CTA, shared memory for `budget`
// bytes per CTA where a tile with its x fits it.
template <typename ST, typename C, typename K>
void near_launch(scd_ctx *c, K kernel, const ST *data, const C *x, int nrhs, int PS, int rg, int threads, size_t budget,
                 NearPass a, const int *done) {
    a.tiles = c->d_tiles; a.grp_order = c->d_grp_order; a.grp_tile = c->d_grp_tile; a.grp_off = c->d_grp_off; a.pslot_base = c->d_pslot_base;
    a.data = data; a.xT = Res<C>::xT(c); a.n = c->n; a.part = Res<C>::part(c); a.part_len = c->part_len;
    a.skip = done; a.nrhs = nrhs;
    a.err = c->d_kerr;
    // xT rows are whole 16-byte units (bulk-copy granularity)
    a.rg_stride = rg;
    while ((a.rg_stride * sizeof(C)) % 16) ++a.rg_stride;
    a.x1_bytes = (uint32_t)(3 * c->max_per_group * a.rg_stride * sizeof(C));
    // the ring fills the budget, and must hold the largest tile with its x
    const size_t max_tile = (size_t)c->max_tile_store * sizeof(ST) + a.x1_bytes;
    size_t ring = (budget - NZ_META - a.x1_bytes) / 16 * 16;
    if (ring < max_tile) ring = std::min((NZ_SMEM_MAX - NZ_META - a.x1_bytes) / 16 * 16, (max_tile + 15) / 16 * 16 * 2);
    if (ring < max_tile) {
        // cannot happen with groups of at most SCD_GROUP_MAX slots; reported
        // by near_status instead of overrunning the ring
        c->near_cfg_err = 1;
        return;
    }
    a.ring_bytes = (uint32_t)ring;
    const dim3 g((unsigned)((c->n + 255) / 256), (nrhs + PS - 1) / PS);
    k_xpose<C><<<g, 256, 0, c->st>>>(x, c->n, c->n, nrhs, PS, a.rg_stride, Res<C>::xT(c));
    c->launches += 1;
    const size_t sh = NZ_META + a.x1_bytes + a.ring_bytes;
    if (c->timing) cudaEventRecord(c->ev[6], c->st);
    const cudaError_t e = launch_dyn<NZ_SMEM_MAX>(kernel, c->ngroups, threads, sh, c->st, a);
    if (e != cudaSuccess) c->launch_err = e;
    if (c->timing) cudaEventRecord(c->ev[7], c->st);
}

template <typename ST, int U>
void near_cf(scd_ctx *c, const ST *data, const cf *x, int nrhs, const int *done) {
    NearPass a{};
    a.nq = U == 1 ? 1 : std::min(NZ_QMAX, (nrhs + U - 1) / U);
    a.half = 32 * ((c->max_per_group * a.nq + 31) / 32);   // lanes per side
    near_launch<ST, cf>(c, k_near_groups<ST, U>, data, x, nrhs, a.nq * U, a.nq * U, 2 * a.half + 32,
                        U == 1 ? NZ_SMEM_4CTA : NZ_SMEM_2CTA, a, done);
}

template <typename ST, int NS>
void near_cd(scd_ctx *c, const ST *data, const cd *x, int nrhs, const int *done) {
    NearPass a{};
    a.nq = 1;
    a.half = 32 * ((2 * NS * c->max_per_group + 31) / 32);   // consumer lanes of the one-column kernel
    // one right-hand side on the FMA units takes 276 us at 43,248 tets; the
    // DMMAs, padded to 8 columns, could not take less than 336 (12.1 GFLOP at
    // 36 TFLOP/s), which they share among two or more
    if (nrhs == 1)
        near_launch<ST, cd>(c, k_near_one<ST, NS>, data, x, 1, 1, 1, a.half + 32, NZ_SMEM_4CTA, a, done);
    else if (nrhs <= 8)
        near_launch<ST, cd>(c, k_near_dmma<ST, 1, NS>, data, x, nrhs, ND_PS<1>, ND_RG<1>, 32 * ND_WARPS + 32, NZ_SMEM_2CTA, a, done);
    else
        near_launch<ST, cd>(c, k_near_dmma<ST, 2, NS>, data, x, nrhs, ND_PS<2>, ND_RG<2>, 32 * ND_WARPS + 32, NZ_SMEM_2CTA, a, done);
}

template <typename ST>
void near_dispatch(scd_ctx *c, const ST *data, const cf *x, int nrhs, const int *done) {
    if (nrhs == 1) near_cf<ST, 1>(c, data, x, nrhs, done);
    else near_cf<ST, 4>(c, data, x, nrhs, done);
}
// near_split 2 (the default): two partial sums per row and column sum, in
// every FP64 kernel, so a column keeps its bits alone and in a batch
template <typename ST>
void near_dispatch(scd_ctx *c, const ST *data, const cd *x, int nrhs, const int *done) {
    if (c->near_split == 2) near_cd<ST, 2>(c, data, x, nrhs, done);
    else near_cd<ST, 1>(c, data, x, nrhs, done);
}

template <typename C>
void near_t(scd_ctx *c, const C *x, int nrhs, const int *done) {
    if (c->ngroups == 0) return;
    if constexpr (std::is_same<C, cf>::value) {
        if (c->nzm_on && c->nzm_ready) {
            near_mma_run(c, x, nrhs, done);
            return;
        }
    }
    if (c->near_prec == SCD_STORE_C64) near_dispatch<cf>(c, (const cf *)c->d_tdata, x, nrhs, done);
    else near_dispatch<cd>(c, (const cd *)c->d_tdata, x, nrhs, done);
    c->launches += 1;
}

template <typename C>
void gather_t(scd_ctx *c, C *y, int nrhs, const int *done) {
    const GridDims G = dims_of(c);
    const unsigned gx = (unsigned)((c->ngroups + WARPS_PER_CTA - 1) / WARPS_PER_CTA);
    if (c->ngroups == 0) return;
    typedef typename CReal<C>::type R;
    const R k2 = (R)(c->k * c->k);
    const int sp = gather_span_of(c, nrhs, c->gather_span);
    if (nrhs >= GC_MIN) {
        constexpr int SR = GC_SR;
        constexpr size_t sh = sizeof(GatherShared<C, SR>);
        const cudaError_t e = launch_dyn<sh>(
            k_gather_cta<C, SR>, dim3((unsigned)c->ngroups, (nrhs + sp - 1) / sp), GCB, sh, c->st, Res<C>::R(c),
            Res<C>::P(c), c->T, c->d_grp_off, c->d_grp_cube, G, k2, Res<C>::part(c), c->part_len, c->d_pslot_base,
            c->d_pslot_cnt, y, c->n, done, nrhs, sp);
        if (e != cudaSuccess) c->launch_err = e;
    } else if (nrhs >= 4) {
        k_gather<C, 4><<<dim3(gx, (nrhs + sp - 1) / sp), 32 * WARPS_PER_CTA, 0, c->st>>>(
            Res<C>::R(c), Res<C>::P(c), c->T, c->d_grp_off, c->d_grp_cube, c->ngroups, G, k2, Res<C>::part(c),
            c->part_len, c->d_pslot_base, c->d_pslot_cnt, y, c->n, done, nrhs, sp);
    } else {
        k_gather<C, 1><<<dim3(gx, (nrhs + sp - 1) / sp), 32 * WARPS_PER_CTA, 0, c->st>>>(
            Res<C>::R(c), Res<C>::P(c), c->T, c->d_grp_off, c->d_grp_cube, c->ngroups, G, k2, Res<C>::part(c),
            c->part_len, c->d_pslot_base, c->d_pslot_cnt, y, c->n, done, nrhs, sp);
    }
    c->launches += 1;
}

template <typename C>
void run_matvec_t(scd_ctx *c, const C *x, C *y, int nrhs, const int *done) {
    if (c->timing) cudaEventRecord(c->ev[0], c->st);
    {
        NvtxRange r("near zone");
        near_t<C>(c, x, nrhs, done);
    }
    if (c->timing) cudaEventRecord(c->ev[1], c->st);
    {
        NvtxRange r("fft convolutions");
        fft_chain_t<C>(c, x, nrhs, done);
    }
    if (c->timing) cudaEventRecord(c->ev[2], c->st);
    {
        NvtxRange r("gather");
        gather_t<C>(c, y, nrhs, done);
    }
    if (c->timing) cudaEventRecord(c->ev[3], c->st);
}

}  // namespace

// twiddle table exp(-2 pi i j / P), j < P
int build_twiddles(scd_ctx *c, int P, cd **out) {
    cudaError_t e = cudaMalloc(out, sizeof(cd) * P);
    if (e != cudaSuccess) return check_cuda(c, e, "twiddles");
    k_twiddles<<<(P + 255) / 256, 256, 0, c->st>>>(*out, P);
    return check_cuda(c, cudaGetLastError(), "twiddles");
}

// complex64 copies of the projectors, the Green octant and the twiddles for
// the mixed-precision inner solves (rounded from the FP64 operator)
int ensure_single(scd_ctx *c) {
    // the tensor-core near zone reads complex64 tiles; by default a context
    // with complex128 storage keeps the CUDA-core kernel, an explicit request
    // is an error (near_mma_prepare)
    if (c->nzm_on && !c->nzm_ready && c->have_near && c->ngroups > 0 &&
        (c->near_prec == SCD_STORE_C64 || c->d.near_kernel != SCD_NEAR_DEFAULT)) {
        const int rc = near_mma_prepare(c);
        if (rc) return rc;
    }
    if (c->f_ready) return SCD_OK;
    const long long np = 4LL * 27 * c->T, no = (long long)c->Hx * c->Hy * c->Hz;
    auto al = [&](cf **p, long long n) -> int {
        if (*p) { cudaFree(*p); *p = nullptr; }
        if (cudaMalloc(p, sizeof(cf) * (size_t)std::max<long long>(n, 1)) != cudaSuccess) {
            cudaGetLastError();
            return set_error(c, SCD_OOM, "complex64 operator copy");
        }
        return SCD_OK;
    };
    int rc;
    if ((rc = al(&c->f_P, np)) || (rc = al(&c->f_Fo, no))) return rc;
    k_narrow<<<1024, 256, 0, c->st>>>(c->d_P, c->f_P, np);
    k_narrow<<<1024, 256, 0, c->st>>>(c->d_Fo, c->f_Fo, no);
    const int Ps[3] = {c->Px, c->Py, c->Pz};
    for (int a = 0; a < 3; ++a) {
        if ((rc = al(&c->f_tw[a], Ps[a]))) return rc;
        k_narrow<<<(Ps[a] + 255) / 256, 256, 0, c->st>>>(c->d_tw[a], c->f_tw[a], Ps[a]);
    }
    rc = check_cuda(c, cudaStreamSynchronize(c->st), "complex64 operator copy");
    if (!rc) c->f_ready = true;
    return rc;
}

int ensure_work_single(scd_ctx *c, int nrhs) {
    if (c->f_cap >= nrhs && c->f_W) return SCD_OK;
    const size_t r = (size_t)nrhs;
    auto al = [&](cf **p, size_t n) -> int {
        if (*p) { cudaFree(*p); *p = nullptr; }
        if (cudaMalloc(p, sizeof(cf) * std::max<size_t>(n, 1)) != cudaSuccess) {
            cudaGetLastError();
            return set_error(c, SCD_OOM, "complex64 work buffers (%d right-hand sides)", nrhs);
        }
        return SCD_OK;
    };
    int rc;
    if ((rc = al(&c->f_bpart, r * c->ncubes * 4 * 27)) || (rc = al(&c->f_W, r * 4 * (size_t)c->Px * c->Py * c->Nz)) ||
        (rc = al(&c->f_R, r * 4 * (size_t)c->Nx * c->Ny * c->Nz)) ||
        (rc = al(&c->f_nzpart, r * (size_t)std::max<long long>(c->part_len, 1))) ||
        (rc = al(&c->f_xT, (size_t)xt_columns(nrhs) * c->n)))
        return rc;
    c->f_cap = nrhs;
    return SCD_OK;
}

void launch_permute_in(scd_ctx *c, const cd *x_orig, cd *x_slot, int nrhs, long long ld) {
    dim3 grid((unsigned)std::min<long long>((3LL * c->T + 255) / 256, 4096), nrhs);
    k_permute_in<<<grid, 256, 0, c->st>>>(x_orig, x_slot, c->d_perm, c->T, ld, c->nb);
}

void launch_permute_out(scd_ctx *c, const cd *x_slot, cd *x_orig, int nrhs, long long ld) {
    dim3 grid((unsigned)std::min<long long>((3LL * c->T + 255) / 256, 4096), nrhs);
    k_permute_out<<<grid, 256, 0, c->st>>>(x_slot, x_orig, c->d_perm, c->T, ld, c->nb);
}

void launch_fft_chain(scd_ctx *c, const cd *x, int nrhs, const int *done) { fft_chain_t<cd>(c, x, nrhs, done); }
void launch_near(scd_ctx *c, const cd *x, int nrhs, const int *done) { near_t<cd>(c, x, nrhs, done); }
void launch_gather(scd_ctx *c, const cd *x, cd *y, int nrhs, const int *done) {
    (void)x;
    gather_t<cd>(c, y, nrhs, done);
}
void run_matvec(scd_ctx *c, const cd *x, cd *y, int nrhs, const int *done) { run_matvec_t<cd>(c, x, y, nrhs, done); }
void run_matvec(scd_ctx *c, const cf *x, cf *y, int nrhs, const int *done) { run_matvec_t<cf>(c, x, y, nrhs, done); }
