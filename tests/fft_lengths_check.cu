// Host check of the fused y-z FFT pass (scadyn_b200/csrc/fft_yz.cuh) over
// every length it takes, at the edges of the padding (N = P/2 and the smallest
// N that selects P) and with x on both sides of Px/2: the pass against a direct
// separable DFT convolution in double precision, with NaN canaries behind the
// plane and the shared-memory image.
#include <cmath>
#include <complex>
#include <cstdio>
#include <vector>

#include "fft_yz.cuh"

typedef std::complex<double> Z;
template <typename C> C mk(double r, double i);
template <> cd mk<cd>(double r, double i) { return make_double2(r, i); }
template <> cf mk<cf>(double r, double i) { return make_float2((float)r, (float)i); }
static unsigned g_state = 777u;
static double urand() {
    g_state = g_state * 1664525u + 1013904223u;
    return (g_state >> 8) / 16777216.0 - 0.5;
}
static int bad = 0;

template <int PY, int PZ, typename C> void check(int Ny, int Nz, int Px, int x, double bound) {
    YzDims D{Px / 2, Ny, Nz, yz_round8(Nz), Px, Px / 2 + 1, PY / 2 + 1, PZ / 2 + 1};
    const int CAN = 64;
    const C nan = mk<C>(std::nan(""), std::nan(""));
    std::vector<C> W(Nz * Ny + CAN, nan), F((size_t)D.Hx * D.Hy * D.Hz), twy(PY), twz(PZ);
    std::vector<Z> in(Nz * Ny);
    for (int i = 0; i < Nz * Ny; ++i) {
        W[i] = mk<C>(urand(), urand());
        in[i] = Z((double)W[i].x, (double)W[i].y);
    }
    for (auto &f : F) f = mk<C>(urand(), urand());
    for (int i = 0; i < PY; ++i) twy[i] = mk<C>(std::cos(-2 * M_PI * i / PY), std::sin(-2 * M_PI * i / PY));
    for (int i = 0; i < PZ; ++i) twz[i] = mk<C>(std::cos(-2 * M_PI * i / PZ), std::sin(-2 * M_PI * i / PZ));
    const long long ns = yz_smem_elems<PY, PZ>(D.Nz, 32);      // one warp's exchange buffer
    std::vector<C> sm(ns + CAN, nan);
    yz_plane_host<PY, PZ, C>(W.data(), F.data(), twy.data(), twz.data(), x, D, sm.data());
    bool can = true;
    for (int i = 0; i < CAN; ++i) can = can && std::isnan((double)W[Nz * Ny + i].x) && std::isnan((double)sm[ns + i].x);
    auto w = [](long long e, int P) { return std::polar(1.0, 2 * M_PI * (double)(e % P) / P); };
    const int fx = yz_fold(x, Px);
    std::vector<Z> T1(Nz * PY), U(PZ * PY), T2(Nz * PY);
    for (int z = 0; z < Nz; ++z)
        for (int ky = 0; ky < PY; ++ky)
            for (int y = 0; y < Ny; ++y) T1[z * PY + ky] += in[z * Ny + y] * std::conj(w((long long)ky * y, PY));
    for (int kz = 0; kz < PZ; ++kz)
        for (int ky = 0; ky < PY; ++ky) {
            Z s = 0;
            for (int z = 0; z < Nz; ++z) s += T1[z * PY + ky] * std::conj(w((long long)kz * z, PZ));
            const C f = F[((long long)fx * D.Hy + yz_fold(ky, PY)) * D.Hz + yz_fold(kz, PZ)];
            U[kz * PY + ky] = s * Z((double)f.x, (double)f.y);
        }
    for (int z = 0; z < Nz; ++z)
        for (int ky = 0; ky < PY; ++ky)
            for (int kz = 0; kz < PZ; ++kz) T2[z * PY + ky] += U[kz * PY + ky] * w((long long)kz * z, PZ);
    double err = 0, nrm = 0;
    for (int z = 0; z < Nz; ++z)
        for (int y = 0; y < Ny; ++y) {
            Z s = 0;
            for (int ky = 0; ky < PY; ++ky) s += T2[z * PY + ky] * w((long long)ky * y, PY);
            err += std::norm(Z((double)W[z * Ny + y].x, (double)W[z * Ny + y].y) - s);
            nrm += std::norm(s);
        }
    const double e = std::sqrt(err / nrm);
    std::printf("%d x %d, %d x %d nodes, %s: %.3e%s\n", PY, PZ, Ny, Nz, sizeof(C) == 16 ? "f64" : "f32", e, can ? "" : " canary");
    if (!(e < bound) || !can) bad = 1;
}
template <int PY, int PZ> void pair(int Ny, int Nz) {
    check<PY, PZ, cd>(Ny, Nz, 64, 5, 1e-13);
    check<PY, PZ, cf>(Ny, Nz, 64, 50, 2e-6);
}

int main() {
    pair<16, 192>(8, 65);
    pair<32, 16>(16, 5);
    pair<40, 32>(18, 9);
    pair<48, 40>(22, 20);
    pair<64, 48>(26, 24);
    pair<80, 64>(40, 32);
    pair<96, 80>(42, 33);
    pair<112, 96>(56, 48);
    pair<128, 112>(58, 50);
    pair<192, 128>(96, 64);
    return bad;
}
