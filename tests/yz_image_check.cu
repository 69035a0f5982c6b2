// The shared-memory image that yz_smem_elems sizes by default is the one the
// host pass of fft_yz.cuh uses, to its last exchange line, so that a check that
// puts canaries behind it sees a write past the pass's end: the last line of the
// image is written, nothing behind it is.
#include <cmath>
#include <cstdio>
#include <vector>

#include "fft_yz.cuh"

template <int PY, int PZ> int check(int Ny, int Nz) {
    YzDims D;
    D.Nx = 8; D.Ny = Ny; D.Nz = Nz; D.NzR = yz_round8(Nz); D.Px = 16;
    D.Hx = 9; D.Hy = PY / 2 + 1; D.Hz = PZ / 2 + 1;
    const cd one = make_double2(1.0, 0.0), nan = make_double2(std::nan(""), std::nan(""));
    std::vector<cd> W(Nz * Ny, one), F((size_t)D.Hx * D.Hy * D.Hz, one), twy(PY, one), twz(PZ, one);
    const long long n = yz_smem_elems<PY, PZ>(Nz), line = std::max(HalfLine<PY>::ES, HalfLine<PZ>::ES);
    std::vector<cd> sm(n + 4096, nan);
    yz_plane_host<PY, PZ, cd>(W.data(), F.data(), twy.data(), twz.data(), 0, D, sm.data());
    bool used = false, past = false;
    for (long long i = n - line; i < n; ++i) used = used || !std::isnan(sm[i].x);
    for (size_t i = n; i < sm.size(); ++i) past = past || !std::isnan(sm[i].x);
    if (!used || past) std::printf("PY %d PZ %d: last line written %d, written behind the image %d\n", PY, PZ, used, past);
    return !used || past;
}

int main() {
    return check<16, 16>(8, 8) + check<40, 32>(20, 16) + check<48, 40>(22, 18) + check<64, 48>(31, 24) +
           check<112, 80>(54, 40) + check<64, 192>(32, 96);
}
