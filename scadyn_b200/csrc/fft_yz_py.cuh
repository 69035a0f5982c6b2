// Instantiates the fused y-z FFT pass (fft_yz.cuh) for y length SCD_YZ_PY and
// every z length, in both precisions; one translation unit per few y lengths,
// so that they compile side by side.
#include <cuda_runtime.h>

#include <algorithm>

#include "fft_yz.cuh"

template <int PY, typename C> void yz_launch(const YzLaunch<C> &l, int Pz) {
    switch (Pz) {
        case 16: yz_launch_t<PY, 16>(l); break;
        case 32: yz_launch_t<PY, 32>(l); break;
        case 40: yz_launch_t<PY, 40>(l); break;
        case 48: yz_launch_t<PY, 48>(l); break;
        case 64: yz_launch_t<PY, 64>(l); break;
        case 80: yz_launch_t<PY, 80>(l); break;
        case 96: yz_launch_t<PY, 96>(l); break;
        case 112: yz_launch_t<PY, 112>(l); break;
        case 128: yz_launch_t<PY, 128>(l); break;
        case 192: yz_launch_t<PY, 192>(l); break;
        default: break;
    }
}
#define SCD_YZ_INSTANCE(PY)                                    \
    template void yz_launch<PY, cf>(const YzLaunch<cf> &, int); \
    template void yz_launch<PY, cd>(const YzLaunch<cd> &, int);
