// Instantiates the fused y-z FFT pass (fft_yz.cuh) for y length SCD_YZ_PY and
// every z length, in both precisions; one translation unit per few y lengths,
// so that they compile side by side.
#include <cuda_runtime.h>

#include <algorithm>

#include "fft_yz.cuh"

template <int PY, typename C> cudaError_t yz_launch(const YzLaunch<C> &l, int Pz) {
    switch (Pz) {
        case 16: return yz_launch_t<PY, 16>(l);
        case 32: return yz_launch_t<PY, 32>(l);
        case 40: return yz_launch_t<PY, 40>(l);
        case 48: return yz_launch_t<PY, 48>(l);
        case 64: return yz_launch_t<PY, 64>(l);
        case 80: return yz_launch_t<PY, 80>(l);
        case 96: return yz_launch_t<PY, 96>(l);
        case 112: return yz_launch_t<PY, 112>(l);
        case 128: return yz_launch_t<PY, 128>(l);
        case 192: return yz_launch_t<PY, 192>(l);
        default: return cudaErrorInvalidValue;
    }
}
#define SCD_YZ_INSTANCE(PY)                                            \
    template cudaError_t yz_launch<PY, cf>(const YzLaunch<cf> &, int); \
    template cudaError_t yz_launch<PY, cd>(const YzLaunch<cd> &, int);
