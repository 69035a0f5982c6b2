#include "fft_yz_py.cuh"

SCD_YZ_INSTANCE(16)
SCD_YZ_INSTANCE(32)
