#include "fft_yz_py.cuh"

SCD_YZ_INSTANCE(96)
SCD_YZ_INSTANCE(112)
