#include "fft_yz_py.cuh"

SCD_YZ_INSTANCE(128)
SCD_YZ_INSTANCE(192)
