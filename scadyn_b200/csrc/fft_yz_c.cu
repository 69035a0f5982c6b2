#include "fft_yz_py.cuh"

SCD_YZ_INSTANCE(64)
SCD_YZ_INSTANCE(80)
