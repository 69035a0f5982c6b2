#include "fft_yz_py.cuh"

SCD_YZ_INSTANCE(40)
SCD_YZ_INSTANCE(48)
