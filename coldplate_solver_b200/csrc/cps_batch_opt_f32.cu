#include "cps_kernels.cuh"

CPS_BATCH_OPTION_KERNELS(, float)
