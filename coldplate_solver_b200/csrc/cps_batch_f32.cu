#include "cps_kernels.cuh"

CPS_BATCH_KERNELS(, float)
