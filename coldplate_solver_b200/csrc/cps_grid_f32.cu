#include "cps_kernels.cuh"

CPS_GRID_KERNELS(, float)
