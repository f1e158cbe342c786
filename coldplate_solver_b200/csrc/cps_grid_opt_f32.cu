#include "cps_kernels.cuh"

CPS_GRID_OPTION_KERNELS(, float)
