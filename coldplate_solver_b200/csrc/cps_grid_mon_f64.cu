#include "cps_kernels.cuh"

CPS_GRID_MONITOR_KERNELS(, double)
