// The batch kernels of regression degree 4 (lsm_persistent.cuh).
#define FO_BATCH_DEGREE 4
#include "lsm_persistent.cuh"
