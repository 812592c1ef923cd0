// The batch kernels of regression degree 3 (lsm_persistent.cuh).
#define FO_BATCH_DEGREE 3
#include "lsm_persistent.cuh"
