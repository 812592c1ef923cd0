// The batch kernels of regression degree 1 (lsm_persistent.cuh).
#define FO_BATCH_DEGREE 1
#include "lsm_persistent.cuh"
