// The batch kernels of regression degree 2 (lsm_persistent.cuh).
#define FO_BATCH_DEGREE 2
#include "lsm_persistent.cuh"
