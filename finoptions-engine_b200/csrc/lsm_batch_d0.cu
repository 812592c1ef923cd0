// The batch kernels of regression degree 0 (lsm_persistent.cuh).
#define FO_BATCH_DEGREE 0
#include "lsm_persistent.cuh"
