// Batch kernels of D3Q19 with FP32 moment storage.
#include "batch_dispatch.cuh"
MRLBM_BATCH_INSTANCE(19, float, 0)
