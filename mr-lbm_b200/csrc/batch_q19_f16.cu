// Batch kernels of D3Q19 with FP16 moment storage.
#include "batch_dispatch.cuh"
MRLBM_BATCH_INSTANCE(19, __half, 0)
