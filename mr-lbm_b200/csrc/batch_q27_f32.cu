// Batch kernels of D3Q27 with FP32 moment storage.
#include "batch_dispatch.cuh"
MRLBM_BATCH_INSTANCE(27, float, 0)
