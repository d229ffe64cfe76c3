// Batch kernels of D3Q27 with FP16 moment storage.
#include "batch_dispatch.cuh"
MRLBM_BATCH_INSTANCE(27, __half, 0)
