// Batch kernels of D3Q27 with split-velocity-FP16 moment storage.
#include "batch_dispatch.cuh"
MRLBM_BATCH_INSTANCE(27, __half, mrlbm::F_SPLITU)
