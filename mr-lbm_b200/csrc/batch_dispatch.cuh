// batch_dispatch.cuh -- shape and launch of the batched kernel for one
// (lattice, storage) pair; instantiated in batch_q*_*.cu so the kernels
// compile in parallel translation units.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>

#include "batch_kernel.cuh"
#include "domain.h"

namespace mrlbm {

// shared memory and persistent grid of the batch kernel of one tile height
template <int Q, typename T, int S, int TYI>
static mrlbm_status batch_shape_t(size_t* smem, int* grid, int sms)
{
    *smem = ZSmem<Q, T, TYI, batch_npm<T, S>(), false, BATCH_STATIC_SMEM, batch_stages(Q)>::bytes;
    cudaError_t e =
        cudaFuncSetAttribute(batch_step<Q, T, S, TYI>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)*smem);
    if (e != cudaSuccess) return fail(MRLBM_ECUDA, "batch attribute: %s", cudaGetErrorString(e));
    int per_sm = 1;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, batch_step<Q, T, S, TYI>, 32 * (TYI + 2), *smem);
    *grid = sms * std::max(per_sm, 1);
    return MRLBM_OK;
}

// both tile heights, by tile kind
template <int Q, typename T, int S>
mrlbm_status batch_shapes(size_t* smem, int* grid, int sms)
{
    mrlbm_status st = batch_shape_t<Q, T, S, TYI_BULK>(smem + tile_kind(TYI_BULK), grid + tile_kind(TYI_BULK), sms);
    return st ? st
              : batch_shape_t<Q, T, S, TYI_WALL>(smem + tile_kind(TYI_WALL), grid + tile_kind(TYI_WALL), sms);
}

template <int Q, typename T, int S>
void batch_launch(int rows, const size_t* smem, const int* grid, const BatchDomain* doms, const BatchItem* items,
                  BatchCtl* ctl, cudaStream_t s)
{
    const int k = tile_kind(rows);
    if (rows == TYI_BULK)
        batch_step<Q, T, S, TYI_BULK><<<grid[k], 32 * (TYI_BULK + 2), smem[k], s>>>(doms, items, ctl);
    else
        batch_step<Q, T, S, TYI_WALL><<<grid[k], 32 * (TYI_WALL + 2), smem[k], s>>>(doms, items, ctl);
}

}  // namespace mrlbm

#define MRLBM_BATCH_INSTANCE(Q, T, S)                                                                              \
    template mrlbm_status mrlbm::batch_shapes<Q, T, S>(size_t*, int*, int);                                         \
    template void mrlbm::batch_launch<Q, T, S>(int, const size_t*, const int*, const mrlbm::BatchDomain*,          \
                                               const mrlbm::BatchItem*, mrlbm::BatchCtl*, cudaStream_t);
