// Launch tables of the insert's search and prune kernels (build_flag.cuh), one entry per element type,
// metric and lane width.
#include <algorithm>

#include "build_flag.cuh"
#include "internal.h"

namespace nbpg {

template <int DT, int MET, int VPL>
static cudaError_t search_v(uint32_t grid, uint32_t warps, size_t smem, const BuildFlagArgs &F, int *blocks, cudaStream_t st)
{
    if (blocks) {  // set-up: the shared memory this launch shape needs, and its residency
        cudaError_t e = raise_smem_limit(build_search_kernel<DT, MET, VPL>, smem);
        if (e == cudaSuccess)
            e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks, build_search_kernel<DT, MET, VPL>, int(warps * 32), smem);
        return e;
    }
    build_search_kernel<DT, MET, VPL><<<grid, warps * 32, smem, st>>>(F);
    return cudaGetLastError();
}

template <int DT, int MET>
static cudaError_t search_t(uint32_t grid, uint32_t warps, size_t smem, const BuildFlagArgs &F, int *blocks, cudaStream_t st)
{
    // row_geometry's choice with four words per lane wanted: rows of less than four words take one
    return F.B.s.vpl == 1 ? search_v<DT, MET, 1>(grid, warps, smem, F, blocks, st)
                          : search_v<DT, MET, 4>(grid, warps, smem, F, blocks, st);
}

template <int DT, int MET>
static cudaError_t prune_t(uint32_t grid, const BuildFlagArgs &F, const PruneLayout &lay, cudaStream_t st)
{
    if (grid == 0) return raise_smem_limit(build_prune_kernel<PRUNE_THREADS, DT, MET>, lay.bytes);
    build_prune_kernel<PRUNE_THREADS, DT, MET><<<grid, PRUNE_THREADS, lay.bytes, st>>>(F, lay);
    return cudaGetLastError();
}

// blocks != NULL: set the kernel up and report its residency, no launch
cudaError_t build_flag_search(uint32_t dtype, uint32_t metric, uint32_t grid, uint32_t warps, size_t smem,
                              const BuildFlagArgs &F, int *blocks, cudaStream_t st)
{
    const bool l2 = metric == NBPG_L2;
    switch (dtype) {
    case NBPG_U8:
        return l2 ? search_t<DT_U8, M_L2>(grid, warps, smem, F, blocks, st) : search_t<DT_U8, M_IP>(grid, warps, smem, F, blocks, st);
    case NBPG_I8:
        return l2 ? search_t<DT_I8, M_L2>(grid, warps, smem, F, blocks, st) : search_t<DT_I8, M_IP>(grid, warps, smem, F, blocks, st);
    default:
        return l2 ? search_t<DT_U4, M_L2>(grid, warps, smem, F, blocks, st) : search_t<DT_U4, M_IP>(grid, warps, smem, F, blocks, st);
    }
}

// grid 0: set the kernel's shared-memory limit only
cudaError_t build_flag_prune(uint32_t dtype, uint32_t metric, uint32_t grid, const BuildFlagArgs &F, const PruneLayout &lay,
                             cudaStream_t st)
{
    const bool l2 = metric == NBPG_L2;
    switch (dtype) {
    case NBPG_U8: return l2 ? prune_t<DT_U8, M_L2>(grid, F, lay, st) : prune_t<DT_U8, M_IP>(grid, F, lay, st);
    case NBPG_I8: return l2 ? prune_t<DT_I8, M_L2>(grid, F, lay, st) : prune_t<DT_I8, M_IP>(grid, F, lay, st);
    default: return l2 ? prune_t<DT_U4, M_L2>(grid, F, lay, st) : prune_t<DT_U4, M_IP>(grid, F, lay, st);
    }
}

}  // namespace nbpg
