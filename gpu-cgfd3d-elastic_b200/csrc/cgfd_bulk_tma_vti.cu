// cgfd_bulk_tma_vti.cu -- the bulk RK-stage kernel's instantiations for the vti medium (every
// operator direction, coefficient storage, wave policy and tile shape).
#include "cgfd_bulk_tma.cuh"

namespace cgfd {
template int launch_bulk_tma_med<MED_VTI>(int, int, int, const StageP &, const TmaP &, const SrcP &,
                                         const BulkTiles &, cudaStream_t);
template cudaError_t prepare_bulk_tma_med<MED_VTI>(int, int, int);
}  // namespace cgfd
