// cgfd_bulk_tma_vis.cu -- the bulk RK-stage kernel's visco-elastic form: the iso stage with the
// attenuation of each point between its right-hand side and its RK combine, so that the 9-field
// right-hand side never reaches memory. Bound by the memory variables' own traffic (18 NM floats
// read and 12 NM written per cell at stages 1-2 beside the iso stage's 45), and by latency: four blocks
// per SM of 32x4 columns at 128 registers run 160x160x80 with 3 mechanisms in 1199 us per step, three
// at 168 in 1244.
#include "cgfd_bulk_tma.cuh"

namespace cgfd {

constexpr int kVisTY = 4, kVisBlocks = 4;

template <int DX, int DY, int DZ, int NM>
__global__ void __launch_bounds__(TX *kVisTY, kVisBlocks)
    k_stage_bulk_vis(const __grid_constant__ StageP p, const __grid_constant__ TmaP tm,
                     const __grid_constant__ VisP v, const __grid_constant__ SrcP sp, const int4 *__restrict__ tiles) {
  const int4 tl = __ldg(tiles + blockIdx.x);
  bulk_tile<MED_ISO, DX, DY, DZ, kVisTY, kVisBlocks, float, 0, NM>(p, tm, tl, sp, &v);
}

using VisSmem = BulkSmem<MED_ISO, kVisTY, float, float, kVisBlocks>;

template <int NM>
static cudaError_t for_each_dir(int code, const StageP *p, const TmaP *tm, const VisP *v, const SrcP *sp, const BulkTiles *t,
                                cudaStream_t st) {
  cudaError_t e = cudaSuccess;
#define CASE(c)                                                                                                  \
  if (!p) {                                                                                                      \
    if (e == cudaSuccess)                                                                                        \
      e = cudaFuncSetAttribute(k_stage_bulk_vis<(c)&1, ((c) >> 1) & 1, ((c) >> 2) & 1, NM>,                      \
                               cudaFuncAttributeMaxDynamicSharedMemorySize, VisSmem::BYTES);                     \
  } else if (code == c) {                                                                                        \
    k_stage_bulk_vis<(c)&1, ((c) >> 1) & 1, ((c) >> 2) & 1, NM>                                                  \
        <<<t->n, dim3(TX, kVisTY), VisSmem::BYTES, st>>>(*p, *tm, *v, *sp, t->list);                                  \
  }
  CASE(0) CASE(1) CASE(2) CASE(3) CASE(4) CASE(5) CASE(6) CASE(7)
#undef CASE
  return e;
}

int vis_bulk_max_mechanisms() { return 4; }
int vis_bulk_resident() { return kVisBlocks; }

static cudaError_t dispatch(int nmax, const StageP *p, const TmaP *tm, const VisP *v, const SrcP *sp, const BulkTiles *t,
                            cudaStream_t st) {
  const int code = p ? p->dir[0] | (p->dir[1] << 1) | (p->dir[2] << 2) : 0;
  switch (nmax) {
    case 1: return for_each_dir<1>(code, p, tm, v, sp, t, st);
    case 2: return for_each_dir<2>(code, p, tm, v, sp, t, st);
    case 3: return for_each_dir<3>(code, p, tm, v, sp, t, st);
    default: return for_each_dir<4>(code, p, tm, v, sp, t, st);
  }
}

cudaError_t tma_prepare_vis(int nmax) { return dispatch(nmax, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr); }

int launch_stage_bulk_vis(const StageP &p, const TmaP &tm, const VisP &v, const SrcP &sp, const BulkTiles &t,
                          cudaStream_t st) {
  if (t.n <= 0) return 0;
  dispatch(v.nmax, &p, &tm, &v, &sp, &t, st);
  return 1;
}

}  // namespace cgfd
