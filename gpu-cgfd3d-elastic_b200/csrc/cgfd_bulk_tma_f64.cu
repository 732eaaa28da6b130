// cgfd_bulk_tma_f64.cu -- the bulk RK-stage kernel of the FP64 build, iso and VTI media (the 21-Cij
// medium's 31 double coefficient fields do not fit beside the wave ring at a useful occupancy; it
// runs the direct-load kernel). Tiles by shared memory: iso 32x4 at two blocks per SM (113 KB
// each), VTI 32x8 at one (202 KB), both 8 warps with 255 registers.
#include "cgfd_bulk_tma.cuh"

namespace cgfd {

template <int MED> struct TileShape64;
template <> struct TileShape64<MED_ISO> { static constexpr int TYT = 4, MINB = 2; };
template <> struct TileShape64<MED_VTI> { static constexpr int TYT = 8, MINB = 1; };

template <int MED>
static cudaError_t each_dir(int code, const StagePT<double> *p, const TmaP *tm, const SrcPT<double> *sp, const BulkTiles *t,
                            cudaStream_t st) {
  constexpr int TYT = TileShape64<MED>::TYT, MINB = TileShape64<MED>::MINB;
  using S = BulkSmem<MED, TYT, double, double, MINB>;
  static_assert(S::BYTES <= 227 * 1024, "one block must fit an SM's shared memory");
  cudaError_t e = cudaSuccess;
#define CASE(c)                                                                                                \
  if (!p) {                                                                                                    \
    if (e == cudaSuccess)                                                                                      \
      e = cudaFuncSetAttribute(                                                                                \
          k_stage_bulk_tma<MED, (c)&1, ((c) >> 1) & 1, ((c) >> 2) & 1, TYT, MINB, double, 0>,                  \
          cudaFuncAttributeMaxDynamicSharedMemorySize, S::BYTES);                                              \
  } else if (code == c) {                                                                                      \
    k_stage_bulk_tma<MED, (c)&1, ((c) >> 1) & 1, ((c) >> 2) & 1, TYT, MINB, double, 0>                         \
        <<<t->n, dim3(TX, TYT), S::BYTES, st>>>(*p, *tm, *sp, t->list);                                             \
  }
  CASE(0) CASE(1) CASE(2) CASE(3) CASE(4) CASE(5) CASE(6) CASE(7)
#undef CASE
  return e;
}

bool tma64_supported(int med) { return med == MED_ISO || med == MED_VTI; }
int tma64_tile_y(int med) { return med == MED_ISO ? TileShape64<MED_ISO>::TYT : TileShape64<MED_VTI>::TYT; }
int tma64_resident(int med) { return med == MED_ISO ? TileShape64<MED_ISO>::MINB : TileShape64<MED_VTI>::MINB; }

cudaError_t tma64_prepare(int med) {
  return med == MED_ISO ? each_dir<MED_ISO>(0, nullptr, nullptr, nullptr, nullptr, nullptr)
                        : each_dir<MED_VTI>(0, nullptr, nullptr, nullptr, nullptr, nullptr);
}

int launch_stage_bulk_tma64(int med, const StagePT<double> &p, const TmaP &tm, const SrcPT<double> &sp,
                            const BulkTiles &t, cudaStream_t st) {
  if (t.n <= 0) return 0;
  const int code = p.dir[0] | (p.dir[1] << 1) | (p.dir[2] << 2);
  if (med == MED_ISO) each_dir<MED_ISO>(code, &p, &tm, &sp, &t, st);
  else each_dir<MED_VTI>(code, &p, &tm, &sp, &t, st);
  return 1;
}

}  // namespace cgfd
