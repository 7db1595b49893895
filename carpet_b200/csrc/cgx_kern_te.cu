// cgx_kern_te.cu -- TMA-staged prolongation kernels of the cell-centred ENO
// families (CCENO<2>, CCENO<3>), both floating-point modes, batched (tile
// configuration TV_FIXED_CFG) and single boxes.
#include "cgx_kern_launch.cuh"

namespace cgx {
int klaunch_tma_eno(int fp, int variant, const Desc *d, const CUtensorMap *maps, const int2 *tmap,
                    long long ntiles, unsigned long long *counter, int *status, cudaStream_t s) {
  constexpr int C = TV_FIXED_CFG;
  const bool o2 = (variant & ~(1 << 30)) / 4 == 10; // bit 30: failure injection
  if (fp)
    return o2 ? kern::launch_tma_family<1, CCENO<2>, C>(variant, d, maps, tmap, ntiles, counter, status, s)
              : kern::launch_tma_family<1, CCENO<3>, C>(variant, d, maps, tmap, ntiles, counter, status, s);
  return o2 ? kern::launch_tma_family<0, CCENO<2>, C>(variant, d, maps, tmap, ntiles, counter, status, s)
            : kern::launch_tma_family<0, CCENO<3>, C>(variant, d, maps, tmap, ntiles, counter, status, s);
}
int klaunch_box_eno(int fp, int variant, const Desc &d, const CUtensorMap *maps, int ntiles, int *status,
                    cudaStream_t s) {
  const bool o2 = (variant & ~(1 << 30)) / 4 == 10;
  if (fp)
    return o2 ? kern::launch_box_family<1, CCENO<2>>(variant, d, maps, ntiles, status, s)
              : kern::launch_box_family<1, CCENO<3>>(variant, d, maps, ntiles, status, s);
  return o2 ? kern::launch_box_family<0, CCENO<2>>(variant, d, maps, ntiles, status, s)
            : kern::launch_box_family<0, CCENO<3>>(variant, d, maps, ntiles, status, s);
}
} // namespace cgx
