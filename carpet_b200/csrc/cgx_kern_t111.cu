// cgx_kern_t111.cu -- TMA-staged prolongation kernels, fused-multiply-add mode,
// families CC<2>, CC<3>, CC<4>, CC<5>, ENO, tile configuration 1 (TMA_CFGS), and their single-box kernels.
#include "cgx_kern_launch.cuh"

namespace cgx {
int klaunch_tma_f1_p1_c1(int variant, const Desc *d, const CUtensorMap *maps, const int2 *tmap,
                         long long ntiles, unsigned long long *counter, int *status, cudaStream_t s) {
  switch ((variant & ~(1 << 30)) / 4) { // bit 30: failure injection
  case 5: return kern::launch_tma_family<1, CC<2>, 1>(variant, d, maps, tmap, ntiles, counter, status, s);
  case 6: return kern::launch_tma_family<1, CC<3>, 1>(variant, d, maps, tmap, ntiles, counter, status, s);
  case 7: return kern::launch_tma_family<1, CC<4>, 1>(variant, d, maps, tmap, ntiles, counter, status, s);
  case 8: return kern::launch_tma_family<1, CC<5>, 1>(variant, d, maps, tmap, ntiles, counter, status, s);
  case 9: return kern::launch_tma_family<1, ENO, 1>(variant, d, maps, tmap, ntiles, counter, status, s);
  }
  return set_error(CGX_EINVAL, "bad prolongation variant %d", variant);
}
// single boxes (k_tma_box)
int klaunch_box_f1_p1(int variant, const Desc &d, const CUtensorMap *maps, int ntiles, int *status,
                      cudaStream_t s) {
  switch ((variant & ~(1 << 30)) / 4) {
  case 5: return kern::launch_box_family<1, CC<2>>(variant, d, maps, ntiles, status, s);
  case 6: return kern::launch_box_family<1, CC<3>>(variant, d, maps, ntiles, status, s);
  case 7: return kern::launch_box_family<1, CC<4>>(variant, d, maps, ntiles, status, s);
  case 8: return kern::launch_box_family<1, CC<5>>(variant, d, maps, ntiles, status, s);
  case 9: return kern::launch_box_family<1, ENO>(variant, d, maps, ntiles, status, s);
  }
  return set_error(CGX_EINVAL, "bad prolongation variant %d", variant);
}
} // namespace cgx
