// stage2d_tall.cu -- the mixed form's 2D stage kernel (stage2d.cuh) at a
// 32x16 tile of 512 threads, for grids that give every SM a tile of that size.
// A taller tile derives and stages 1.63 region cells per cell instead of
// 2.08; the FP64 form, whose arrays then allow one block fewer per SM, gains
// nothing from it (4096^2: 6.38 against 6.43 ms per RK4 step; 512x256: 0.126
// against 0.115).
#include "kernels.cuh"

namespace smaug {
namespace t32x16 {

constexpr int TX = 32, TY = 16;
constexpr int RX = TX + 2 * HALO, RY = TY + 2 * HALO;
constexpr int RC = RX * RY;
constexpr int NTHREADS = TX * TY;

#undef SMAUG_MINB2D_MIX
#define SMAUG_MINB2D_MIX 2
#include "stage2d.cuh"

}  // namespace t32x16

cudaError_t launch_stage2d_tall(int mode, const KParams& K, const KBufs& B, cudaStream_t st) {
  return mode == SMAUG_INT_EULER ? t32x16::launch_stage2d<SMAUG_INT_EULER, true>(K, B, st)
                                 : t32x16::launch_stage2d<SMAUG_INT_RK4, true>(K, B, st);
}

cudaError_t stage2d_tall_set_attributes() {
  cudaError_t e;
#define SMAUG_ATTR2(M, BG)                                              \
  if ((e = t32x16::stage2d_attr<M, BG, true, false>())) return e;       \
  if ((e = t32x16::stage2d_attr<M, BG, true, true>())) return e;
  SMAUG_ATTR2(SMAUG_INT_EULER, true)
  SMAUG_ATTR2(SMAUG_INT_EULER, false)
  SMAUG_ATTR2(SMAUG_INT_RK4, true)
  SMAUG_ATTR2(SMAUG_INT_RK4, false)
#undef SMAUG_ATTR2
  return cudaSuccess;
}

}  // namespace smaug
