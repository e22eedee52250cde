// Host side of the FP64 M2L (m2l_parity.cuh; its instances are compiled per
// kernel family).
#include <cuda_runtime.h>

#include "internal.h"
#include "kernels.h"

namespace fmmb {

void m2l_parity_laplace(int p, const ParityArgs* a, cudaStream_t st);
void m2l_parity_helmholtz(int p, const ParityArgs* a, cudaStream_t st);
void m2l_parity_yukawa(int p, const ParityArgs* a, cudaStream_t st);

size_t parity_img_stride(int mode, int p) {
  const int te = parity_tiles((p + 1) * (p + 2) / 2), to = parity_tiles(p * (p + 1) / 2);
  return (mode == 1 ? 3 : 1) * (parity_block(te) + parity_block(to));
}

// a null: sets the shared-memory limit of the order's instance
static void dispatch(int mode, int p, const ParityArgs* a, cudaStream_t st) {
  if (mode == 0) m2l_parity_laplace(p, a, st);
  else if (mode == 1) m2l_parity_helmholtz(p, a, st);
  else m2l_parity_yukawa(p, a, st);
}

void prepare_m2l_parity(int mode, int p) { dispatch(mode, p, nullptr, nullptr); }

void launch_m2l_parity(int mode, const ParityArgs& a, cudaStream_t st) {
  if (a.ntile <= 0) return;
  dispatch(mode, a.p, &a, st);
  FMMB_CHECK_LAUNCH();
}

}  // namespace fmmb
