// FP64 M2L of the Yukawa kernel: the instances of m2l_parity.cuh.
#include "m2l_parity.cuh"

namespace fmmb {
void m2l_parity_yukawa(int p, const ParityArgs* a, cudaStream_t st) { parity::run<2, 1>(p, a, st); }
}  // namespace fmmb
