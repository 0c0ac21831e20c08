// Instantiations of the 3-center derivative kernels of bra class (l1, l2) = (3, 1), see grad3c.cuh.
#include "grad3c.cuh"

namespace dfjk {

bool launch_grad3c_31(int lc, unsigned npair, cudaStream_t s, const Grad3cArgs& a) {
  return launch_grad3c_lc<3, 1>(lc, npair, s, a);
}

void launch_pair_deriv_31(int64_t npp, cudaStream_t s, const PairDerivArgs& a) {
  launch_pair_deriv_t<3, 1>(npp, s, a);
}

}  // namespace dfjk
