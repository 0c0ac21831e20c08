// Instantiations of the 3-center derivative kernels of bra class (l1, l2) = (1, 0), see grad3c.cuh.
#include "grad3c.cuh"

namespace dfjk {

bool launch_grad3c_10(int lc, unsigned npair, cudaStream_t s, const Grad3cArgs& a) {
  return launch_grad3c_lc<1, 0>(lc, npair, s, a);
}

void launch_pair_deriv_10(int64_t npp, cudaStream_t s, const PairDerivArgs& a) {
  launch_pair_deriv_t<1, 0>(npp, s, a);
}

}  // namespace dfjk
