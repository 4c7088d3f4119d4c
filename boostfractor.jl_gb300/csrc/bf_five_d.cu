// Fused stage kernels of the length 80, complex128.
#include "bf_five.cuh"

namespace bf {

void init_roots_five_d() { upload_roots(); }

int launch_five_d(int N, const FusedArgs<double2>& a, int nsteps, cudaStream_t st) {
  switch (N) {
    case 80: return launch_five_t<double, 80>(a, nsteps, st);
    default: return (int)cudaErrorInvalidValue;
  }
}

std::vector<int> five_variants_d(int N, int nby) {
  switch (N) {
    case 80: return five_variants_t<double, 80>(nby);
    default: return {kFusedRule};
  }
}

}  // namespace bf
