// Fused stage kernels of the lengths 40, 80 and 160, complex64.
#include "bf_five.cuh"

namespace bf {

void init_roots_five_f() { upload_roots(); }

int launch_five_f(int N, const FusedArgs<float2>& a, int nsteps, cudaStream_t st) {
  switch (N) {
    case 40: return launch_five_t<float, 40>(a, nsteps, st);
    case 80: return launch_five_t<float, 80>(a, nsteps, st);
    case 160: return launch_five_t<float, 160>(a, nsteps, st);
    default: return (int)cudaErrorInvalidValue;
  }
}

std::vector<int> five_variants_f(int N, int nby) {
  switch (N) {
    case 40: return five_variants_t<float, 40>(nby);
    case 80: return five_variants_t<float, 80>(nby);
    case 160: return five_variants_t<float, 160>(nby);
    default: return {kFusedRule};
  }
}

}  // namespace bf
