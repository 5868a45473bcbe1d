// Boussinesq phi stage on the rows of the FP64 contractions (legendre_f64.cu).
#include "nl_bouss.cuh"

namespace mt {

int launch_nl_bouss_f64(bool mag, bool chem, const NlBoussArgs& a, cudaStream_t st) {
  return launch_nl_bouss_io<false>(mag, chem, a, st);
}

}  // namespace mt
