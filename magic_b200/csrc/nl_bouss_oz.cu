// Boussinesq phi stage on the rows of the digit-split contractions (ozaki.cu).
#include "nl_bouss.cuh"

namespace mt {

int launch_nl_bouss_oz(bool mag, bool chem, const NlBoussArgs& a, cudaStream_t st) {
  return launch_nl_bouss_io<true>(mag, chem, a, st);
}

}  // namespace mt
