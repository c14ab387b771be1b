// Adjoint of the split refracted kernel: the single-crossing path's
// instantiations (device code in ss_refracted_adjoint.cuh).
#include "ss_refracted_adjoint.cuh"

namespace ss {

int adjoint_launch_one(RefArgs &a, const RefSplitConsts &k, const AdjArgs &j,
                       size_t smem, cudaStream_t st) {
  return adjoint_launch_ni<kOneNI>(a, k, j, smem, st);
}

}  // namespace ss
