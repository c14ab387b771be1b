// Split refracted kernels (fast pass and fix-up) for the joint solve through 4 interfaces.
#include "ss_refracted_split.cuh"

namespace ss {

int split_launch_ni4(RefArgs &a, const RefSplitConsts &k, const Plan &p,
                     size_t smem, cudaStream_t st) {
  return lean_joint(a) ? launch_split_r<lean_class(4)>(a, k, p, smem, st)
                       : launch_split_r<4>(a, k, p, smem, st);
}

int refracted_batch_launch_ni4(const RefBatchJob *jobs, int n_jobs,
                               long long n_items, long long n_words,
                               unsigned long long *counter, int rough_kind,
                               bool plain, int ctas, size_t smem,
                               size_t fix_smem, cudaStream_t st) {
  return ref_batch_launch_r<4>(jobs, n_jobs, n_items, n_words, counter,
                               rough_kind, plain, ctas, smem, fix_smem, st);
}

int refracted_batch_occupancy_ni4(int rough_kind, bool plain, size_t smem) {
  return ref_batch_occupancy<4>(rough_kind, plain, smem);
}

int refracted_batch_launch_nilean4(const RefBatchJob *jobs, int n_jobs,
                                   long long n_items, long long n_words,
                                   unsigned long long *counter,
                                   int rough_kind, bool plain, int ctas,
                                   size_t smem, size_t fix_smem,
                                   cudaStream_t st) {
  return ref_batch_launch_r<lean_class(4)>(jobs, n_jobs, n_items, n_words,
                                           counter, rough_kind, plain, ctas,
                                           smem, fix_smem, st);
}

int refracted_batch_occupancy_nilean4(int rough_kind, bool plain,
                                      size_t smem) {
  return ref_batch_occupancy<lean_class(4)>(rough_kind, plain, smem);
}

}  // namespace ss
