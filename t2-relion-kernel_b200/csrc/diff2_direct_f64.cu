// diff2_direct_f64.cu -- FP64 instantiations of the CUDA-core coarse diff2.
#include "direct_kernel.cuh"

namespace b200d2 {

template <bool CC>
static int launch_f64(const DirectArgs& a, int P, int K, cudaStream_t s) {
  const int tt = dir_rows(a.T);
  if (tt <= 1) return dir_launch_tt<PairD, 512, 16, 1, CC>(a, P, K, s);
  if (tt <= 2) return dir_launch_tt<PairD, 512, 16, 2, CC>(a, P, K, s);
  if (tt <= 4) return dir_launch_tt<PairD, 512, 16, 4, CC>(a, P, K, s);
  return dir_launch_tt<PairD, 512, 16, 8, CC>(a, P, K, s);
}

int launch_direct_f64(const DirectArgs& a, int P, cudaStream_t s) {
  const int K = dir_listed(a.view, a.N_img);
  return a.cc ? launch_f64<true>(a, P, K, s) : launch_f64<false>(a, P, K, s);
}

}  // namespace b200d2
