// diff2_direct.cu -- plain CUDA-core coarse diff2: the FP32 drop-in, the FP64
// form and the CC scores (kernel and tile choice in direct_kernel.cuh).
#include "direct_kernel.cuh"

namespace b200d2 {

int launch_direct_f64(const DirectArgs& a, int P, cudaStream_t s);  // diff2_direct_f64.cu

template <bool CC>
static int launch_f32(const DirectArgs& a, int P, int K, cudaStream_t s) {
  const int rows = dir_rows(a.T);
  // up to 32 translations the fetches weigh most: two CTAs of 256 threads a SM
  // hide each other's barriers, unless the tiles are too few to give half of the
  // SMs a 128-orientation one, where the larger CTAs' clusters spread them better
  // (image 64, two translations' heights: 64 particles x 4608 orientations 4.07
  // and 3.77 ms, 64 x 400 0.52 and 0.41; 8 x 400 80 and 103 us, 1 x 4608 96 and
  // 104 us; 49 translations: 8 x 1703 at image 96 0.74 and 1.03 ms)
  if (rows <= 2 && 2LL * P * ((a.O + 127) / 128) >= dir_sms())
    return rows == 1 ? dir_launch_tt<PairF, 256, 16, 1, CC>(a, P, K, s) : dir_launch_tt<PairF, 256, 16, 2, CC>(a, P, K, s);
  switch (rows) {
    case 1: return dir_launch_tt<PairF, 512, 16, 1, CC>(a, P, K, s);
    case 2: return dir_launch_tt<PairF, 512, 16, 2, CC>(a, P, K, s);
    case 3: return dir_launch_tt<PairF, 512, 16, 3, CC>(a, P, K, s);
    case 4: return dir_launch_tt<PairF, 512, 32, 2, CC>(a, P, K, s);
    case 5: return dir_launch_tt<PairF, 512, 16, 5, CC>(a, P, K, s);
    case 6: return dir_launch_tt<PairF, 512, 32, 3, CC>(a, P, K, s);
    default: return dir_launch_tt<PairF, 512, 32, 4, CC>(a, P, K, s);
  }
}

static int launch_direct_f32(const DirectArgs& a, int P, cudaStream_t s) {
  const int K = dir_listed(a.view, a.N_img);
  return a.cc ? launch_f32<true>(a, P, K, s) : launch_f32<false>(a, P, K, s);
}

int minloc_preload();  // minloc.cu

// Every kernel a FP32 request can launch.
int direct_preload() {
  cudaError_t e = dir_preload_tt<PairF, 256, 16, 1, false>();
  if (e == cudaSuccess) e = dir_preload_tt<PairF, 256, 16, 2, false>();
  if (e == cudaSuccess) e = dir_preload_tt<PairF, 512, 16, 1, false>();
  if (e == cudaSuccess) e = dir_preload_tt<PairF, 512, 16, 2, false>();
  if (e == cudaSuccess) e = dir_preload_tt<PairF, 512, 16, 3, false>();
  if (e == cudaSuccess) e = dir_preload_tt<PairF, 512, 32, 2, false>();
  if (e == cudaSuccess) e = dir_preload_tt<PairF, 512, 16, 5, false>();
  if (e == cudaSuccess) e = dir_preload_tt<PairF, 512, 32, 3, false>();
  if (e == cudaSuccess) e = dir_preload_tt<PairF, 512, 32, 4, false>();
  return e == cudaSuccess ? minloc_preload() : status_from_cuda(e);
}

static int check_common(const b200d2_view* view, const void* tx, const void* ty,
                        const void* corr, const void* re, const void* im,
                        const void* eul, const void* out, size_t O, size_t T,
                        size_t N_img) {
  if (!view || !tx || !ty || !corr || !re || !im || !eul || !out)
    return B200D2_ERR_INVALID;
  if (O > 0x7fffffff || T > 0x7fffffff || N_img > 0x7fffffff) return B200D2_ERR_INVALID;
  if ((size_t)view->imgX * (size_t)view->imgY < N_img) return B200D2_ERR_INVALID;
  if (view->mdlZ == 0) return B200D2_ERR_UNSUPPORTED;
  if (view->interp == B200D2_INTERP_TEXTURE && (!view->tex_re || !view->tex_im))
    return B200D2_ERR_INVALID;
  if (view->interp == B200D2_INTERP_LINEAR && (!view->lin_re || !view->lin_im))
    return B200D2_ERR_INVALID;
  if (view->imgX > 32767 || view->imgY > 32767) return B200D2_ERR_UNSUPPORTED;
  return B200D2_OK;
}

// Batched entry used by the library's own batch API and benchmarks: P
// particles sharing eulers and translations, images and outputs strided.
int direct_batch(const b200d2_view& view, const float* eulers, const float* tx,
                 const float* ty, const float* re, const float* im,
                 const float* corr, long long img_stride, void* out,
                 long long out_stride, int O, int T, int N_img, int P,
                 bool fp64, int filter_img, cudaStream_t s, int cc, int accumulate) {
  DirectArgs a;
  a.view = view;
  a.eulers = eulers;
  a.trans_x = tx;
  a.trans_y = ty;
  a.re = re;
  a.im = im;
  a.corr = corr;
  a.diff2 = out;
  a.img_stride = img_stride;
  a.out_stride = out_stride;
  a.O = O;
  a.T = T;
  a.N_img = N_img;
  a.o_tiles = 1;
  a.exw = a.off_tab = 0;
  a.filter_img = filter_img;
  a.cc = cc;
  a.accumulate = accumulate;
  if (a.O <= 0 || a.T <= 0 || a.N_img <= 0 || P <= 0) return B200D2_OK;
  return fp64 ? launch_direct_f64(a, P, s) : launch_direct_f32(a, P, s);
}

}  // namespace b200d2

namespace b200d2 {
int single_particle_tc(const b200d2_view& v, const float* tx, const float* ty, const float* corr, const float* re,
                       const float* im, const float* eulers, float* diff2s, int O, int T, int N_img, int precision,
                       cudaStream_t s);
}  // namespace b200d2

extern "C" int b200d2_diff2_coarse(const b200d2_view* view,
                                   const float* d_trans_x,
                                   const float* d_trans_y, const float* d_corr,
                                   const float* d_real, const float* d_imag,
                                   const float* d_eulers, float* d_diff2s,
                                   size_t O, size_t T, size_t N_img,
                                   void* stream, int precision) {
  b200d2::NvtxRange range("b200d2_diff2_coarse");
  int st = b200d2::check_common(view, d_trans_x, d_trans_y, d_corr, d_real,
                                d_imag, d_eulers, d_diff2s, O, T, N_img);
  if (st != B200D2_OK) return st;
  if (b200d2::is_tc_precision(precision)) {
    if (O > 0x7fffffff || T > 0x7fffffff || N_img > 0x7fffffff) return B200D2_ERR_UNSUPPORTED;
    return b200d2::single_particle_tc(*view, d_trans_x, d_trans_y, d_corr, d_real, d_imag, d_eulers, d_diff2s,
                                      (int)O, (int)T, (int)N_img, precision, (cudaStream_t)stream);
  }
  if (precision != B200D2_PREC_FP32) return B200D2_ERR_UNSUPPORTED;
  return b200d2::direct_batch(*view, d_eulers, d_trans_x, d_trans_y, d_real,
                              d_imag, d_corr, 0, d_diff2s, 0, (int)O, (int)T,
                              (int)N_img, 1, false, 0, (cudaStream_t)stream, 0, 1);
}

extern "C" int b200d2_diff2_coarse_f64(const b200d2_view* view,
                                       const float* d_trans_x,
                                       const float* d_trans_y,
                                       const float* d_corr,
                                       const float* d_real,
                                       const float* d_imag,
                                       const float* d_eulers, double* d_diff2s,
                                       size_t O, size_t T, size_t N_img,
                                       int filter_img, void* stream) {
  int st = b200d2::check_common(view, d_trans_x, d_trans_y, d_corr, d_real,
                                d_imag, d_eulers, d_diff2s, O, T, N_img);
  if (st != B200D2_OK) return st;
  return b200d2::direct_batch(*view, d_eulers, d_trans_x, d_trans_y, d_real,
                              d_imag, d_corr, 0, d_diff2s, 0, (int)O, (int)T,
                              (int)N_img, 1, true, filter_img,
                              (cudaStream_t)stream, 0, 1);
}

extern "C" int b200d2_diff2_coarse_cc(const b200d2_view* view, const float* d_trans_x,
                                      const float* d_trans_y, const float* d_corr,
                                      const float* d_real, const float* d_imag,
                                      const float* d_eulers, float* d_diff2s, size_t O,
                                      size_t T, size_t N_img, void* stream, int precision) {
  int st = b200d2::check_common(view, d_trans_x, d_trans_y, d_corr, d_real,
                                d_imag, d_eulers, d_diff2s, O, T, N_img);
  if (st != B200D2_OK) return st;
  if (precision != B200D2_PREC_FP32) return B200D2_ERR_UNSUPPORTED;
  return b200d2::direct_batch(*view, d_eulers, d_trans_x, d_trans_y, d_real,
                              d_imag, d_corr, 0, d_diff2s, 0, (int)O, (int)T,
                              (int)N_img, 1, false, 0, (cudaStream_t)stream, 1, 0);
}

extern "C" int b200d2_diff2_coarse_cc_f64(const b200d2_view* view, const float* d_trans_x,
                                          const float* d_trans_y, const float* d_corr,
                                          const float* d_real, const float* d_imag,
                                          const float* d_eulers, double* d_diff2s, size_t O,
                                          size_t T, size_t N_img, void* stream) {
  int st = b200d2::check_common(view, d_trans_x, d_trans_y, d_corr, d_real,
                                d_imag, d_eulers, d_diff2s, O, T, N_img);
  if (st != B200D2_OK) return st;
  return b200d2::direct_batch(*view, d_eulers, d_trans_x, d_trans_y, d_real,
                              d_imag, d_corr, 0, d_diff2s, 0, (int)O, (int)T,
                              (int)N_img, 1, true, 0, (cudaStream_t)stream, 1, 0);
}
