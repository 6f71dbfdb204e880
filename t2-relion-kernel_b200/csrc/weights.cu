// weights.cu -- coarse-pass weights: per-particle exp(-(diff2 - min)) in FP64,
// their deterministic per-particle sums and normalisation.
//
// Reference: the step after the coarse pass in RELION's E-step, whose driver
// kernel_weights_exponent_coarse is a commented stub in the reference harness
// (src/utilities.h:405-443: per sample pdf_orientation * pdf_offset *
// exp(-(diff2 - min_diff2)) over nr_coarse_orient x nr_coarse_trans samples;
// a zero prior gives a zero weight here).
//
// Layout: diff2[p][o][t] (the coarse output), n = O*T samples per particle.
// Each particle's block is cut into fixed chunks of kChunk samples; a CTA sums
// one chunk in a fixed order and the last CTA of a particle (completion
// counter) adds the chunk sums in chunk order, so sums are bit-reproducible.
// Every kernel streams diff2 once from HBM and takes one FP64 exp per sample.
// Neither a unit nor HBM is full (64 particles x 520704 samples: FP64 pipe 33 %
// active in the sums and 41 % in the writes, issue slots 50 and 70 %, DRAM 14 and
// 35 %): the exp's dependent FP64 chain and the loads are what the warps wait
// for, half of the resident warps at 48 registers.  A sample's
// (o, t) is carried along by 32-bit additions (a thread's samples are
// kWThreads apart) and the normalisation multiplies by the sum's reciprocal
// with one correction step: with 64-bit divisions by T and an FP64 division
// per sample, 64 particles x 520704 samples took 180 us for the sums and 225 us
// for the writes, now 119 and 118 us.
#include <cuda_runtime.h>

#include <algorithm>

#include "common.cuh"

namespace b200d2 {

constexpr int kWThreads = 256;
constexpr int kWUnroll = 4;  // scores loaded together per thread
constexpr long long kChunk = 32768;

int minloc(const float* d, long long n, int P, double* mn, long long* arg, cudaStream_t s);

// The (o, t) of a thread's samples of one chunk: samples threadIdx.x + k
// kWThreads of the chunk, in order, by additions alone.
struct SampleWalk {
  unsigned T, o, t, dq, dr;
  __device__ __forceinline__ SampleWalk(long long lo, int T_) : T((unsigned)T_) {
    // t < T < 2^31 and kWThreads more stay within 32 bits
    const unsigned r = (unsigned)(lo % T_) + threadIdx.x;
    o = (unsigned)(lo / T_) + r / T;
    t = r % T;
    dq = kWThreads / T;
    dr = kWThreads % T;
  }
  __device__ __forceinline__ void next() {
    t += dr;
    o += dq;
    if (t >= T) {
      t -= T;
      ++o;
    }
  }
};

__device__ __forceinline__ double weight_of(float d, const SampleWalk& k, double mn,
                                            const double* __restrict__ pdf_o,
                                            const double* __restrict__ pdf_t) {
  double w = exp(-((double)d - mn));
  if (pdf_o) w *= pdf_o[k.o];
  if (pdf_t) w *= pdf_t[k.t];
  return w;
}

// v / s for one s and many v.  r = 1 / s; q0 = v r is within an ulp or two of
// the quotient, its remainder v - q0 s is exact in one FMA, and q0 + r rem
// rounds to the quotient (P. Markstein, IBM J. Res. Dev. 34 (1990) 111).  The
// steps need the remainder's low bits above the subnormals, so sums or values
// outside [2^-900, 2^900] divide.
struct Quotient {
  double s, r;
  bool fast;
  __device__ __forceinline__ explicit Quotient(double s_) : s(s_), r(1.0 / s_) {
    fast = s_ >= 0x1p-900 && s_ <= 0x1p900;
  }
  __device__ __forceinline__ double operator()(double v) const {
    if (fast && v == 0.0) return v;
    if (!fast || !(v >= 0x1p-900 && v <= 0x1p900)) return v / s;
    const double q0 = __dmul_rn(v, r);
    return __fma_rn(__fma_rn(-q0, s, v), r, q0);
  }
};

// Sum over the CTA in a fixed order (shuffle tree, then warps in order).
__device__ __forceinline__ double block_sum(double v) {
  __shared__ double s_part[kWThreads / 32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) s_part[threadIdx.x >> 5] = v;
  __syncthreads();
  double t = 0.0;
  for (int w = 0; w < kWThreads / 32; ++w) t += s_part[w];
  return t;
}

__global__ void __launch_bounds__(kWThreads) weights_sum_kernel(const float* __restrict__ d2, long long n, int T,
                                                                const double* __restrict__ mn,
                                                                const double* __restrict__ pdf_o,
                                                                const double* __restrict__ pdf_t, double* partial,
                                                                unsigned* count, int nchunk, double* sum) {
  const int p = blockIdx.y, c = blockIdx.x;
  const float* row = d2 + (long long)p * n;
  const double m = mn[p];
  const long long lo = (long long)c * kChunk, hi = min(n, lo + kChunk);
  double acc = 0.0;
  SampleWalk k(lo, T);
  long long i = lo + threadIdx.x;
  for (; i + (kWUnroll - 1) * kWThreads < hi; i += kWUnroll * kWThreads) {
    float d[kWUnroll];
#pragma unroll
    for (int u = 0; u < kWUnroll; ++u) d[u] = row[i + u * kWThreads];
#pragma unroll
    for (int u = 0; u < kWUnroll; ++u) {
      acc += weight_of(d[u], k, m, pdf_o, pdf_t);
      k.next();
    }
  }
  for (; i < hi; i += kWThreads) {
    acc += weight_of(row[i], k, m, pdf_o, pdf_t);
    k.next();
  }
  acc = block_sum(acc);
  __shared__ bool s_last;
  if (threadIdx.x == 0) {
    partial[(long long)p * nchunk + c] = acc;
    __threadfence();
    s_last = atomicAdd(&count[p], 1u) == (unsigned)(nchunk - 1);
  }
  __syncthreads();
  if (s_last && threadIdx.x == 0) {
    __threadfence();
    const volatile double* pp = partial + (long long)p * nchunk;
    double s = 0.0;
    for (int k = 0; k < nchunk; ++k) s += pp[k];
    sum[p] = s;
    count[p] = 0;  // ready for the next call
  }
}

__global__ void __launch_bounds__(kWThreads) weights_write_kernel(const float* __restrict__ d2, long long n, int T,
                                                                  const double* __restrict__ mn,
                                                                  const double* __restrict__ pdf_o,
                                                                  const double* __restrict__ pdf_t,
                                                                  const double* __restrict__ sum, int normalize,
                                                                  double* __restrict__ w) {
  const int p = blockIdx.y;
  const float* row = d2 + (long long)p * n;
  double* out = w + (long long)p * n;
  const double m = mn[p];
  const Quotient div(sum[p]);
  const long long lo = (long long)blockIdx.x * kChunk, hi = min(n, lo + kChunk);
  SampleWalk k(lo, T);
  long long i = lo + threadIdx.x;
  for (; i + (kWUnroll - 1) * kWThreads < hi; i += kWUnroll * kWThreads) {
    float d[kWUnroll];
#pragma unroll
    for (int u = 0; u < kWUnroll; ++u) d[u] = row[i + u * kWThreads];
#pragma unroll
    for (int u = 0; u < kWUnroll; ++u) {
      const double v = weight_of(d[u], k, m, pdf_o, pdf_t);
      k.next();
      out[i + u * kWThreads] = normalize ? div(v) : v;
    }
  }
  for (; i < hi; i += kWThreads) {
    const double v = weight_of(row[i], k, m, pdf_o, pdf_t);
    k.next();
    out[i] = normalize ? div(v) : v;
  }
}

static inline size_t wal(size_t v) { return (v + 255) / 256 * 256; }

static int nchunks(long long n) { return (int)((n + kChunk - 1) / kChunk); }

}  // namespace b200d2

extern "C" size_t b200d2_coarse_weights_workspace(int P, long long n) {
  using namespace b200d2;
  if (P <= 0 || n <= 0) return 0;
  return wal(sizeof(double) * P) + wal(sizeof(double) * (size_t)P * nchunks(n)) + wal(sizeof(unsigned) * P);
}

extern "C" int b200d2_coarse_weights(const float* d_diff2, int P, int O, int T, const double* d_min,
                                     const double* d_pdf_orient, const double* d_pdf_offset, int normalize,
                                     double* d_weights, double* d_sum, void* d_workspace, size_t workspace_bytes,
                                     void* stream) {
  using namespace b200d2;
  if (P < 0 || O < 0 || T < 0) return B200D2_ERR_INVALID;
  const long long n = (long long)O * T;
  if (P == 0 || n == 0) return B200D2_OK;
  if (!d_diff2 || !d_sum || (!d_weights && normalize)) return B200D2_ERR_INVALID;
  if (P > 65535 || nchunks(n) > 0x7fffffff) return B200D2_ERR_UNSUPPORTED;
  const size_t need = b200d2_coarse_weights_workspace(P, n);
  if (!d_workspace || workspace_bytes < need) return B200D2_ERR_INVALID;
  cudaStream_t s = (cudaStream_t)stream;
  uint8_t* ws = static_cast<uint8_t*>(d_workspace);
  double* mn = reinterpret_cast<double*>(ws);
  double* partial = reinterpret_cast<double*>(ws + wal(sizeof(double) * P));
  unsigned* count = reinterpret_cast<unsigned*>(ws + wal(sizeof(double) * P) +
                                                wal(sizeof(double) * (size_t)P * nchunks(n)));
  const double* use_min = d_min;
  if (!d_min) {
    const int st = minloc(d_diff2, n, P, mn, nullptr, s);
    if (st != B200D2_OK) return st;
    use_min = mn;
  } else if ((d_min < d_sum + P && d_sum < d_min + P) ||
             (d_weights && d_min < d_weights + P * n && d_weights < d_min + P) ||
             (reinterpret_cast<const uint8_t*>(d_min) < ws + need && ws < reinterpret_cast<const uint8_t*>(d_min + P))) {
    // the caller's minima share memory with an output or the workspace: keep a copy of them
    B200D2_CUDA_TRY(cudaMemcpyAsync(mn, d_min, sizeof(double) * P, cudaMemcpyDeviceToDevice, s));
    use_min = mn;
  }
  B200D2_CUDA_TRY(cudaMemsetAsync(count, 0, sizeof(unsigned) * P, s));
  const dim3 grid(nchunks(n), P);
  weights_sum_kernel<<<grid, kWThreads, 0, s>>>(d_diff2, n, T, use_min, d_pdf_orient, d_pdf_offset, partial, count,
                                                nchunks(n), d_sum);
  count_launch();
  B200D2_CUDA_TRY(cudaGetLastError());
  if (d_weights) {
    weights_write_kernel<<<grid, kWThreads, 0, s>>>(d_diff2, n, T, use_min, d_pdf_orient, d_pdf_offset, d_sum,
                                                    normalize, d_weights);
    count_launch();
    B200D2_CUDA_TRY(cudaGetLastError());
  }
  return B200D2_OK;
}
