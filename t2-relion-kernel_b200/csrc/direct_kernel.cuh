// direct_kernel.cuh -- the CUDA-core coarse diff2 kernel and its tile choice,
// instantiated for FP32 (diff2_direct.cu) and FP64 (diff2_direct_f64.cu).
//
// Semantics of cuda_kernel_diff2_coarse (src/diff2.cuh:369-537) and its FP64
// twin (src/diff2.cuh:205-365): for every orientation o and translation t
//   diff2s[o*T + t] += sum_{px < N_img} ((A_o - S_t)_re^2 + (A_o - S_t)_im^2) * corr/2
// with A_o the projection (project3Dmodel) and S_t the phase-shifted image
// (translatePixel), the squared differences summed in the working precision.
//
// B200 design (not the reference's loop structure):
//  * a CTA of 512 threads (256 and two CTAs a SM where up to 32 translations
//    leave the fetches the most work) owns an output tile of one particle, 16
//    to 128 translations by 16 to 128 orientations; a cluster of 1, 2, 4 or 8
//    CTAs shares a tile and splits its pixels, so that few tiles still reach
//    every SM.  The cluster's partial sums are added through distributed shared
//    memory in rank order, so each output is written once and the result does
//    not depend on timing;
//  * the pixels an orientation can see (a prefix of every image row) are
//    walked in chunks of KC; the others contribute |S|^2 corr/2 = |X|^2 corr/2
//    to every (o, t), added once per tile;
//  * per chunk the CTA stages the shifted image S[k][t] and the projections
//    A[k][o] in shared memory, neighbouring lanes on neighbouring orientations
//    (in-plane rotations of one pixel: 11.5 ms for 64 particles x 4608
//    orientations on the linear projector, 16.2 with lanes along the pixels).
//    In FP32 both are scaled by sqrt(corr/2), so that a (o, t, pixel) costs one
//    subtraction and one multiply-add for each of the two components: two
//    packed (f32x2) instructions, 2 lane operations each, the real and the
//    imaginary squares in separate sums.  FP64 and negative or infinite
//    weights subtract first and weight the square;
//  * the phase e^{i(x tx + y ty)} is the product of two table entries built
//    once per CTA (FP64 sincos, rounded), where they fit; else a sincos per
//    (pixel, translation) as the reference does;
//  * the next chunk's texture fetches and shifted images are produced while
//    the current one is summed (two buffers, one barrier a chunk); its pixels
//    are copied to shared memory a chunk ahead of that.
// Bound: the FP32 pipe and its operands.  4608 x 113 samples of one particle at
// image 64: 95 us for 4 lane operations per (o, t, pixel) at 128 a clock and SM,
// 107 with the tile's 128 translations; 188 us here (issue slots 55 % busy, the
// shared-memory and texture path 56 %, 16 warps a SM), 449 us with a
// 32-orientation tile per CTA, a sincosf per (pixel, translation, tile) and 5
// operations.
//
// The CC form (cuda_kernel_diff2_CC_coarse, src/diff2.cuh:691-809) runs the
// same tiles with S scaled by corr and A plain: one packed multiply-add per
// (o, t, pixel) for sum corr Re(conj(A) S); the output is -cross / sqrt(norm),
// written (or added with accumulate).  Pixels outside the projector radius have
// A = 0 and are skipped.  sum corr |A|^2 is added up by the threads that stage
// A: in the tile it was repeated by every translation's lanes and its registers
// spilled (64 particles x 4608 x 113: 17.5 ms, now 6.7).
#pragma once

#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <type_traits>

#include "cluster_capacity.h"
#include "common.cuh"

namespace b200d2 {

namespace cg = cooperative_groups;

struct DirectArgs {
  b200d2_view view;
  const float* eulers;
  const float* trans_x;
  const float* trans_y;
  const float* re;
  const float* im;
  const float* corr;
  void* diff2;
  long long img_stride;  // elements between consecutive particles' images
  long long out_stride;  // elements between consecutive particles' outputs
  int O, T, N_img;
  int o_tiles;
  int filter_img;
  int cc;          // 1: cross-correlation score
  int accumulate;  // CC: add onto the output instead of writing it
  int exw;      // phase tables: x extent (0: no tables)
  int off_tab;  // byte offset of the row index and the tables in dynamic shared memory
};

// CTAs of so many threads that share a SM
constexpr int dir_min_ctas(int threads) { return 512 / threads; }

// Pairs (re, im) in the working precision.  FP32 uses packed f32x2
// instructions on 64-bit registers.
struct PairF {
  using V = unsigned long long;
  using E = float;
  static constexpr int KC = 16;
  __device__ static __forceinline__ V make(float x, float y) {
    V v;
    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(x), "f"(y));
    return v;
  }
  __device__ static __forceinline__ V zero() { return 0ull; }
  __device__ static __forceinline__ V add(V a, V b) {
    V d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
  }
  __device__ static __forceinline__ void load2(const V* p, V& a, V& b) {  // p: 16-byte aligned
    const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(p);
    a = v.x;
    b = v.y;
  }
  __device__ static __forceinline__ V mul(V a, V b) {
    V d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
  }
  __device__ static __forceinline__ V fma(V a, V b, V c) {
    V d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
  }
  __device__ static __forceinline__ void parts(V v, float& x, float& y) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(v));
  }
};
struct PairD {
  using V = double2;
  using E = double;
  static constexpr int KC = 8;
  __device__ static __forceinline__ V make(double x, double y) { return make_double2(x, y); }
  __device__ static __forceinline__ V zero() { return make_double2(0.0, 0.0); }
  __device__ static __forceinline__ V add(V a, V b) { return make_double2(a.x + b.x, a.y + b.y); }
  __device__ static __forceinline__ void load2(const V* p, V& a, V& b) {
    a = p[0];
    b = p[1];
  }
  __device__ static __forceinline__ void parts(V v, double& x, double& y) {
    x = v.x;
    y = v.y;
  }
};
__device__ __forceinline__ void copy_async(float* dst, const float* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void copy_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// The sums of one (orientation, translation) over the pixels.
//  FP32: the pair of the real and the imaginary parts' sums.  diff2 scales A and
//    S by sqrt(corr/2) (mac of the difference with itself) or leaves the weight
//    to the sum (weighted); CC's S carries corr (mac).
//  FP64: one sum; diff2 with the weight in it.
template <class PR, bool CC>
struct Acc {
  typename PR::E v;
  __device__ __forceinline__ void clear() { v = 0; }
  __device__ __forceinline__ void mac(typename PR::V a, typename PR::V b) {
    typename PR::E ax, ay, bx, by;
    PR::parts(a, ax, ay);
    PR::parts(b, bx, by);
    v = ::fma(ax, bx, ::fma(ay, by, v));
  }
  __device__ __forceinline__ void weighted(typename PR::V d, typename PR::E w) {
    typename PR::E x, y;
    PR::parts(d, x, y);
    v = ::fma(::fma(x, x, y * y), w, v);
  }
  __device__ __forceinline__ typename PR::E total() const { return v; }
};
template <bool CC>
struct Acc<PairF, CC> {
  PairF::V v;
  __device__ __forceinline__ void clear() { v = PairF::zero(); }
  __device__ __forceinline__ void mac(PairF::V a, PairF::V b) { v = PairF::fma(a, b, v); }
  __device__ __forceinline__ void weighted(PairF::V d, float w) {
    v = PairF::fma(PairF::mul(d, PairF::make(w, w)), d, v);
  }
  __device__ __forceinline__ float total() const {
    float x, y;
    PairF::parts(v, x, y);
    return x + y;
  }
};

// A listed pixel of a chunk, for the shifted images (x and its image row's
// place among the CTA's rows as offsets into the phase tables; the image value,
// times sqrt(corr/2) for FP32 diff2, times corr for CC; negated for diff2:
// A - S is an add) and for the projections (coordinates, their scale, and the
// weight left for the sum).
template <class E>
struct alignas(16) ChunkPixel {
  int xo, yo;
  E xr, xi;
};
template <class E>
struct alignas(16) ChunkSample {
  float fx, fy;
  E sa, wk;
};

// Listed pixels lie in a prefix of every image row: how many of row iy.
__device__ __forceinline__ int row_count(const b200d2_view& v, int iy, int N_img) {
  const int y = iy > v.maxR ? iy - v.imgY : iy;
  const int there = min(v.imgX, max(0, N_img - iy * v.imgX));
  int lo = 0, hi = there;  // first x outside: pixel_maybe_inside falls with x
  while (lo < hi) {
    const int mid = (lo + hi) / 2;
    if (pixel_maybe_inside(mid, y, v.padding_factor, v.maxR2_padded))
      lo = mid + 1;
    else
      hi = mid;
  }
  return lo;
}

// Shared memory of a tile configuration: the two buffers (or the partial
// sums), the row index and, where they fit, the phase tables.
template <class PR, int NT, int L, int TT, int TO>
struct DirCfg {
  static constexpr int BT = L * TT, BO = NT / L * TO;
  // row stride of the projections: the stores of one orientation's pixels, a
  // half-warp's, shift by 16 bytes a row (8 where a thread reads one at a time)
  static constexpr int LA = BO + (TO > 1 && sizeof(typename PR::V) == 8 ? 2 : 1);
  static constexpr size_t kTiles = 2 * PR::KC * (BT + LA) * sizeof(typename PR::V);
  static constexpr size_t kPart = ((size_t)BO * BT + BO + NT) * sizeof(typename PR::E);
  static constexpr size_t kBase = ((kTiles > kPart ? kTiles : kPart) + 15) / 16 * 16;
};
template <class PR, int NT, int L, int TT, int TO, bool CC>
__global__ void __launch_bounds__(NT, dir_min_ctas(NT)) diff2_direct_kernel(const __grid_constant__ DirectArgs a) {
  using E = typename PR::E;
  using V = typename PR::V;
  constexpr int BT = L * TT, BO = NT / L * TO, KC = PR::KC;
  constexpr int LA = DirCfg<PR, NT, L, TT, TO>::LA;
  constexpr int NF = (BO * KC + NT - 1) / NT;  // projections a thread stages per chunk
  extern __shared__ __align__(16) uint8_t dir_smem[];
  // [2][KC][BT] shifted images, [2][KC][LA] projections; after the loop the
  // tile's partial sums [BO][BT] (and the norms [BO])
  V* s_S = reinterpret_cast<V*>(dir_smem);
  V* s_A = s_S + 2 * KC * BT;
  int* s_row = reinterpret_cast<int*>(dir_smem + a.off_tab);  // [imgY + 1] listed pixels before each row
  V* s_ex = reinterpret_cast<V*>(s_row + (a.view.imgY + 4) / 4 * 4);  // [exw][BT] e^{i x tx}
  V* s_ey = s_ex + a.exw * BT;                                        // [rows of this CTA's pixels][BT] e^{i y ty}
  __shared__ float s_eul[BO][6];
  __shared__ float s_tx[BT], s_ty[BT];
  __shared__ ChunkPixel<E> s_px[3][KC];
  __shared__ ChunkSample<E> s_wt[3][KC];
  __shared__ int s_warp[NT / 32];
  __shared__ int s_slow[3];  // FP32 diff2: the chunk's weights stay in the sum
  __shared__ E s_red[NT / 32];

  cg::cluster_group cl = cg::this_cluster();
  const int CS = (int)cl.num_blocks(), rank = (int)cl.block_rank();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const long long p = blockIdx.z;
  const int tile = blockIdx.x / CS;
  const int o0 = (tile % a.o_tiles) * BO;
  const int t0 = (tile / a.o_tiles) * BT;
  const b200d2_view& v = a.view;
  const float* __restrict__ g_re = a.re + p * a.img_stride;
  const float* __restrict__ g_im = a.im + p * a.img_stride;
  const float* __restrict__ g_corr = a.corr + p * a.img_stride;

  constexpr bool kScaled = !CC && std::is_same<E, float>::value;
  __shared__ float s_x2[2][KC];  // kScaled: sum corr/2 |X|^2 of the scaled pixels (even and odd chunks)
  if (kScaled && tid < 2 * KC) s_x2[tid / KC][tid % KC] = 0.f;
  for (int i = tid; i < BO * 6; i += NT) {
    const int o = o0 + i / 6, c = i % 6;
    const int src = (c >> 1) * 3 + (c & 1);  // e0 e1 e3 e4 e6 e7
    s_eul[i / 6][c] = o < a.O ? a.eulers[(size_t)o * 9 + src] : 0.f;
  }
  for (int i = tid; i < BT; i += NT) {
    const int t = t0 + i;
    s_tx[i] = t < a.T ? a.trans_x[t] : 0.f;
    s_ty[i] = t < a.T ? a.trans_y[t] : 0.f;
  }
  // listed pixels before each image row
  int run = 0;
  for (int base = 0; base < v.imgY; base += NT) {
    const int iy = base + tid;
    const int c = iy < v.imgY ? row_count(v, iy, a.N_img) : 0;
    int inc = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int n = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += n;
    }
    __syncthreads();
    if (lane == 31) s_warp[warp] = inc;
    __syncthreads();
    int off = run, total = 0;
    for (int w = 0; w < NT / 32; ++w) {
      off += w < warp ? s_warp[w] : 0;
      total += s_warp[w];
    }
    if (iy < v.imgY) s_row[iy] = off + inc - c;
    run += total;
  }
  if (tid == 0) s_row[v.imgY] = run;
  __syncthreads();
  const int K = run;
  const int kb = (int)((long long)K * rank / CS), ke = (int)((long long)K * (rank + 1) / CS);
  auto row_of = [&](int k) {  // image row of listed pixel k < K
    int lo = 0, hi = v.imgY;
    while (hi - lo > 1) {
      const int mid = (lo + hi) / 2;
      if (s_row[mid] <= k)
        lo = mid;
      else
        hi = mid;
    }
    return lo;
  };
  auto filtered = [&](int x, int y) {  // reference filter test (src/diff2.cuh:339-345), in double
    return a.filter_img &&
           (double)(x * x + y * y) * v.padding_factor * v.padding_factor > (double)v.maxR2_padded;
  };
  // pixels no orientation sees, this CTA's share of the image
  E out_part = E(0);
  if (!CC) {
    const int i0 = (int)((long long)a.N_img * rank / CS), i1 = (int)((long long)a.N_img * (rank + 1) / CS);
    for (int i = i0 + tid; i < i1; i += NT) {
      int x, y;
      pixel_coor(i, v.imgX, v.imgY, v.maxR, x, y);
      if (pixel_maybe_inside(x, y, v.padding_factor, v.maxR2_padded)) continue;
      const bool z = filtered(x, y);
      const E re = z ? E(0) : (E)g_re[i], im = z ? E(0) : (E)g_im[i];
      out_part += (re * re + im * im) * (E)(g_corr[i] / 2);
    }
  }
  const int row0 = kb < ke ? row_of(kb) : 0, nrows = kb < ke ? row_of(ke - 1) - row0 + 1 : 0;
  if (a.exw > 0) {
    // Runs of kRun entries of one translation: FP32 takes two sincos a run and
    // multiplies on in FP64 (a few 2^-53 off before the rounding to FP32), FP64
    // one sincos an entry.
    constexpr int kRun = std::is_same<E, float>::value ? 8 : 1;
    const int gx = (a.exw + kRun - 1) / kRun, gy = (nrows + kRun - 1) / kRun;
    for (int e = tid; e < (gx + gy) * BT; e += NT) {
      const int j = e / BT, t = e % BT;
      const bool isx = j < gx;
      const int i0 = (isx ? j : j - gx) * kRun, n = isx ? a.exw : nrows;
      const double slope = isx ? (double)s_tx[t] : (double)s_ty[t];
      V* dst = (isx ? s_ex : s_ey) + t;
      double sn = 0.0, cs = 1.0, s1, c1;
      if (kRun > 1) sincos(slope, &s1, &c1);
      int last = 0x7fffffff;
#pragma unroll
      for (int r = 0; r < kRun; ++r) {
        const int i = i0 + r;
        if (i >= n) break;
        // the image rows' coordinates count up by one, but for the wrap to
        // negative ones after row maxR
        const int at = isx ? i : row0 + i > v.maxR ? row0 + i - v.imgY : row0 + i;
        if (r == 0 || at != last + 1) {
          sincos((double)at * slope, &sn, &cs);
        } else {
          const double c2 = cs * c1 - sn * s1;
          sn = cs * s1 + sn * c1;
          cs = c2;
        }
        last = at;
        dst[i * BT] = PR::make((E)cs, (E)sn);
      }
    }
  }

  // a thread's sums: translations t_of(i) and orientations oq TO + j
  const int tq = lane % L, oq = tid / L;
  auto t_of = [&](int i) { return i < (TT & ~1) ? L * (i & ~1) + 2 * tq + (i & 1) : L * (TT - 1) + tq; };
  Acc<PR, CC> acc[TT][TO];

  const int nchunk = (ke - kb + KC - 1) / KC;
  // FP32 diff2 scales A and S by sqrt(corr/2) before it subtracts them; `plain`
  // takes the differences first and leaves the weights to the sums
  bool plain = false;
  // Pixels of a chunk into slot c % 3, by the first lanes of warp c % (NT / 32):
  // their places and loads first (into shared memory: registers are short here),
  // the values a chunk later, when they have landed.
  struct RawPixel {
    int x, row;
    float re, im, corr;
  };
  __shared__ RawPixel s_raw[4][KC];
  auto begin_pixels = [&](int c) {
    if (warp != c % (NT / 32) || lane >= KC) return;
    const int k = kb + c * KC + lane;
    if (k < ke) {
      RawPixel& r = s_raw[c & 3][lane];
      const int iy = row_of(k), x = k - s_row[iy], i = iy * v.imgX + x;
      r.x = x;
      r.row = iy;
      copy_async(&r.re, g_re + i);
      copy_async(&r.im, g_im + i);
      copy_async(&r.corr, g_corr + i);
    }
  };
  auto end_pixels = [&](int c) {
    if (warp != c % (NT / 32)) return;
    bool slow = false;
    if (lane < KC) {
      ChunkPixel<E> q;
      ChunkSample<E> g;
      q.xo = q.yo = 0;
      g.fx = g.fy = 0.f;
      q.xr = q.xi = g.sa = g.wk = E(0);  // past the end: the origin, without weight
      if (kb + c * KC + lane < ke) {
        copy_async_wait();
        const RawPixel& r = s_raw[c & 3][lane];
        const int x = r.x, y = r.row > v.maxR ? r.row - v.imgY : r.row;
        const bool zero = filtered(x, y);
        const E re = zero ? E(0) : (E)r.re, im = zero ? E(0) : (E)r.im;
        const float cf = r.corr;
        q.xo = x * BT;
        q.yo = (r.row - row0) * BT;
        g.fx = (float)x;
        g.fy = (float)y;
        g.sa = E(1);
        if (CC) {
          g.wk = (E)cf;
          q.xr = g.wk * re;
          q.xi = g.wk * im;
        } else if (kScaled && !plain && cf >= 0.f && cf < __int_as_float(0x7f800000)) {
          g.sa = sqrt((E)(cf / 2));
          g.wk = E(1);
          q.xr = -g.sa * re;
          q.xi = -g.sa * im;
          s_x2[c & 1][lane] += (float)(q.xr * q.xr + q.xi * q.xi);
        } else {
          g.wk = (E)(cf / 2);
          q.xr = -re;
          q.xi = -im;
          slow = true;
        }
      }
      s_px[c % 3][lane] = q;
      s_wt[c % 3][lane] = g;
    }
    if (kScaled) {
      slow = __any_sync(0xffffffffu, slow);
      if (lane == 0) s_slow[c % 3] = slow;
    }
  };
  // shifted images of chunk c
  auto shifted = [&](int c, int k, int t) {
    const ChunkPixel<E> q = s_px[c % 3][k];
    E cs, sn;
    if (a.exw > 0) {
      const V fx = s_ex[q.xo + t], fy = s_ey[q.yo + t];
      const E* x = reinterpret_cast<const E*>(&fx);
      const E* y = reinterpret_cast<const E*>(&fy);
      cs = x[0] * y[0] - x[1] * y[1];
      sn = x[0] * y[1] + x[1] * y[0];
    } else {
      const ChunkSample<E> g = s_wt[c % 3][k];
      if constexpr (std::is_same<E, float>::value)
        sincosf(__fmaf_rn(g.fx, s_tx[t], __fmul_rn(g.fy, s_ty[t])), &sn, &cs);
      else
        sincos((double)g.fx * (double)s_tx[t] + (double)g.fy * (double)s_ty[t], &sn, &cs);
    }
    return PR::make(cs * q.xr - sn * q.xi, cs * q.xi + sn * q.xr);
  };
  auto stage_S = [&](int c) {
    V* d = s_S + (c & 1) * KC * BT;
    if constexpr (NT % BT == 0 && KC % (NT / BT) == 0) {  // a thread keeps its translation
      const int t = tid % BT;
#pragma unroll
      for (int i = 0; i < KC / (NT / BT); ++i) {
        const int k = tid / BT + i * (NT / BT);
        d[k * BT + t] = shifted(c, k, t);
      }
    } else {
      for (int e = tid; e < KC * BT; e += NT) d[e] = shifted(c, e / BT, e % BT);
    }
  };
  PixelFetch<NF> f;
  E nrm[NF];  // CC: this thread's share of sum corr |A|^2 of the orientations it stages
#pragma unroll
  for (int u = 0; u < NF; ++u) nrm[u] = E(0);
  // sample u of a thread: pixel a_k(u), orientation a_o(u) of the chunk's tile
  auto a_k = [&](int u) { return (tid + u * NT) / BO; };
  auto a_o = [&](int u) { return (tid + u * NT) % BO; };
  auto fetch_A = [&](int c) {
    float fx[NF], fy[NF];
    const float* e[NF];
#pragma unroll
    for (int u = 0; u < NF; ++u) {
      const int k = min(a_k(u), KC - 1);
      fx[u] = s_wt[c % 3][k].fx;
      fy[u] = s_wt[c % 3][k].fy;
      e[u] = s_eul[min(a_o(u), BO - 1)];
    }
    f.issue(v, fx, fy, e);
  };
  auto store_A = [&](int c) {
    V* d = s_A + (c & 1) * KC * LA;
#pragma unroll
    for (int u = 0; u < NF; ++u) {
      const int k = a_k(u), o = a_o(u);
      if (BO * KC % NT != 0 && (o >= BO || k >= KC)) continue;
      const float2 b = f.finish(u);
      E x = (E)b.x, y = (E)b.y;
      if (CC) nrm[u] = fma(fma(x, x, y * y), s_wt[c % 3][k].wk, nrm[u]);
      if (kScaled) {
        x *= s_wt[c % 3][k].sa;
        y *= s_wt[c % 3][k].sa;
      }
      d[k * LA + o] = PR::make(x, y);
    }
  };
  auto sums = [&](int c, auto weighted) {
    constexpr bool W = decltype(weighted)::value;
    const V* S = s_S + (c & 1) * KC * BT;
    const V* A = s_A + (c & 1) * KC * LA;
#pragma unroll (W && kScaled ? 1 : KC)
    for (int k = 0; k < KC; ++k) {
      V sv[TT], av[TO];
#pragma unroll
      for (int i = 0; i + 1 < TT; i += 2) PR::load2(S + k * BT + L * i + 2 * tq, sv[i], sv[i + 1]);
      if (TT & 1) sv[TT - 1] = S[k * BT + L * (TT - 1) + tq];
      if constexpr (TO == 1) {
        av[0] = A[k * LA + oq];
      } else {
#pragma unroll
        for (int j = 0; j < TO; j += 2) PR::load2(A + k * LA + oq * TO + j, av[j], av[j + 1]);
      }
      [[maybe_unused]] const E w = W ? s_wt[c % 3][k].wk : E(0);
#pragma unroll
      for (int i = 0; i < TT; ++i)
#pragma unroll
        for (int j = 0; j < TO; ++j) {
          if constexpr (CC) {
            acc[i][j].mac(av[j], sv[i]);
          } else {
            const V d = PR::add(av[j], sv[i]);
            if constexpr (W)
              acc[i][j].weighted(d, w);
            else
              acc[i][j].mac(d, d);
          }
        }
    }
  };
  auto walk = [&]() {  // the sums over this CTA's pixels
#pragma unroll
    for (int i = 0; i < TT; ++i)
#pragma unroll
      for (int j = 0; j < TO; ++j) acc[i][j].clear();
    for (int c = 0; c < 3; ++c) begin_pixels(c);
    for (int c = 0; c < 2; ++c) end_pixels(c);
    __syncthreads();  // the tables and the first two chunks' pixels
    if (nchunk > 0) {
      fetch_A(0);
      stage_S(0);
      store_A(0);
    }
    for (int c = 0; c < nchunk; ++c) {
      __syncthreads();  // chunk c's tiles and chunk c + 1's pixels are there; chunk c - 1's tiles are free
      auto stage = [&]() {  // chunk c + 1's tiles and chunk c + 2's pixels
        begin_pixels(c + 3);
        if (c + 1 < nchunk) {
          fetch_A(c + 1);
          stage_S(c + 1);
        }
        end_pixels(c + 2);
        if (c + 1 < nchunk) store_A(c + 1);
      };
      // two warps of each sub-partition stage first and two sum first, so that
      // the staging's loads and integer work run beside the FP32 pipe's sums
      const int turn = (warp >> 2) & 1;
#pragma unroll 1
      for (int h = 0; h < 2; ++h) {
        if (h == turn)
          stage();
        else if (!CC && (!kScaled || s_slow[c % 3]))
          sums(c, std::true_type());
        else if (CC || kScaled)
          sums(c, std::false_type());
      }
    }
  };
  if constexpr (kScaled) {
    // Scaled operands are rounded before they are subtracted: a relative error
    // of up to 2^-22 sqrt(sum corr/2 |X|^2 / score) in a score (over this CTA's
    // pixels).  Where one is below kNear of that power the tile is summed
    // again, differences first, as the error could pass 4e-6; noisy images are
    // not (ratios around 1), a projection of the volume itself is.
    constexpr float kNear = 1.f / 256.f;
    static_assert(2 * KC == 32, "one warp's worth of partial sums");
#pragma unroll 1
    for (int pass = 0; pass < 2; ++pass) {
      plain = pass > 0;
      walk();
      __syncthreads();  // s_x2
      float near = (&s_x2[0][0])[lane];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) near += __shfl_xor_sync(0xffffffffu, near, o);
      near *= kNear;
      bool below = false;
#pragma unroll
      for (int i = 0; i < TT; ++i)
#pragma unroll
        for (int j = 0; j < TO; ++j)
          below |= acc[i][j].total() < near && o0 + oq * TO + j < a.O && t0 + t_of(i) < a.T;
      if (!__syncthreads_or(below && pass == 0)) break;
    }
  } else {
    walk();
  }

  // the out-of-radius constant of this CTA
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) out_part += __shfl_xor_sync(0xffffffffu, out_part, o);
  if (lane == 0) s_red[warp] = out_part;
  __syncthreads();  // (and the tiles are free)
  E out_total = E(0);
#pragma unroll
  for (int w = 0; w < NT / 32; ++w) out_total += s_red[w];

  E* __restrict__ g_out = reinterpret_cast<E*>(a.diff2) + p * a.out_stride;
  auto put = [&](int o, int t, E sum, E norm) {
    if (o >= a.O || t >= a.T) return;
    E* dst = g_out + (size_t)o * a.T + t;
    if (CC) {
      const E c = -(sum / sqrt(norm));
      *dst = a.accumulate ? *dst + c : c;
    } else {
      *dst = *dst + sum;
    }
  };
  // partial sums [BO][BT] (clusters) and norms (CC) into this CTA's shared
  // memory; each rank then adds its share of the tile over the cluster, in rank
  // order
  E* part = reinterpret_cast<E*>(dir_smem);
  E* pnrm = part + BO * BT;
  if (CC) {
    // an orientation's pixels were staged by threads BO apart
    E* pn = pnrm + BO;  // [max(1, NT / BO)][BO]
    constexpr int G = NT / BO > 1 ? (NT / BO < KC ? NT / BO : KC) : 1;
    E n = nrm[0];
#pragma unroll
    for (int u = 1; u < NF; ++u) n += nrm[u];
    if (tid < G * BO) pn[tid] = n;
    __syncthreads();
    if (tid < BO) {
      E n = E(0);
      for (int g = 0; g < G; ++g) n += pn[g * BO + tid];
      pnrm[tid] = n;
    }
  }
  if (CS == 1) {
    if (CC) __syncthreads();
#pragma unroll
    for (int j = 0; j < TO; ++j)
#pragma unroll
      for (int i = 0; i < TT; ++i)
        put(o0 + oq * TO + j, t0 + t_of(i), CC ? acc[i][j].total() : acc[i][j].total() + out_total, CC ? pnrm[oq * TO + j] : E(0));
    return;
  }
#pragma unroll
  for (int j = 0; j < TO; ++j)
#pragma unroll
    for (int i = 0; i < TT; ++i)
      part[(oq * TO + j) * BT + t_of(i)] = CC ? acc[i][j].total() : acc[i][j].total() + out_total;
  cl.sync();
  const int e0 = (int)((long long)BO * BT * rank / CS), e1 = (int)((long long)BO * BT * (rank + 1) / CS);
  for (int e = e0 + tid; e < e1; e += NT) {
    double sum = 0.0, norm = 0.0;
    for (int r = 0; r < CS; ++r) {
      sum += (double)cl.map_shared_rank(part, r)[e];
      if (CC) norm += (double)cl.map_shared_rank(pnrm, r)[e / BT];
    }
    put(o0 + e / BT, t0 + e % BT, (E)sum, (E)norm);
  }
  cl.sync();  // no CTA leaves while another reads its sums
}

constexpr size_t kDirSmem = 212 * 1024;  // dynamic shared memory of a CTA, at most

// Fills the fields that depend on the tile and the shared-memory size; false
// when the tile does not fit beside the row index of a very tall image.
template <class PR, int NT, int L, int TT, int TO>
static bool dir_smem_layout(DirectArgs& a, size_t& bytes) {
  using C = DirCfg<PR, NT, L, TT, TO>;
  a.o_tiles = (a.O + C::BO - 1) / C::BO;
  a.off_tab = (int)C::kBase;
  bytes = C::kBase + ((size_t)a.view.imgY + 4) / 4 * 16;
  if (bytes > kDirSmem) return false;
  // a listed pixel has x <= sqrt((maxR2_padded + 2) / pf^2)
  const double r = std::sqrt((double)a.view.maxR2_padded + 2.0) / (double)a.view.padding_factor;
  const long long exw = std::min<long long>(a.view.imgX, (long long)std::min(r, 1e6) + 2);
  const size_t tab = (size_t)(exw + a.view.imgY) * C::BT * sizeof(typename PR::V);
  a.exw = 0;
  if (bytes + tab <= kDirSmem) {
    a.exw = (int)exw;
    bytes += tab;
  }
  return true;
}

template <class PR, int NT, int L, int TT, int TO, bool CC>
static cudaLaunchConfig_t dir_config(cudaLaunchAttribute* at, size_t bytes, int cs) {
  cudaLaunchConfig_t cfg = {};
  cfg.blockDim = dim3(NT);
  cfg.dynamicSmemBytes = bytes;
  at->id = cudaLaunchAttributeClusterDimension;
  at->val.clusterDim.x = (unsigned)cs;
  at->val.clusterDim.y = at->val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cfg;
}

// Clusters of cs CTAs that run at once on the current device (512 threads: 1 CTA
// per SM; 256: 2 while their shared memory fits twice).
template <class PR, int NT, int L, int TT, int TO, bool CC>
static int dir_capacity(size_t bytes, int cs) {
  static ClusterCapacity known[2];
  int dev = -1;
  cudaGetDevice(&dev);
  return known[bytes > kDirSmem / 2].get(dev, cs, [&]() {
    cudaLaunchAttribute at;
    cudaLaunchConfig_t cfg = dir_config<PR, NT, L, TT, TO, CC>(&at, bytes, cs);
    cfg.gridDim = dim3((unsigned)cs);
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, diff2_direct_kernel<PR, NT, L, TT, TO, CC>, &cfg) != cudaSuccess) {
      cudaGetLastError();
      return 0;
    }
    return n;
  });
}

static inline int dir_sms() {
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return sms;
}

// A tile width and cluster size with its estimated time in lane operations
// per SM.
struct DirChoice {
  double cost = 1e300;
  int to = 0, cs = 0;
};

// Estimates every cluster size for one tile width.  Per CTA: its share of the
// listed pixels at (ops per (o, t, pixel)) lane operations a sample, the
// staging of a pixel (about 18 a translation and 60 an orientation), the phase
// tables (FP64 sincos) and a fixed part of about 5 us; times the waves of
// clusters.  One particle at C2 takes 64-orientation tiles on pairs (72 tiles,
// one wave); 128-wide tiles on clusters of 4 would need 36 clusters at once.
template <class PR, int NT, int L, int TT, int TO, bool CC>
static void dir_consider(const DirectArgs& a0, int P, int K, DirChoice& best) {
  using C = DirCfg<PR, NT, L, TT, TO>;
  constexpr bool D = std::is_same<PR, PairD>::value;
  DirectArgs a = a0;
  size_t bytes = 0;
  if (!dir_smem_layout<PR, NT, L, TT, TO>(a, bytes)) return;
  static std::atomic<unsigned long long> opted{0};
  if (smem_opt_in(diff2_direct_kernel<PR, NT, L, TT, TO, CC>, (int)kDirSmem, opted) != cudaSuccess) {
    cudaGetLastError();
    return;
  }
  const int sms = dir_sms();
  const double tiles = (double)P * a.o_tiles * ((a.T + C::BT - 1) / C::BT);
  // lane operations a sample, or what its shared-memory reads take
  const double lds = 128.0 * (D ? 2.0 : 1.0) * (2.0 * TT + TO) / (32.0 * TT * TO);
  const double ops = std::max((CC ? 2.0 : 4.0) * (D ? 2 : 1), lds);
  for (int l = 0; l < 4; ++l) {
    const int cs = 1 << l;
    const double waves = std::ceil(tiles / dir_capacity<PR, NT, L, TT, TO, CC>(bytes, cs));
    const double loads = std::max(waves, std::ceil(tiles * cs / sms));  // CTAs that the fullest SM works through
    const double share = std::ceil((double)K / cs);
    const double stage = (a.exw ? 18.0 * (D ? 2 : 1) : D ? 300.0 : 60.0) * C::BT + 60.0 * C::BO;
    const double tab = a.exw ? 140.0 * (a.exw + (double)a.view.imgY / cs) * C::BT : 0.0;
    const double cost = loads * (share * (ops * C::BT * C::BO + stage) + tab) + waves * (1.2e6 + (cs > 1 ? 2e5 : 0.0));
    if (cost < best.cost) best = DirChoice{cost, TO, cs};
  }
}

template <class PR, int NT, int L, int TT, int TO, bool CC>
static int dir_launch(const DirectArgs& a0, int P, int cs, cudaStream_t s) {
  using C = DirCfg<PR, NT, L, TT, TO>;
  DirectArgs a = a0;
  size_t bytes = 0;
  if (!dir_smem_layout<PR, NT, L, TT, TO>(a, bytes)) return B200D2_ERR_UNSUPPORTED;
  const long long nx = (long long)a.o_tiles * ((a.T + C::BT - 1) / C::BT) * cs;
  if (nx > 0x7fffffffLL || P > 65535) return B200D2_ERR_UNSUPPORTED;
  cudaLaunchAttribute at;
  cudaLaunchConfig_t cfg = dir_config<PR, NT, L, TT, TO, CC>(&at, bytes, cs);
  cfg.gridDim = dim3((unsigned)nx, 1, (unsigned)P);
  cfg.stream = s;
  B200D2_CUDA_TRY(cudaLaunchKernelEx(&cfg, diff2_direct_kernel<PR, NT, L, TT, TO, CC>, a));
  count_launch();
  return status_from_cuda(cudaGetLastError());
}

// One tile height in three widths (128, 64 and 32 orientations).  A thread's
// TT x TO tile reads TT + TO pairs of shared memory per pixel: TT cost 2 clocks
// of the SM's shared-memory return path each, TO (the same address for a warp
// or half-warp) one, against TT TO of the FP32 pipe.  So heights that are
// multiples of 32 put 32 lanes along the translations and more orientations in
// a thread (4 x 4 needs 12 clocks for 16, where 8 x 2 on 16 lanes needs 18: at
// C2 one particle took 255 us with that).
template <class PR, int NT, int L, int TT, bool CC>
static int dir_launch_tt(const DirectArgs& a, int P, int K, cudaStream_t s) {
  constexpr int W = L / 16;
  DirChoice c;
  dir_consider<PR, NT, L, TT, 4 * W, CC>(a, P, K, c);
  dir_consider<PR, NT, L, TT, 2 * W, CC>(a, P, K, c);
  dir_consider<PR, NT, L, TT, W, CC>(a, P, K, c);
  switch (c.to) {
    case 4 * W: return dir_launch<PR, NT, L, TT, 4 * W, CC>(a, P, c.cs, s);
    case 2 * W: return dir_launch<PR, NT, L, TT, 2 * W, CC>(a, P, c.cs, s);
    case W: return dir_launch<PR, NT, L, TT, W, CC>(a, P, c.cs, s);
    default: return B200D2_ERR_UNSUPPORTED;
  }
}

// Loads the tile's kernels (instead of at their first launch, which can wait
// for running work).
template <class PR, int NT, int L, int TT, bool CC>
static cudaError_t dir_preload_tt() {
  constexpr int W = L / 16;
  cudaFuncAttributes a;
  cudaError_t e = cudaFuncGetAttributes(&a, (const void*)diff2_direct_kernel<PR, NT, L, TT, 4 * W, CC>);
  if (e == cudaSuccess) e = cudaFuncGetAttributes(&a, (const void*)diff2_direct_kernel<PR, NT, L, TT, 2 * W, CC>);
  if (e == cudaSuccess) e = cudaFuncGetAttributes(&a, (const void*)diff2_direct_kernel<PR, NT, L, TT, W, CC>);
  return e;
}

// Listed pixels of the image (an estimate for the tile choice).
static int dir_listed(const b200d2_view& v, int N_img) {
  const double r2 = ((double)v.maxR2_padded + 2.0) / ((double)v.padding_factor * v.padding_factor);
  double n = 0.0;
  for (int iy = 0; iy < v.imgY && (long long)iy * v.imgX < N_img; ++iy) {
    const double y = iy > v.maxR ? iy - v.imgY : iy;
    if (y * y < r2) n += std::min((double)v.imgX, std::sqrt(r2 - y * y) + 1.0);
  }
  return (int)std::min(n, (double)N_img);
}

// Rows of 16 translations per tile: the fewest tiles of up to 128
// translations, as even as the instantiated heights allow.
static inline int dir_rows(int T) {
  const int tiles = (T + 127) / 128;
  return ((T + tiles - 1) / tiles + 15) / 16;
}

}  // namespace b200d2
