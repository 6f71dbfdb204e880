// fine.cu -- fine-pass diff2 over a job list (b200d2_diff2_fine).
//
// Replaces cuda_kernel_diff2_fine (src/diff2.cuh:540-682, 2D image against a
// 3D reference).  After the coarse pass, RELION rescores only the significant
// samples on oversampled orientation and translation grids.  The work arrives
// as jobs: job j scores orientation rot_idx[job_idx[j]] against the job_num[j]
// consecutive translations starting at trans_idx[job_idx[j]], and writes
//   diff2s[job_idx[j] + i] = sum_init + sum_px corr/2 |proj - shift_i(img)|^2
// for i < job_num[j] (written, not accumulated, as the reference does).
//
// One CTA per job.  Each thread projects its pixels once (texture or linear
// projector, the same sample positions as the coarse kernels) and keeps the
// job's translations in registers (up to kFineMaxTrans per pass; longer jobs
// take several passes over the pixels), so the projection is shared by all of
// the job's translations; the per-translation sums are reduced with warp
// shuffles and one shared-memory step in a fixed order.  The phase shift
// e^{i(x tx + y ty)} is the product of two table entries e^{i x tx} and
// e^{i y ty}, built per pass in shared memory (one sincos per table entry,
// not per pixel).  With the tables the score is taken expanded,
//   sum w|A - S|^2 = sum w(|A|^2 + |X|^2) - 2 sum Re(q e^{i x tx} e^{i y ty}),
//   q = w conj(A) X,
// so a (pixel, translation) pair costs one complex multiply and a real part
// (the norms are per pixel, in FP64); the per-thread cross sums are combined
// in FP64 and the final difference is taken in FP64.  Jobs on images too
// large for the tables take sincosf per pixel and sum w|A - S|^2 directly, as
// the reference does.  Pixel coordinates
// follow the fine kernel's mapping (src/diff2.cuh:612-626): rows past maxR
// wrap to negative y when they lie within maxR of the end, otherwise their x
// is set to maxR (outside the projector radius).
//
// The same kernel with CC = true replaces cuda_kernel_diff2_CC_fine
// (src/diff2.cuh:811-960): per (job, translation) it writes
//   diff2s[job_idx[j] + i] = -sum_px corr Re(conj(proj) shift_i(img)) / sqrt(sum_px corr |proj|^2)
// (full corr, no sum_init, written).  The cross sums are taken as above with
// q = corr conj(A) X; the norm is summed in FP64 and the quotient taken in
// FP64.
#include <cuda_runtime.h>

#include <algorithm>

#include "common.cuh"

namespace b200d2 {

constexpr int kFineThreads = 128;
constexpr int kFineMaxTrans = 16;
constexpr size_t kFineTableBytes = 96 * 1024;  // largest phase-table area per CTA

__device__ __forceinline__ void fine_pixel_coor(int pixel, int imgX, int imgY, int maxR, int& x, int& y) {
  x = pixel % imgX;
  y = pixel / imgX;
  if (y > maxR) {
    if (y >= imgY - maxR)
      y -= imgY;
    else
      x = maxR;
  }
}

template <int NT, bool TABLES, bool CC>
__global__ void __launch_bounds__(kFineThreads) diff2_fine_kernel(
    b200d2_view v, const float* __restrict__ eulers, const float* __restrict__ re, const float* __restrict__ im,
    const float* __restrict__ tx, const float* __restrict__ ty, const float* __restrict__ corr,
    float* __restrict__ diff2s, int image_size, float sum_init, const uint64_t* __restrict__ rot_idx,
    const uint64_t* __restrict__ trans_idx, const uint64_t* __restrict__ job_idx,
    const uint64_t* __restrict__ job_num) {
  const uint64_t jb = job_idx[blockIdx.x];
  const int ntrans = (int)job_num[blockIdx.x];
  const uint64_t o = rot_idx[jb];
  const uint64_t t0 = trans_idx[jb];
  const float* eo = eulers + o * 9;
  float e[6] = {eo[0], eo[1], eo[3], eo[4], eo[6], eo[7]};
  __shared__ float s_part[kFineThreads / 32][NT];
  __shared__ double s_cross[kFineThreads / 32][NT], s_norm[kFineThreads / 32];
  // TABLES: [NT][exw] e^{i x tx} for x in [0, exw), then [NT][eyw] e^{i y ty}
  // for y in [-maxR, imgY); fine_pixel_coor yields x < max(imgX, maxR + 1)
  // and -maxR <= y < imgY.
  extern __shared__ float2 s_tab[];
  const int exw = max(v.imgX, v.maxR + 1), eyw = v.imgY + v.maxR;
  float2* s_ex = s_tab;
  float2* s_ey = s_tab + NT * exw;
  for (int base = 0; base < ntrans; base += NT) {  // passes of NT translations
    const int nt = min(NT, ntrans - base);
    float ftx[NT], fty[NT], acc[NT];
#pragma unroll
    for (int i = 0; i < NT; ++i) {
      ftx[i] = i < nt ? tx[t0 + base + i] : 0.f;
      fty[i] = i < nt ? ty[t0 + base + i] : 0.f;
      acc[i] = 0.f;
    }
    if (TABLES) {
      for (int e2 = threadIdx.x; e2 < NT * (exw + eyw); e2 += kFineThreads) {
        float sn = 0.f, cs = 1.f;
        if (e2 < NT * exw) {
          const int i = e2 / exw, x = e2 - i * exw;
          if (i < nt) sincosf(__fmul_rn((float)x, tx[t0 + base + i]), &sn, &cs);
          s_ex[e2] = make_float2(cs, sn);
        } else {
          const int j = e2 - NT * exw, i = j / eyw, y = j - i * eyw - v.maxR;
          if (i < nt) sincosf(__fmul_rn((float)y, ty[t0 + base + i]), &sn, &cs);
          s_ey[j] = make_float2(cs, sn);
        }
      }
      __syncthreads();
    }
    double nrm = 0.0;  // this thread's sum w(|A|^2 + |X|^2) (tables) or sum corr |A|^2 (CC)
    for (int pixel = threadIdx.x; pixel < image_size; pixel += kFineThreads) {
      int x, y;
      fine_pixel_coor(pixel, v.imgX, v.imgY, v.maxR, x, y);
      const float2 a = project_pixel(v, (float)x, (float)y, e);
      const float xr = re[pixel], xi = im[pixel];
      const float w = CC ? corr[pixel] : 0.5f * corr[pixel];
      if (CC) {  // the CC denominator: sum corr |A|^2
        const double ad = a.x, bd = a.y;
        nrm = fma((double)w, fma(ad, ad, bd * bd), nrm);
      }
      if (TABLES) {
        const double ad = a.x, bd = a.y, xd = xr, yd = xi;
        if (!CC) nrm = fma((double)w, fma(ad, ad, fma(bd, bd, fma(xd, xd, yd * yd))), nrm);
        const float qr = __fmul_rn(w, __fmaf_rn(a.x, xr, __fmul_rn(a.y, xi)));   // w Re(conj(A) X)
        const float qi = __fmul_rn(w, __fmaf_rn(a.x, xi, -__fmul_rn(a.y, xr)));  // w Im(conj(A) X)
        const float2* pex = s_ex + x;
        const float2* pey = s_ey + y + v.maxR;
#pragma unroll
        for (int i = 0; i < NT; ++i) {
          if (i < nt) {
            const float2 ex = pex[i * exw], ey = pey[i * eyw];
            const float ur = __fmaf_rn(qr, ex.x, -__fmul_rn(qi, ex.y));
            const float ui = __fmaf_rn(qr, ex.y, __fmul_rn(qi, ex.x));
            acc[i] = __fmaf_rn(ur, ey.x, __fmaf_rn(-ui, ey.y, acc[i]));
          }
        }
      } else {
#pragma unroll
        for (int i = 0; i < NT; ++i) {
          if (i < nt) {
            float s, c;
            sincosf(__fmaf_rn((float)x, ftx[i], __fmul_rn((float)y, fty[i])), &s, &c);
            if (CC) {  // corr Re(conj(A) S), S = X e^{i(x tx + y ty)}
              const float sr = __fmaf_rn(c, xr, -__fmul_rn(s, xi));
              const float si = __fmaf_rn(c, xi, __fmul_rn(s, xr));
              acc[i] = __fmaf_rn(__fmaf_rn(a.x, sr, __fmul_rn(a.y, si)), w, acc[i]);
              continue;
            }
            const float dr = a.x - __fmaf_rn(c, xr, -__fmul_rn(s, xi));
            const float di = a.y - __fmaf_rn(c, xi, __fmul_rn(s, xr));
            acc[i] = __fmaf_rn(__fmaf_rn(dr, dr, __fmul_rn(di, di)), w, acc[i]);
          }
        }
      }
    }
    // fixed-order reduction: shuffle tree inside each warp, then warps in order
    if (TABLES || CC) {
#pragma unroll
      for (int i = 0; i < NT; ++i) {
        double vsum = (double)acc[i];
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) vsum += __shfl_xor_sync(0xffffffffu, vsum, off);
        if ((threadIdx.x & 31) == 0) s_cross[threadIdx.x >> 5][i] = vsum;
      }
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) nrm += __shfl_xor_sync(0xffffffffu, nrm, off);
      if ((threadIdx.x & 31) == 0) s_norm[threadIdx.x >> 5] = nrm;
    } else {
#pragma unroll
      for (int i = 0; i < NT; ++i) {
        float vsum = acc[i];
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) vsum += __shfl_xor_sync(0xffffffffu, vsum, off);
        if ((threadIdx.x & 31) == 0) s_part[threadIdx.x >> 5][i] = vsum;
      }
    }
    __syncthreads();
    if (threadIdx.x < nt) {
      if (TABLES || CC) {
        double cr = 0.0, nt2 = 0.0;
#pragma unroll
        for (int w = 0; w < kFineThreads / 32; ++w) {
          cr += s_cross[w][threadIdx.x];
          nt2 += s_norm[w];
        }
        diff2s[jb + base + threadIdx.x] = CC ? (float)(-cr / sqrt(nt2)) : (float)(fma(-2.0, cr, nt2) + (double)sum_init);
      } else {
        float tot = 0.f;
#pragma unroll
        for (int w = 0; w < kFineThreads / 32; ++w) tot += s_part[w][threadIdx.x];
        diff2s[jb + base + threadIdx.x] = tot + sum_init;
      }
    }
    __syncthreads();
  }
}

// Table path with the phase factored by rows.  With e^{i(x tx + y ty)} =
// e^{i x tx} e^{i y ty},
//   sum_px Re(q e^{i x tx} e^{i y ty}) = sum_x Re(e^{i x tx} R(x)),  R(x) = sum_y q(x, y) e^{i y ty},
// and rows y and -y of a column share their phases:
//   q+ e^{iya} + q- e^{-iya} = (q+ + q-) cos(ya) + i (q+ - q-) sin(ya).
// A thread owns one image column and a range of its rows.  Phase 1: it projects
// its pixels once per job (four unconditional fetches in flight) and keeps
// q = w conj(A) X in shared memory, with the per-pixel FP64 norms of
// diff2_fine_kernel.  Phase 2: it accumulates R over its rows |y|, 4 FMAs per
// pair of pixels and translation (8 when both are taken apart) for the job's
// translations rounded up to four, the row's phases of two translations in one
// 16-byte shared-memory load (the same address for every lane of a row);
// e^{i x tx} is applied once at the end.  The tables need y >= 0 only.  Rows
// that the fine mapping sends to x = maxR (between maxR and imgY - maxR) lie
// outside the projector radius, so their q is zero; a nonzero q there enters
// R(col) as q e^{i x' tx} conj(e^{i col tx}) e^{i y ty} (x' = maxR).  The
// threads' cross sums of a translation go through shared memory to one warp.
// Bound by the fetches' latency and by instruction issue (1.9 of 4 a clock with
// three CTAs a SM): 2048 jobs of 1 to 16 translations at image 64 take 61 us (72
// before: rows taken apart, fetches one by one, all 16 translations computed, FP64
// halving exchanges); of these the fetches are 27 us, phase 2 is 12, the
// tables 2.  Eight fetches in flight or four CTAs a SM spill: 80 us.
constexpr int kFineColsMaxThreads = 288;
__host__ __device__ inline int fine_cols_rows(int imgY, int maxR) { return max(maxR, imgY - maxR - 1) + 1; }
// Tables, q and sums of a CTA, at most: with its fixed part they stay within the
// 196 KB step of the shared-memory carve-out.  1024 jobs of 16 translations at
// image 200 (190 KB): 406 us, 629 with the pixels' own phases below; at image 212
// (214 KB, which leaves the fetches a 28 KB L1) 561 and 713 with the texture, but
// 3586 and 2718 with the linear projector.
constexpr size_t kFineColsSmem = 194 * 1024;
constexpr int kFineColsHalf = 8;              // translations whose sums are in shared memory at a time

// Phase 2 of diff2_fine_cols_kernel for the first NC of NT translations: folded
// rows [f0, f1) of column `col`, whose q lie imgX apart.
template <int NC, int NT>
__device__ __forceinline__ void fine_fold_rows(const float2* s_q, const float2* s_ey, int imgX, int imgY, int maxR,
                                               int col, int f0, int f1, int image_size, float (&rr)[NT],
                                               float (&ri)[NT]) {
  for (int f = f0; f < f1; ++f) {
    const int m = imgY - f;  // the row of y = -f
    const int p0 = f * imgX + col, p1 = m * imgX + col;
    const float2 qa = p0 < image_size ? s_q[p0] : make_float2(0.f, 0.f);
    const float2 qb = f > 0 && m > maxR && p1 < image_size ? s_q[p1] : make_float2(0.f, 0.f);
    const float sx = qa.x + qb.x, sy = qa.y + qb.y, dx = qa.x - qb.x, dy = qa.y - qb.y;
    const float4* pey = reinterpret_cast<const float4*>(s_ey + f * NT);
#pragma unroll
    for (int k = 0; k < NC / 2; ++k) {
      const float4 e = pey[k];  // (cos, sin) of translations 2k and 2k + 1
      rr[2 * k] = __fmaf_rn(sx, e.x, __fmaf_rn(-dy, e.y, rr[2 * k]));
      ri[2 * k] = __fmaf_rn(dx, e.y, __fmaf_rn(sy, e.x, ri[2 * k]));
      rr[2 * k + 1] = __fmaf_rn(sx, e.z, __fmaf_rn(-dy, e.w, rr[2 * k + 1]));
      ri[2 * k + 1] = __fmaf_rn(dx, e.w, __fmaf_rn(sy, e.z, ri[2 * k + 1]));
    }
  }
}

template <int NT, bool CC>
__global__ void __launch_bounds__(kFineColsMaxThreads, 3) diff2_fine_cols_kernel(
    b200d2_view v, const float* __restrict__ eulers, const float* __restrict__ re, const float* __restrict__ im,
    const float* __restrict__ tx, const float* __restrict__ ty, const float* __restrict__ corr,
    float* __restrict__ diff2s, int image_size, float sum_init, int groups, const uint64_t* __restrict__ rot_idx,
    const uint64_t* __restrict__ trans_idx, const uint64_t* __restrict__ job_idx,
    const uint64_t* __restrict__ job_num) {
  static_assert(NT == 16, "phase 2 is written for up to 16 translations");
  constexpr int kWarpsMax = kFineColsMaxThreads / 32, kHalf = kFineColsHalf;
  const uint64_t jb = job_idx[blockIdx.x];
  const int ntrans = (int)job_num[blockIdx.x];
  const uint64_t o = rot_idx[jb];
  const uint64_t t0 = trans_idx[jb];
  const float* eo = eulers + o * 9;
  const float e[6] = {eo[0], eo[1], eo[3], eo[4], eo[6], eo[7]};
  __shared__ double s_norm[kWarpsMax];
  __shared__ float s_t[2][NT];  // a pass' translations
  extern __shared__ __align__(16) float2 s_tab[];
  const int exw = max(v.imgX, v.maxR + 1), eyw = fine_cols_rows(v.imgY, v.maxR);
  float2* s_ex = s_tab;             // [NT][exw], x fastest
  float2* s_ey = s_tab + NT * exw;  // [eyw][NT], translation fastest, row y
  float2* s_q = s_ey + NT * eyw;    // [image_size]
  float* s_c = reinterpret_cast<float*>(s_q + image_size);  // [kHalf][threads]
  const int nthr = blockDim.x, nwarps = nthr >> 5, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int col = threadIdx.x % v.imgX, grp = threadIdx.x / v.imgX;
  const bool active = grp < groups;
  // (rows x groups stays below 2^23: the tables of the rows fit in shared memory)
  const int y0 = active ? (int)((unsigned)(grp * v.imgY) / (unsigned)groups) : 0;
  const int y1 = active ? (int)((unsigned)((grp + 1) * v.imgY) / (unsigned)groups) : 0;
  // phase 2's rows: y (and -y) in [f0, f1), and the rows in between in [m0, m1)
  const int nf = min(v.maxR, v.imgY - 1) + 1, nm = max(v.imgY - v.maxR - nf, 0);
  const int f0 = active ? (int)((unsigned)(grp * nf) / (unsigned)groups) : 0;
  const int f1 = active ? (int)((unsigned)((grp + 1) * nf) / (unsigned)groups) : 0;
  const int m0 = nf + (active ? (int)((unsigned)(grp * nm) / (unsigned)groups) : 0);
  const int m1 = nf + (active ? (int)((unsigned)((grp + 1) * nm) / (unsigned)groups) : 0);
  // the first pass' translations arrive while phase 1 runs
  if (threadIdx.x < 2 * NT) {
    const int i = threadIdx.x % NT;
    if (i < ntrans) s_t[threadIdx.x / NT][i] = (threadIdx.x < NT ? tx : ty)[t0 + i];
  }
  // phase 1 (once per job): q of this thread's pixels and its norm
  double nrm = 0.0;
  constexpr int kQ = 4;
  for (int yb = y0; yb < y1; yb += kQ) {
    float fx[kQ], fy[kQ], xr[kQ], xi[kQ], w[kQ];
    int pix[kQ];
    const float* es[kQ];
#pragma unroll
    for (int u = 0; u < kQ; ++u) {
      const int ys = yb + u;
      int x = col, y = ys;
      if (y > v.maxR) {  // the fine kernel's mapping (fine_pixel_coor)
        if (y >= v.imgY - v.maxR)
          y -= v.imgY;
        else
          x = v.maxR;
      }
      fx[u] = (float)x;
      fy[u] = (float)y;
      es[u] = e;
      pix[u] = ys < y1 ? ys * v.imgX + col : image_size;
      const int at = min(pix[u], image_size - 1);
      xr[u] = re[at];
      xi[u] = im[at];
      w[u] = corr[at];
    }
    PixelFetch<kQ, true> fetch;
    fetch.issue(v, fx, fy, es);
#pragma unroll
    for (int u = 0; u < kQ; ++u) {
      if (pix[u] >= image_size) continue;
      const float2 a = fetch.finish(u);
      const float wu = CC ? w[u] : 0.5f * w[u];
      const double ad = a.x, bd = a.y;
      if (CC) {
        nrm = fma((double)wu, fma(ad, ad, bd * bd), nrm);
      } else {
        const double xd = xr[u], yd = xi[u];
        nrm = fma((double)wu, fma(ad, ad, fma(bd, bd, fma(xd, xd, yd * yd))), nrm);
      }
      s_q[pix[u]] = make_float2(__fmul_rn(wu, __fmaf_rn(a.x, xr[u], __fmul_rn(a.y, xi[u]))),    // w Re(conj(A) X)
                                __fmul_rn(wu, __fmaf_rn(a.x, xi[u], -__fmul_rn(a.y, xr[u]))));  // w Im(conj(A) X)
    }
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) nrm += __shfl_xor_sync(0xffffffffu, nrm, off);
  if (lane == 0) s_norm[warp] = nrm;
  for (int base = 0; base < ntrans; base += NT) {  // passes of NT translations
    const int nt = min(NT, ntrans - base);
    if (base > 0 && threadIdx.x < 2 * NT) {
      const int i = threadIdx.x % NT;
      if (i < nt) s_t[threadIdx.x / NT][i] = (threadIdx.x < NT ? tx : ty)[t0 + base + i];
    }
    __syncthreads();
    const int nc = (nt + 3) & ~3;  // translations of phase 2, nt of them real
    for (int e2 = threadIdx.x; e2 < nc * (exw + eyw); e2 += nthr) {
      float sn = 0.f, cs = 1.f;
      if (e2 < nc * exw) {
        const int i = (int)((unsigned)e2 / (unsigned)exw), x = e2 - i * exw;
        if (i < nt) sincosf(__fmul_rn((float)x, s_t[0][i]), &sn, &cs);
        s_ex[e2] = make_float2(cs, sn);
      } else {
        const int j = e2 - nc * exw, i = (int)((unsigned)j / (unsigned)eyw), y = j - i * eyw;
        if (i < nt) sincosf(__fmul_rn((float)y, s_t[1][i]), &sn, &cs);
        s_ey[y * NT + i] = make_float2(cs, sn);
      }
    }
    __syncthreads();  // tables (and, on the first pass, q and the norms) ready
    // phase 2: R for this thread's column and rows
    float rr[NT], ri[NT];
#pragma unroll
    for (int i = 0; i < NT; ++i) rr[i] = ri[i] = 0.f;
    if (nc == 4)
      fine_fold_rows<4, NT>(s_q, s_ey, v.imgX, v.imgY, v.maxR, col, f0, f1, image_size, rr, ri);
    else if (nc == 8)
      fine_fold_rows<8, NT>(s_q, s_ey, v.imgX, v.imgY, v.maxR, col, f0, f1, image_size, rr, ri);
    else if (nc == 12)
      fine_fold_rows<12, NT>(s_q, s_ey, v.imgX, v.imgY, v.maxR, col, f0, f1, image_size, rr, ri);
    else
      fine_fold_rows<16, NT>(s_q, s_ey, v.imgX, v.imgY, v.maxR, col, f0, f1, image_size, rr, ri);
    for (int ys = m0; ys < m1; ++ys) {
      const int pixel = ys * v.imgX + col;
      if (pixel >= image_size) break;  // later rows of this column lie further on
      const float2 q = s_q[pixel];
      if (q.x == 0.f && q.y == 0.f) continue;
      const float2* pey = s_ey + ys * NT;  // a remapped row with a nonzero projection
#pragma unroll
      for (int i = 0; i < NT; ++i) {
        if (i >= nc) continue;
        const float2 ex = s_ex[i * exw + v.maxR], cx = s_ex[i * exw + col], ey = pey[i];
        // d = e^{i x' tx} conj(e^{i col tx}) e^{i y ty}
        const bool same = col == v.maxR;
        const float dr0 = same ? 1.f : __fmaf_rn(ex.x, cx.x, __fmul_rn(ex.y, cx.y));
        const float di0 = same ? 0.f : __fmaf_rn(ex.y, cx.x, -__fmul_rn(ex.x, cx.y));
        const float dr = __fmaf_rn(dr0, ey.x, -__fmul_rn(di0, ey.y));
        const float di = __fmaf_rn(dr0, ey.y, __fmul_rn(di0, ey.x));
        rr[i] = __fmaf_rn(q.x, dr, __fmaf_rn(-q.y, di, rr[i]));
        ri[i] = __fmaf_rn(q.x, di, __fmaf_rn(q.y, dr, ri[i]));
      }
    }
    // this thread's cross sums Re(e^{i col tx} R); then a warp adds up the
    // threads' sums of one translation in FP64, in a fixed order.  Eight
    // translations at a time: the area for all sixteen would cost images of
    // 104 to 112 pixels their third CTA on a SM.
#pragma unroll
    for (int h = 0; h < NT; h += kHalf) {
      if (h >= nt) break;
      if (h > 0) __syncthreads();
#pragma unroll
      for (int i = 0; i < kHalf; ++i) {
        if (h + i >= nc) break;
        const float2 f = s_ex[(h + i) * exw + col];
        s_c[i * nthr + threadIdx.x] = active ? __fmaf_rn(f.x, rr[h + i], -__fmul_rn(f.y, ri[h + i])) : 0.f;
      }
      __syncthreads();
      for (int i = warp; i < kHalf && h + i < nt; i += nwarps) {
        double cr = 0.0, nt2 = 0.0;
#pragma unroll
        for (int w = 0; w < kWarpsMax; ++w)
          if (w < nwarps) cr += (double)s_c[i * nthr + w * 32 + lane];
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) cr += __shfl_xor_sync(0xffffffffu, cr, off);
        if (lane == 0) {
          for (int w = 0; w < nwarps; ++w) nt2 += s_norm[w];
          diff2s[jb + base + h + i] = CC ? (float)(-cr / sqrt(nt2)) : (float)(fma(-2.0, cr, nt2) + (double)sum_init);
        }
      }
    }
    __syncthreads();  // the sums and the tables are reused by the next pass
  }
}

}  // namespace b200d2

namespace {

template <bool CC>
int launch_fine(const b200d2_view* view, const float* d_eulers, const float* d_real, const float* d_imag,
                const float* d_trans_x, const float* d_trans_y, const float* d_corr, float* d_diff2s,
                size_t image_size, float sum_init, size_t todo_blocks, const uint64_t* d_rot_idx,
                const uint64_t* d_trans_idx, const uint64_t* d_job_idx, const uint64_t* d_job_num, void* stream) {
  using namespace b200d2;
  if (!view) return B200D2_ERR_INVALID;
  if (todo_blocks == 0 || image_size == 0) return B200D2_OK;
  if (!d_eulers || !d_real || !d_imag || !d_trans_x || !d_trans_y || !d_corr || !d_diff2s || !d_rot_idx ||
      !d_trans_idx || !d_job_idx || !d_job_num)
    return B200D2_ERR_INVALID;
  if (view->mdlZ == 0) return B200D2_ERR_UNSUPPORTED;  // 2D references are outside the ported branch
  if ((long long)view->imgX * view->imgY < (long long)image_size || image_size > 0x7fffffffull)
    return B200D2_ERR_INVALID;
  if (view->interp == B200D2_INTERP_TEXTURE && (!view->tex_re || !view->tex_im)) return B200D2_ERR_INVALID;
  if (view->interp == B200D2_INTERP_LINEAR && (!view->lin_re || !view->lin_im)) return B200D2_ERR_INVALID;
  if (todo_blocks > 0x7fffffffull) return B200D2_ERR_UNSUPPORTED;
  const size_t exw = (size_t)std::max(view->imgX, view->maxR + 1);
  const size_t tab_bytes = sizeof(float2) * kFineMaxTrans * (exw + view->imgY + view->maxR);
  // one thread per (column, row group), about 256 threads, whole warps
  const int groups = view->imgX <= 0 ? 1 : std::max(1, std::min(view->imgY, std::min((256 + view->imgX / 2) / view->imgX,
                                                                                      kFineColsMaxThreads / view->imgX)));
  const size_t threads = ((size_t)view->imgX * groups + 31) / 32 * 32;
  const size_t cols_bytes =  // tables, q and the threads' sums
      sizeof(float2) * (kFineMaxTrans * (exw + (size_t)fine_cols_rows(view->imgY, view->maxR)) + image_size) +
      sizeof(float) * kFineColsHalf * threads;
  if (view->maxR >= 0 && view->imgX > 0 && view->imgY > 0 && cols_bytes <= kFineColsSmem &&
      view->imgX <= kFineColsMaxThreads) {
    static std::atomic<unsigned long long> opted{0};  // above 48 KB of dynamic shared memory
    B200D2_CUDA_TRY(smem_opt_in(diff2_fine_cols_kernel<kFineMaxTrans, CC>, (int)kFineColsSmem, opted));
    diff2_fine_cols_kernel<kFineMaxTrans, CC><<<(unsigned)todo_blocks, (unsigned)threads, cols_bytes, (cudaStream_t)stream>>>(
        *view, d_eulers, d_real, d_imag, d_trans_x, d_trans_y, d_corr, d_diff2s, (int)image_size, sum_init, groups,
        d_rot_idx, d_trans_idx, d_job_idx, d_job_num);
  } else if (view->maxR >= 0 && view->imgX > 0 && view->imgY > 0 && tab_bytes <= kFineTableBytes) {
    static std::atomic<unsigned long long> opted{0};  // above 48 KB of dynamic shared memory
    B200D2_CUDA_TRY(smem_opt_in(diff2_fine_kernel<kFineMaxTrans, true, CC>, (int)kFineTableBytes, opted));
    diff2_fine_kernel<kFineMaxTrans, true, CC><<<(unsigned)todo_blocks, kFineThreads, tab_bytes,
                                                 (cudaStream_t)stream>>>(
        *view, d_eulers, d_real, d_imag, d_trans_x, d_trans_y, d_corr, d_diff2s, (int)image_size, sum_init,
        d_rot_idx, d_trans_idx, d_job_idx, d_job_num);
  } else {
    diff2_fine_kernel<kFineMaxTrans, false, CC><<<(unsigned)todo_blocks, kFineThreads, 0, (cudaStream_t)stream>>>(
        *view, d_eulers, d_real, d_imag, d_trans_x, d_trans_y, d_corr, d_diff2s, (int)image_size, sum_init,
        d_rot_idx, d_trans_idx, d_job_idx, d_job_num);
  }
  count_launch();
  return status_from_cuda(cudaGetLastError());
}

}  // namespace

extern "C" int b200d2_diff2_fine(const b200d2_view* view, const float* d_eulers, const float* d_real,
                                 const float* d_imag, const float* d_trans_x, const float* d_trans_y,
                                 const float* d_corr, float* d_diff2s, size_t image_size, float sum_init,
                                 size_t todo_blocks, const uint64_t* d_rot_idx, const uint64_t* d_trans_idx,
                                 const uint64_t* d_job_idx, const uint64_t* d_job_num, void* stream) {
  return launch_fine<false>(view, d_eulers, d_real, d_imag, d_trans_x, d_trans_y, d_corr, d_diff2s, image_size,
                            sum_init, todo_blocks, d_rot_idx, d_trans_idx, d_job_idx, d_job_num, stream);
}

extern "C" int b200d2_diff2_fine_cc(const b200d2_view* view, const float* d_eulers, const float* d_real,
                                    const float* d_imag, const float* d_trans_x, const float* d_trans_y,
                                    const float* d_corr, float* d_diff2s, size_t image_size, size_t todo_blocks,
                                    const uint64_t* d_rot_idx, const uint64_t* d_trans_idx,
                                    const uint64_t* d_job_idx, const uint64_t* d_job_num, void* stream) {
  return launch_fine<true>(view, d_eulers, d_real, d_imag, d_trans_x, d_trans_y, d_corr, d_diff2s, image_size,
                           0.f, todo_blocks, d_rot_idx, d_trans_idx, d_job_idx, d_job_num, stream);
}
