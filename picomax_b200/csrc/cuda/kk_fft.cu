// Kramers-Kronig transform of uniform frequency grids by FFT.
//
// src/pmx_chi.cpp:272-309: Re_f += ds sum_{s != f} K_fs Im_s, Im_f += ds
// sum_{s != f} K_fs Re0_s with K_fs = w_s / (w_s^2 - w_f^2), ds = 2 dw / pi, both
// from the values before the transform. On the grid w_s = dw s
//   dw K_fs = 1/2 [ 1 / (s - f) + 1 / (s + f) ]      (s != f),
// a Toeplitz and a Hankel matrix, so both sums of a row are circular convolutions
// of length L >= 2 nf - 1: with X the transform of the row,
//   Y_k = i alpha_k X_k + H_k X_{-k},
//   alpha_k = sum_{d=1}^{nf-1} sin(2 pi k d / L) / d,   H = transform of 1 / (2 g), 1 <= g <= 2 nf - 2,
// less the s = f entry of the Hankel part, x_f / (4 f). Re and Im of a row are the
// two halves of one complex sequence, so a row costs one forward and one inverse
// complex FFT. The adjoint's transposed transform (kk_t) is the same with -alpha.
//
// One CTA per row, the sequence in shared memory: radix-8 passes in place, forward
// by decimation in frequency (bit-reversed result), inverse by decimation in time
// from that order, so nothing is reordered. In the bit-reversed order the partner
// -k of position p is p with all bits below its highest one flipped: a mirrored
// contiguous run. Bound by shared-memory passes (8 per row at nf 2000), not by the
// HBM bytes of the rows; the direct sum it replaces was bound by the FP64 pipe
// (4 nf^2 per row and one division per kernel entry and tile). Measured on a B200
// at 2000 frequencies: 3402 rows 4.62 -> 0.29 ms, 15930 rows 21.1 -> 1.29 ms; at
// 1000, 1080 rows 0.41 -> 0.058 ms. Error against 80-bit sums at 2000 frequencies
// 2.4e-16 of the norm (the direct sum, whose kernel entries lose digits in
// w_s^2 - w_f^2, 3.7e-14).
//
// Re and Im of a row are scaled by powers of two to the same size before they share
// a sequence, and a row that is zero stays exactly zero in the other's sum; entry 0,
// which the forward transform does not weigh, has no part in that size. Rows with
// non-finite or (but for entry 0) huge entries, which a transform would spread over
// the row, take the direct sum, its kernel from a table of reciprocals in the sequence's
// place (call on 400 rows of 2000 with a NaN each: 5.7 ms by the tiled direct kernel, 7.9
// with a division per term here, 6.7 with the table; without a NaN the FFT takes over).
#include <algorithm>
#include <cfloat>
#include <cmath>

#include "pmx_chi.hpp"
#include "pmx_common.cuh"

namespace pmx {
namespace dev {

namespace {

constexpr int kMinLog = 4, kMaxLog = 13;  // L = 16 .. 8192 (144 KB of shared memory)
constexpr int kMaxThr = 256;
constexpr double kTwoOverPi = 0.63661977236758134308;

// one entry of padding per 8: accesses of stride 8, 64, ... stay free of bank conflicts
__host__ __device__ __forceinline__ int pad(int i) { return i + (i >> 3); }

inline int log_len(int nf) {
  int b = kMinLog;
  while ((1 << b) < 2 * nf - 1) ++b;
  return b;
}
inline size_t smem_bytes(int logl) { return sizeof(double2) * (size_t)pad(1 << logl) + 64 * sizeof(double); }

__device__ __forceinline__ double2 mul_mi(double2 a) { return make_double2(a.y, -a.x); }  // -i a

// forward: exp(-2 pi i j / L) as stored; inverse: its conjugate
template <bool INV>
__device__ __forceinline__ double2 tw(const double2* __restrict__ w, int j) {
  double2 v = __ldg(w + j);
  if (INV) v.y = -v.y;
  return v;
}

// R = 2^LR elements at distance q of one block, LR radix-2 stages in registers.
// Forward (decimation in frequency): difference times twiddle; inverse
// (decimation in time, the same stages backwards): twiddle, then sum and
// difference. t[0] = w_block^i, t[1] = t[0]^2, t[2] = t[0]^4 (table entries).
template <int LR, bool INV>
__device__ __forceinline__ void butterflies(double2 (&v)[1 << LR], const double2 (&t)[3]) {
  constexpr int R = 1 << LR;
  constexpr double kH = 0.70710678118654752440;
#pragma unroll
  for (int s0 = 0; s0 < LR; ++s0) {
    const int s = INV ? LR - 1 - s0 : s0;
    const int half = R >> (s + 1);
#pragma unroll
    for (int m = 0; m < R; ++m) {
      if (m & half) continue;
      const int pos = m & (half - 1);
      // w_(2 half)^pos, 2 half in {2, 4, 8}: eighth roots, as turns of -pi/4 (forward)
      const int e8 = pos * (8 / (2 * half));
      auto turn = [&](double2 a) {
        if (e8 == 0) return a;
        if (INV) {
          if (e8 == 1) return make_double2(kH * (a.x - a.y), kH * (a.x + a.y));
          if (e8 == 2) return make_double2(-a.y, a.x);
          return make_double2(-kH * (a.x + a.y), kH * (a.x - a.y));
        }
        if (e8 == 1) return make_double2(kH * (a.x + a.y), kH * (a.y - a.x));
        if (e8 == 2) return mul_mi(a);
        return make_double2(kH * (a.y - a.x), -kH * (a.x + a.y));
      };
      const double2 a = v[m];
      if (!INV) {
        const double2 b = v[m + half];
        v[m] = cadd(a, b);
        v[m + half] = cmul(turn(csub(a, b)), t[s]);
      } else {
        const double2 b = turn(cmul(v[m + half], t[s]));
        v[m] = cadd(a, b);
        v[m + half] = csub(a, b);
      }
    }
  }
}

template <int LR, bool INV>
__device__ __forceinline__ void pass(double2* z, const double2* __restrict__ w, int logl, int logblock) {
  constexpr int R = 1 << LR;
  const int logq = logblock - LR, q = 1 << logq;
  for (int idx = threadIdx.x; idx < (1 << (logl - LR)); idx += blockDim.x) {
    const int i = idx & (q - 1), base = ((idx >> logq) << logblock) + i;
    double2 v[R], t[3];
#pragma unroll
    for (int m = 0; m < R; ++m) v[m] = z[pad(base + (m << logq))];
#pragma unroll
    for (int s = 0; s < 3; ++s) t[s] = s < LR ? tw<INV>(w, (i << s) << (logl - logblock)) : make_double2(1, 0);
    butterflies<LR, INV>(v, t);
#pragma unroll
    for (int m = 0; m < R; ++m) z[pad(base + (m << logq))] = v[m];
  }
  __syncthreads();
}

// in place, natural -> bit-reversed order
__device__ __forceinline__ void fft_forward(double2* z, const double2* __restrict__ w, int logl) {
  int b = logl;
  if (logl % 3 == 1) {
    pass<1, false>(z, w, logl, b);
    b -= 1;
  } else if (logl % 3 == 2) {
    pass<2, false>(z, w, logl, b);
    b -= 2;
  }
  for (; b > 0; b -= 3) pass<3, false>(z, w, logl, b);
}
// in place, bit-reversed -> natural order, without the factor 1 / L
__device__ __forceinline__ void fft_inverse(double2* z, const double2* __restrict__ w, int logl) {
  int b = 3;
  for (; b <= logl; b += 3) pass<3, true>(z, w, logl, b);
  if (logl % 3 == 1) pass<1, true>(z, w, logl, logl);
  if (logl % 3 == 2) pass<2, true>(z, w, logl, logl);
}

// positions p (k) and p' (-k) of the pair u in [0, L / 2); u = 0 is (0, L / 2)
__device__ __forceinline__ void pair_pos(int u, int& p, int& pm) {
  if (u == 0) {
    p = 0;
    pm = 1;
    return;
  }
  const int hb = 32 - __clz(u);  // 2^(hb-1) <= u < 2^hb
  p = (1 << hb) + (u - (1 << (hb - 1)));
  pm = p ^ ((1 << hb) - 1);
}

// tables of one grid length: w [L] roots of unity, alpha [L / 2] and H [L / 2] in
// pair order (H of pair 0 is (H_0, H_{L/2}), both real)
struct Tables {
  double2* w;
  double2* h;
  double* alpha;
};
inline size_t table_bytes(int logl) { return (sizeof(double2) * 3 / 2 + sizeof(double) / 2) * ((size_t)1 << logl); }
inline Tables tables(void* ws, int logl) {
  Tables t;
  t.w = reinterpret_cast<double2*>(ws);
  t.h = t.w + ((size_t)1 << logl);
  t.alpha = reinterpret_cast<double*>(t.h + ((size_t)1 << (logl - 1)));
  return t;
}

__global__ void kk_roots_kernel(double2* __restrict__ w, int l) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= l) return;
  double s, c;
  sincospi(2.0 * j / l, &s, &c);
  w[j] = make_double2(c, -s);
}

// block 0: alpha, block 1: H
__global__ void __launch_bounds__(kMaxThr) kk_tables_kernel(Tables t, int nf, int logl) {
  extern __shared__ __align__(16) unsigned char smraw[];
  double2* z = reinterpret_cast<double2*>(smraw);
  const int l = 1 << logl;
  for (int j = threadIdx.x; j < l; j += blockDim.x) {
    double v = 0.0;
    if (blockIdx.x == 0) {
      if (j >= 1 && j <= nf - 1) v = -0.5 / j;
      if (l - j >= 1 && l - j <= nf - 1) v = 0.5 / (l - j);
    } else if (j >= 1 && j <= 2 * nf - 2) {
      v = 0.5 / j;
    }
    z[pad(j)] = make_double2(v, 0.0);
  }
  __syncthreads();
  fft_forward(z, t.w, logl);
  for (int u = threadIdx.x; u < l / 2; u += blockDim.x) {
    int p, pm;
    pair_pos(u, p, pm);
    const double2 a = z[pad(p)];
    if (blockIdx.x == 0)
      t.alpha[u] = u == 0 ? 0.0 : a.y;
    else
      t.h[u] = u == 0 ? make_double2(a.x, z[pad(pm)].x) : a;
  }
}

// largest of a value over the block; every thread gets it. red: 32 doubles
__device__ __forceinline__ double block_max(double v, double* red) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
  const int nw = blockDim.x >> 5;
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  double m = red[0];
  for (int i = 1; i < nw; ++i) m = fmax(m, red[i]);
  __syncthreads();
  return m;
}

// in: [2][rows][nf] (Re block, then Im block), out the same; TR: the transposed
// transform. One CTA per row.
template <bool TR>
__global__ void __launch_bounds__(kMaxThr, 3) kk_fft_kernel(const double* __restrict__ in, double* __restrict__ out,
                                                         int rows, int nf, double dfreq, Tables t, int logl) {
  extern __shared__ __align__(16) unsigned char smraw[];
  double2* z = reinterpret_cast<double2*>(smraw);
  const int l = 1 << logl;
  double* red = reinterpret_cast<double*>(z + pad(l));
  const size_t o = (size_t)blockIdx.x * nf, blk = (size_t)rows * nf;
  const double* re = in + o;
  const double* im = in + blk + o;
  // entry 0 of the input has no weight (w_0 = 0) in the forward transform: it stays out
  // of the sequence and of the sizes that scale it (a NaN or Inf there still spreads)
  double mr = 0.0, mi = 0.0;
  int bad = 0;
  for (int s = threadIdx.x; s < nf; s += blockDim.x) {
    const double a = re[s], b = im[s];
    if (!TR && s == 0) {
      bad |= !isfinite(a) | !isfinite(b);
      z[0] = make_double2(0, 0);
      continue;
    }
    bad |= !(fabs(a) <= 1e290) | !(fabs(b) <= 1e290);
    mr = fmax(mr, fabs(a));
    mi = fmax(mi, fabs(b));
    z[pad(s)] = make_double2(a, b);
  }
  for (int s = nf + threadIdx.x; s < l; s += blockDim.x) z[pad(s)] = make_double2(0, 0);
  bad = __syncthreads_or(bad);
  if (bad) {  // direct sums of this row, dw K_fs from a table of 1 / (2 g), g < 2 nf - 1 <= l
    double* rc = reinterpret_cast<double*>(z);
    for (int g = threadIdx.x; g < 2 * nf - 1; g += blockDim.x) rc[g] = 0.5 / g;
    __syncthreads();
    for (int f = threadIdx.x; f < nf; f += blockDim.x) {
      double ar = 0.0, ai = 0.0;
#pragma unroll 8
      for (int s = 0; s < f; ++s) {
        const double k = TR ? rc[s + f] + rc[f - s] : rc[s + f] - rc[f - s];
        ar = fma(im[s], k, ar);
        ai = fma(re[s], k, ai);
      }
#pragma unroll 8
      for (int s = f + 1; s < nf; ++s) {
        const double k = TR ? rc[s + f] - rc[s - f] : rc[s + f] + rc[s - f];
        ar = fma(im[s], k, ar);
        ai = fma(re[s], k, ai);
      }
      out[o + f] = re[f] + kTwoOverPi * ar;
      out[blk + o + f] = im[f] + kTwoOverPi * ai;
    }
    return;
  }
  mr = block_max(mr, red);
  mi = block_max(mi, red + 32);
  const bool has_re = mr > 0.0, has_im = mi > 0.0;
  const int er = has_re ? ilogb(mr) : 0, ei = has_im ? ilogb(mi) : 0;
  for (int s = threadIdx.x; s < nf; s += blockDim.x) {
    const double2 v = z[pad(s)];
    z[pad(s)] = make_double2(scalbn(v.x, -er), scalbn(v.y, -ei));
  }
  __syncthreads();
  fft_forward(z, t.w, logl);
  for (int u = threadIdx.x; u < l / 2; u += blockDim.x) {
    int p, pm;
    pair_pos(u, p, pm);
    const double2 x = z[pad(p)], y = z[pad(pm)], h = t.h[u];
    if (u == 0) {
      z[pad(p)] = cscale(x, h.x);
      z[pad(pm)] = cscale(y, h.y);
    } else {
      const double al = TR ? -t.alpha[u] : t.alpha[u];
      // i al x + h y, and at -k: -i al y + conj(h) x
      const double2 a = cmul(h, y), b = cmulc(h, x);
      z[pad(p)] = make_double2(a.x - al * x.y, a.y + al * x.x);
      z[pad(pm)] = make_double2(b.x + al * y.y, b.y - al * y.x);
    }
  }
  __syncthreads();
  fft_inverse(z, t.w, logl);
  const double il = 1.0 / l;  // a power of two
  for (int f = threadIdx.x; f < nf; f += blockDim.x) {
    const double a = re[f], b = im[f];
    const double2 y = z[pad(f)];
    const double c = f > 0 ? 0.25 / f : 0.0;
    // sums over re and im, less the Hankel entry s = f; entry 0 of the transposed one is zero
    double yr = has_re ? scalbn(y.x * il, er) - c * a : 0.0;
    double yi = has_im ? scalbn(y.y * il, ei) - c * b : 0.0;
    if (TR && f == 0) yr = yi = 0.0;
    out[o + f] = a + kTwoOverPi * yi;
    out[blk + o + f] = b + kTwoOverPi * yr;
  }
}

}  // namespace

// the longest grid whose transform fits in shared memory (L = 8192, 144 KB)
int kk_fft_max_nf() { return ((1 << kMaxLog) + 1) / 2; }

size_t kk_fft_table_bytes(int nf) { return table_bytes(log_len(nf)); }

cudaError_t launch_kk_tables(int nf, void* ws, cudaStream_t st) {
  if (nf < 1 || nf > kk_fft_max_nf()) return cudaErrorInvalidValue;
  const int logl = log_len(nf);
  const Tables t = tables(ws, logl);
  kk_roots_kernel<<<((1 << logl) + 255) / 256, 256, 0, st>>>(t.w, 1 << logl);
  const cudaError_t e =
      cudaFuncSetAttribute(kk_tables_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes(logl));
  if (e != cudaSuccess) return e;
  kk_tables_kernel<<<2, kMaxThr, smem_bytes(logl), st>>>(t, nf, logl);
  return cudaGetLastError();
}

cudaError_t launch_kk_fft(const double* in, double* out, int rows, int nf, double dfreq, bool transposed, void* ws,
                          cudaStream_t st) {
  if (rows <= 0) return cudaSuccess;
  if (nf < 1 || nf > kk_fft_max_nf()) return cudaErrorInvalidValue;
  const int logl = log_len(nf);
  const int thr = std::min(kMaxThr, std::max(32, 1 << (logl - 3)));
  auto kernel = transposed ? kk_fft_kernel<true> : kk_fft_kernel<false>;
  const cudaError_t e =
      cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes(logl));
  if (e != cudaSuccess) return e;
  kernel<<<rows, thr, smem_bytes(logl), st>>>(in, out, rows, nf, dfreq, tables(ws, logl), logl);
  return cudaGetLastError();
}

}  // namespace dev
}  // namespace pmx
