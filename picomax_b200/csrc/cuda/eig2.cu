// Two-stage batched FP64 Hermitian eigensolver: dense -> band -> tridiagonal.
//
// Replaces Eigen::SelfAdjointEigenSolver (src/pmx_epm.cpp:232, :402,
// src/pmx_chi.cpp:388, :476) for n from 96 up to a padded size of 1216. The
// one-stage reduction (epm.cu) passes over the whole trailing block once per
// column; here the Householder reduction is
// split the way blocked LAPACK/PLASMA solvers split it (Bischof, Lang, Sun,
// "A framework for symmetric band reduction", ACM TOMS 26 (2000); Haidar,
// Ltaief, Dongarra, SC'11), each stage B200-shaped:
//
//  1. sb_kernel (one CTA per matrix): panels of 16 columns. A panel is
//     QR-factorised in shared memory (Householder, compact WY T factor), then
//     the trailing block is updated two-sidedly with two passes of 16 x 16
//     complex tiles on the FP64 tensor cores (mma.sync m8n8k4 .f64):
//       Y = A V          (all tiles, the upper ones read as conj-transposes)
//       X = Y T - 1/2 V (T^H V^H Y T)
//       A -= V X^H + X V^H   (lower tiles and the diagonal tiles in full)
//     Each pass reads (and the second writes) the trailing block once per
//     panel instead of once per column. The panel's reflectors stay in place
//     below the band (LAPACK layout); T goes into the free upper tile.
//     Up to ld = 416 the panel V and Y live in shared memory; beyond that
//     (ld <= 800) Y lives in the item's slot of the reflector buffer (L2),
//     and beyond ld = 800 (ld <= 1216) V as well.
//  2. sbtrd_kernel (one CTA per matrix): the band (16 sub-diagonals plus 16
//     for the bulge) lives in shared memory up to ld = 416, beyond that in
//     the item's slot of the reflector buffer (L1/L2); sweeps chase their bulges down
//     the band, eight at a time (four in large batches of small matrices; a pair of
//     warps per sweep), each step of a
//     sweep waiting only for the previous sweep to leave its rows (progress
//     words in shared memory, no block-wide barrier). Reflectors go to
//     global memory.
//  3. tri_val_kernel, tri_vec_kernel: bisection and inverse iteration on the
//     tridiagonal matrix (pmx_trieig.cuh), one CTA per matrix, so that many
//     matrices share an SM.
//  4. band_back_kernel: eigenvectors of T -> of the band (the bulge-chasing
//     reflectors, 16 sweeps at a time, the vectors' rows in registers);
//     panel_back_kernel: -> of H (the panels' compact WY factors in reverse).
//
// The matrix dimension is padded to ld = a multiple of 16 with zero rows and
// columns: every reflector then has zero components in the padding, so T is
// block diagonal with the n x n block of the unpadded problem (e[n-1] = 0
// exactly) and the eigenvectors are exactly zero in the padding.
#include <algorithm>
#include <cfloat>
#include <climits>
#include <cmath>

#include "pmx_common.cuh"
#include "pmx_device.hpp"
#include "pmx_dmma.cuh"
#include "pmx_trieig.cuh"

namespace pmx {
namespace dev {

namespace {

constexpr int kNB = 16;        // panel width = band width
constexpr int kThr = 256;      // threads per CTA of every stage
constexpr int kNW = kThr / 32;
constexpr int kMaxLd = 1216;   // largest padded dimension
constexpr int kVSmemLd = 800;  // largest one whose stage-1 V fits in shared memory
constexpr int kSmallLd = 160;  // up to it stages 1 and 2 run two CTAs per SM
constexpr int kSmemLd = 416;   // largest one whose stage-1 Y and stage-2 band fit in shared memory

// element (r, c) of an m x 16 complex panel in shared memory: rows of 16,
// columns XOR-swizzled by the row so that the tensor-core fragment loads of
// 8 rows x 4 columns and of 4 rows x 8 columns are free of bank conflicts
__device__ __forceinline__ int pidx(int r, int c) { return r * kNB + (c ^ (r & 7)); }

// acc -= a * conj(b') where the B fragment element is b'(row k, col j) taken
// from a matrix stored as X[j][k] (so the product is V X^H)
__device__ __forceinline__ void cmma_sub_herm(double (&cr)[2], double (&ci)[2], double2 a, double2 x) {
  dmma(cr[0], cr[1], -a.x, x.x);
  dmma(cr[0], cr[1], -a.y, x.y);
  dmma(ci[0], ci[1], a.x, x.y);
  dmma(ci[0], ci[1], -a.y, x.x);
}

// acc += a b, acc += conj(a) b, acc -= a b, acc -= a conj(b)
__device__ __forceinline__ void cfma(double2& acc, double2 a, double2 b) {
  acc.x = fma(a.x, b.x, fma(-a.y, b.y, acc.x));
  acc.y = fma(a.x, b.y, fma(a.y, b.x, acc.y));
}
__device__ __forceinline__ void cfmac(double2& acc, double2 a, double2 b) {
  acc.x = fma(a.x, b.x, fma(a.y, b.y, acc.x));
  acc.y = fma(a.x, b.y, fma(-a.y, b.x, acc.y));
}
__device__ __forceinline__ void cfms(double2& acc, double2 a, double2 b) {
  acc.x = fma(-a.x, b.x, fma(a.y, b.y, acc.x));
  acc.y = fma(-a.x, b.y, fma(-a.y, b.x, acc.y));
}
__device__ __forceinline__ void cfmsc(double2& acc, double2 a, double2 b) {
  acc.x = fma(-a.x, b.x, fma(-a.y, b.y, acc.x));
  acc.y = fma(a.x, b.y, fma(-a.y, b.x, acc.y));
}

// sum over the first `w` lanes' groups: xor reductions within 16 lanes
__device__ __forceinline__ double sum16(double v) {
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Householder reflector in the zlarfg convention: H^H (alpha; x) = (beta; 0),
// H = I - tau v v^H, v[0] = 1, beta real. From alpha and |x|^2 gives tau, beta
// and the scale 1 / (alpha - beta) of x.
struct Refl {
  double2 tau;
  double beta;
  double2 scal;
};
// 1 / beta is the reciprocal square root, beta its product with the sum corrected
// by one Newton step (to the rounding of a square root): one rsqrt and one
// reciprocal, where a square root and two divisions took twice the instructions
// on the chain that every column and every bulge waits for.
__device__ __forceinline__ Refl make_refl(double2 alpha, double xn) {
  Refl r;
  if (xn == 0.0 && alpha.y == 0.0) {
    r.tau = make_double2(0, 0);
    r.beta = alpha.x;
    r.scal = make_double2(1, 0);
  } else {
    const double s2 = fma(alpha.x, alpha.x, fma(alpha.y, alpha.y, xn));
    const double rs = rsqrt(s2);
    double nrm = s2 * rs;
    nrm = fma(0.5 * rs, fma(-nrm, nrm, s2), nrm);
    r.beta = -copysign(nrm, alpha.x);
    const double ib = -copysign(rs, alpha.x);
    const double2 den = make_double2(alpha.x - r.beta, alpha.y);
    const double idd = 1.0 / fma(den.x, den.x, den.y * den.y);
    r.tau = make_double2(fma(-alpha.x, ib, 1.0), -alpha.y * ib);
    r.scal = make_double2(den.x * idd, -den.y * idd);
  }
  return r;
}

// number of bulge-chasing tasks (= reflectors) of sweep s of an ld x ld band
__host__ __device__ __forceinline__ int sweep_steps(int ld, int s) { return (ld - 1 - s + kNB - 1) / kNB; }
// sum_{m=1}^{M} ceil(m / 16)
__host__ __device__ __forceinline__ long long ceil_sum(long long M) {
  const long long q = M / kNB, r = M % kNB;
  return kNB * q * (q + 1) / 2 + r * (q + 1);
}
// index of the first reflector of sweep s
__host__ __device__ __forceinline__ long long sweep_first(int ld, int s) { return ceil_sum(ld - 1) - ceil_sum(ld - 1 - s); }
// Slot of an item in the reflector buffer (double2 offsets): the band
// reflectors [ceil_sum(ld - 1)][16], the tridiagonal (2 ld doubles), and, in
// launches with ld > kSmemLd, a work area of 32 (ld + 16) double2: stage 1's Y
// (16 (ld - 16)) and, for ld > kVSmemLd, V after it (16 (ld - 16)); then
// stage 2's band (32 (ld + 16)).
__host__ __device__ __forceinline__ long long band_off(int ld) { return ceil_sum(ld - 1) * kNB + ld; }

// ------------------------------------------------------------------ stage 1
struct SbSmem {
  double2* V;     // [mmax * 16] panel / reflectors V (explicit unit lower trapezoid)
  double2* Y;     // [mmax * 16] Y = A V, then X
  double2* T;     // [16 * 17]
  double2* M;     // [16 * 17] V^H Y (the panel QR's T dots before that)
  double2* P;     // [16 * 17] T^H M
  double2* taus;  // [16]
  // panel QR work arrays, inside Y (free until Y = A V is formed)
  double2* part;  // [2][8][16] partial sums of the panel QR
  double2* rowj;  // [2][16] the current row of the panel QR
  double2* pvw;   // [8][2][MR] per-warp pivot buffers of the panel QR
};

// register rows per thread of the panel QR for a padded dimension ld
inline int sb_rows(int ld) {
  return ld <= 160 ? 9 : (ld <= 288 ? 17 : (ld <= 416 ? 25 : (ld <= 592 ? 36 : (ld <= 800 ? 49 : 75))));
}

// double2 of the panel QR's work arrays (red, rowj, pvw)
__host__ __device__ inline int sb_qr_work(int mr) { return 2 * 8 * 16 + 2 * 16 + 16 * mr; }
// V [mmax][16] (unless in global memory); then Y [mmax][16] in shared
// memory, or (Y in global memory) the panel QR's work arrays after the
// T/M/P/tau block (ld = 800: 231 KB)
__host__ __device__ inline size_t sb_smem_bytes(int ld, int mr, bool yg, bool vg) {
  const int mmax = ld - kNB;
  return sizeof(double2) * ((vg ? 0 : (size_t)mmax * kNB) + (yg ? (size_t)sb_qr_work(mr) : (size_t)mmax * kNB) +
                            3 * kNB * 17 + kNB);
}

// Householder QR of the m x 16 panel (rows r0.. of columns c0..c0+15 of A)
// and its compact WY factor T; leaves R and the reflectors in A (LAPACK
// layout: R on and above the diagonal, v below it) and the explicit V (unit
// diagonal, zeros above) in shared memory. Thread (column c = tid % 16,
// row group g = tid / 16) holds rows g, g + 16, ... of column c in registers.
// Per column j one CTA-wide reduction of one value per thread, the same
// product for every column, sum_{r > j} conj(a_j[r]) a_c[r]: for c > j it
// gives v^H a_c once the reflector's scale is known, for c = j the norm
// |x|^2, for c < j (conjugated) the dot v_c^H v_j of the T column (zlarft).
// The two row groups of a warp are summed with one shuffle, the eight warps'
// sums in shared memory. The update of the columns has one form for every
// column, a_c[r] -= a_j[r] s_c (s_c = scal w_c for c > j, else 0), so that the lanes
// of a warp do not diverge; the columns keep a_c unscaled and become v_c = scal a_c at
// the end (a_c - a_c (1 - scal) in the common update lost eps |A| of v_c, all of it at
// |A| = 1e16; 296 matrices of n = 274 5.17 -> 5.25 ms, 148 of n = 401 7.48 -> 7.43, of
// n = 570 17.2 -> 17.5). Rows go four at a time (slots past the panel hold zeros), so
// that four loads of the pivot column and four chains are in flight: with a check per
// row the two warps of a scheduler waited for one load after another at large n. The
// pivot column reaches the threads of a row group through the warp's own shared-memory
// buffer (the group's 16 threads share a warp). red/rowj: [2][8][16] / [2][16]; pvw
// [8][2][MR]; dsm [16][16]; tsm, ssm (scales) [16]; T [16][17].
// With VS (V in shared memory) the panel passes through V on its way between
// global memory and the registers, so that a warp reads and writes 32 consecutive
// rows of a column there; straight from the registers every access touches 16
// columns (14 k cycles a panel, with T, at n = 274; 8 k now).
template <int MR, bool VS>
__device__ void panel_qr(double2* __restrict__ A, int ld, int c0, int r0, int m, double2* V, double2* T,
                         double2* red, double2* rowj, double2* pvw, double2* dsm, double2* tsm, double2* ssm) {
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int c = tid & 15, g = tid >> 4;
  const int Mt = m / kNB;  // m is a multiple of 16: row slots t < Mt are inside the panel
  double2* pv = pvw + (size_t)wid * 2 * MR + (g & 1) * MR;  // this group's pivot buffer
  double2 col[MR];
  double2* Ap = A + (size_t)c0 * ld + r0;  // element (r, c) of the panel at Ap[c ld + r]
  if (VS) {
#pragma unroll 2
    for (int cc = wid; cc < kNB; cc += kNW)
#pragma unroll 4
      for (int r = lane; r < m; r += 32) V[pidx(r, cc)] = Ap[(size_t)cc * ld + r];
    __syncthreads();
  }
#pragma unroll
  for (int t = 0; t < MR; ++t) {
    const int r = g + 16 * t;
    col[t] = t < Mt ? (VS ? V[pidx(r, c)] : Ap[(size_t)c * ld + r]) : make_double2(0, 0);
  }
  // the group's rows of column 0 become the first pivot
  if (c == 0) {
#pragma unroll
    for (int t = 0; t < MR; ++t) pv[t] = col[t];
  }
  __syncwarp();
  for (int j = 0; j < kNB; ++j) {
    const int buf = j & 1;
    // ---- partial sums over this thread's rows r > j (four chains)
    double2 sum[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) sum[u] = make_double2(0, 0);
    if (g > j) cfmac(sum[0], pv[0], col[0]);
#pragma unroll
    for (int t0 = 0; t0 < MR; t0 += 4) {
      if (t0 < Mt) {
        double2 aj[4];
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (t0 + u > 0 && t0 + u < MR) aj[u] = pv[t0 + u];
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (t0 + u > 0 && t0 + u < MR) cfmac(sum[u], aj[u], col[t0 + u]);
      }
    }
    double2 acc = cadd(cadd(sum[0], sum[1]), cadd(sum[2], sum[3]));
    acc.x += __shfl_xor_sync(0xffffffffu, acc.x, 16);
    acc.y += __shfl_xor_sync(0xffffffffu, acc.y, 16);
    if (lane < 16) red[(buf * 8 + wid) * 16 + c] = acc;
    if (g == j) rowj[buf * 16 + c] = col[0];  // row j = row group j, slot 0
    __syncthreads();
    double2 tq[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) tq[q] = red[(buf * 8 + q) * 16 + c];
    const double2 tot = cadd(cadd(cadd(tq[0], tq[1]), cadd(tq[2], tq[3])), cadd(cadd(tq[4], tq[5]), cadd(tq[6], tq[7])));
    const double xn = __shfl_sync(0xffffffffu, tot.x, (lane & 16) | j);  // column j's own sum
    const double2 alpha = rowj[buf * 16 + j], rj = rowj[buf * 16 + c];
    const Refl R = make_refl(alpha, xn);
    // w_c = conj(tau) v^H a_c (v = (1; scal a_j)); a_c -= v w_c
    const double2 w = cmul(cconj(R.tau), cadd(rj, cmulc(R.scal, tot)));
    const double2 sc = cmul(R.scal, w);
    const long long up = c > j ? ~0ll : 0ll;  // a mask, so that no branch goes around the products
    const double2 sw = make_double2(__longlong_as_double(__double_as_longlong(sc.x) & up),
                                    __longlong_as_double(__double_as_longlong(sc.y) & up));
    if (g > j) cfms(col[0], pv[0], sw);
#pragma unroll
    for (int t0 = 0; t0 < MR; t0 += 4) {
      if (t0 < Mt) {
        double2 aj[4];
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (t0 + u > 0 && t0 + u < MR) aj[u] = pv[t0 + u];
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (t0 + u > 0 && t0 + u < MR) cfms(col[t0 + u], aj[u], sw);
      }
    }
    if (g == j) col[0] = c > j ? csub(col[0], w) : (c == j ? make_double2(R.beta, 0.0) : col[0]);
    if (g == 2 && c < j) dsm[j * 16 + c] = cadd(cconj(rj), cmul(R.scal, cconj(tot)));  // v_c^H v_j / conj(scal_c)
    if (tid == 64) tsm[j] = R.tau;
    if (tid == 96) ssm[j] = R.scal;
    // the next pivot column reaches the group through the warp's buffer
    __syncwarp();
    if (j + 1 < kNB && c == j + 1) {
#pragma unroll
      for (int t = 0; t < MR; ++t)
        if ((t & ~3) < Mt) pv[t] = col[t];
    }
    __syncwarp();
  }
  __syncthreads();
  if (c < g) dsm[g * 16 + c] = cmulc(ssm[c], dsm[g * 16 + c]);
  // R and the reflectors back in place (band and back-transform); V explicit
  // (unit diagonal, zeros above it)
  if (VS) {
#pragma unroll
    for (int t = 0; t < MR; ++t)
      if (t < Mt) V[pidx(g + 16 * t, c)] = col[t];
    __syncthreads();
#pragma unroll 2
    for (int cc = wid; cc < kNB; cc += kNW) {
      const double2 own = ssm[cc];
#pragma unroll 4
      for (int r = lane; r < m; r += 32) {
        const double2 v = V[pidx(r, cc)], x = r > cc ? cmul(v, own) : v;
        V[pidx(r, cc)] = x;
        Ap[(size_t)cc * ld + r] = x;
      }
    }
    __syncthreads();
    if (g <= c) V[pidx(g, c)] = make_double2(g == c ? 1.0 : 0.0, 0.0);
  } else {
#pragma unroll
    for (int t = 0; t < MR; ++t) {
      const int r = g + 16 * t;
      if (t < Mt) {
        const double2 v = r > c ? cmul(col[t], ssm[c]) : col[t];
        Ap[(size_t)c * ld + r] = v;
        V[pidx(r, c)] = r < c ? make_double2(0, 0) : (r == c ? make_double2(1, 0) : v);
      }
    }
    __syncthreads();
  }
  // T[0:j, j] = -tau_j T[0:j, 0:j] (v_0 .. v_{j-1})^H v_j (zlarft), column after
  // column: lane i of warp 0 keeps row i, its two halves take every other term
  if (wid == 0) {
    const int i = lane & 15, h = lane >> 4;
    double2 row[kNB];
#pragma unroll
    for (int j = 0; j < kNB; ++j) {
      double2 p = make_double2(0, 0);
#pragma unroll
      for (int q = 0; q < kNB; ++q)
        if (q < j && (q & 1) == h) cfma(p, row[q], dsm[j * 16 + q]);
      p.x += __shfl_xor_sync(0xffffffffu, p.x, 16);
      p.y += __shfl_xor_sync(0xffffffffu, p.y, 16);
      const double2 tj = tsm[j];
      row[j] = i < j ? cmul(make_double2(-tj.x, -tj.y), p) : (i == j ? tj : make_double2(0, 0));
      if (h == 0) T[i * 17 + j] = row[j];
    }
  }
  __syncthreads();
}

// Y[m x 16] = A22 V: every warp owns 8-row blocks; the upper tiles of the
// Hermitian trailing block are read as conjugate transposes of the lower ones,
// the diagonal tiles (kept full) directly.
// PF: V in global memory, its fragments of column block J + 1 loaded while
// block J is multiplied
template <bool PF>
__device__ void pass_y(const double2* __restrict__ A, int ld, int r0, int Mt, const double2* V, double2* Y) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int gr = lane >> 2, gk = lane & 3;
  for (int I8 = wid; I8 < 2 * Mt; I8 += kNW) {
    const int I = I8 >> 1;
    const int row = r0 + 8 * I8 + gr;  // this lane's A row
    double cr[2][2], ci[2][2];
#pragma unroll
    for (int nb = 0; nb < 2; ++nb) cr[nb][0] = cr[nb][1] = ci[nb][0] = ci[nb][1] = 0.0;
    auto load_a = [&](int J, double2 (&f)[4]) {
#pragma unroll
      for (int kb = 0; kb < 4; ++kb) {
        const int col = r0 + 16 * J + 4 * kb + gk;
        if (I >= J)
          f[kb] = A[(size_t)col * ld + row];
        else
          f[kb] = cconj(A[(size_t)row * ld + col]);
      }
    };
    if (PF) {
      double2 a[4], an[4], bf[4][2], bfn[4][2];
      auto load_b = [&](int J, double2 (&f)[4][2]) {
#pragma unroll
        for (int kb = 0; kb < 4; ++kb)
#pragma unroll
          for (int nb = 0; nb < 2; ++nb) f[kb][nb] = V[pidx(16 * J + 4 * kb + gk, 8 * nb + gr)];
      };
      load_a(0, a);
      load_b(0, bf);
      for (int J = 0; J < Mt; ++J) {
        if (J + 1 < Mt) {
          load_a(J + 1, an);
          load_b(J + 1, bfn);
        }
#pragma unroll
        for (int kb = 0; kb < 4; ++kb)
#pragma unroll
          for (int nb = 0; nb < 2; ++nb) cmma(cr[nb], ci[nb], a[kb], bf[kb][nb]);
#pragma unroll
        for (int kb = 0; kb < 4; ++kb) {
          a[kb] = an[kb];
#pragma unroll
          for (int nb = 0; nb < 2; ++nb) bf[kb][nb] = bfn[kb][nb];
        }
      }
    } else {
      // the blocks J + kAhead, ... are on their way while J is multiplied
      constexpr int kAhead = 3;
      double2 a[kAhead + 1][4];
#pragma unroll
      for (int u = 0; u < kAhead; ++u)
        if (u < Mt) load_a(u, a[u]);
      for (int J0 = 0; J0 < Mt; J0 += kAhead + 1) {
#pragma unroll
        for (int u = 0; u <= kAhead; ++u) {
          const int J = J0 + u;
          if (J < Mt) {
            if (J + kAhead < Mt) load_a(J + kAhead, a[(u + kAhead) % (kAhead + 1)]);
#pragma unroll
            for (int kb = 0; kb < 4; ++kb)
#pragma unroll
              for (int nb = 0; nb < 2; ++nb)
                cmma(cr[nb], ci[nb], a[u][kb], V[pidx(16 * J + 4 * kb + gk, 8 * nb + gr)]);
          }
        }
      }
    }
#pragma unroll
    for (int nb = 0; nb < 2; ++nb)
#pragma unroll
      for (int i = 0; i < 2; ++i) Y[pidx(8 * I8 + gr, 8 * nb + 2 * gk + i)] = make_double2(cr[nb][i], ci[nb][i]);
  }
}

// A22 -= V X^H + X V^H on the lower 16 x 16 tiles (diagonal tiles in full).
__device__ void pass_u(double2* __restrict__ A, int ld, int r0, int Mt, const double2* V, const double2* X) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int gr = lane >> 2, gk = lane & 3;
  int I = 0, J = wid;
  while (I < Mt && J > I) {  // tile t = wid in lower-triangle order
    J -= I + 1;
    ++I;
  }
  double2 c[2][2][2], cn[2][2][2];
  auto addr = [&](int TI, int TJ, int rb, int nb, int i) {
    return (size_t)(r0 + 16 * TJ + 8 * nb + 2 * gk + i) * ld + (r0 + 16 * TI + 8 * rb + gr);
  };
  auto load_c = [&](int TI, int TJ, double2 (&f)[2][2][2]) {
#pragma unroll
    for (int rb = 0; rb < 2; ++rb)
#pragma unroll
      for (int nb = 0; nb < 2; ++nb)
#pragma unroll
        for (int i = 0; i < 2; ++i) f[rb][nb][i] = A[addr(TI, TJ, rb, nb, i)];
  };
  auto advance = [&](int& TI, int& TJ) {  // 8 tiles further in lower-triangle order
    TJ += kNW;
    while (TI < Mt && TJ > TI) {
      TJ -= TI + 1;
      ++TI;
    }
  };
  if (I < Mt) load_c(I, J, c);
  while (I < Mt) {
    int In = I, Jn = J;
    advance(In, Jn);
    if (In < Mt) load_c(In, Jn, cn);
    double cr[2][2][2], ci[2][2][2];
#pragma unroll
    for (int rb = 0; rb < 2; ++rb)
#pragma unroll
      for (int nb = 0; nb < 2; ++nb)
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          cr[rb][nb][i] = c[rb][nb][i].x;
          ci[rb][nb][i] = c[rb][nb][i].y;
        }
#pragma unroll
    for (int kb = 0; kb < 4; ++kb) {
      double2 vi[2], xi[2], vj[2], xj[2];
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        vi[q] = V[pidx(16 * I + 8 * q + gr, 4 * kb + gk)];
        xi[q] = X[pidx(16 * I + 8 * q + gr, 4 * kb + gk)];
        vj[q] = V[pidx(16 * J + 8 * q + gr, 4 * kb + gk)];
        xj[q] = X[pidx(16 * J + 8 * q + gr, 4 * kb + gk)];
      }
#pragma unroll
      for (int rb = 0; rb < 2; ++rb)
#pragma unroll
        for (int nb = 0; nb < 2; ++nb) {
          cmma_sub_herm(cr[rb][nb], ci[rb][nb], vi[rb], xj[nb]);
          cmma_sub_herm(cr[rb][nb], ci[rb][nb], xi[rb], vj[nb]);
        }
    }
#pragma unroll
    for (int rb = 0; rb < 2; ++rb)
#pragma unroll
      for (int nb = 0; nb < 2; ++nb)
#pragma unroll
        for (int i = 0; i < 2; ++i) A[addr(I, J, rb, nb, i)] = make_double2(cr[rb][nb][i], ci[rb][nb][i]);
    I = In;
    J = Jn;
#pragma unroll
    for (int rb = 0; rb < 2; ++rb)
#pragma unroll
      for (int nb = 0; nb < 2; ++nb)
#pragma unroll
        for (int i = 0; i < 2; ++i) c[rb][nb][i] = cn[rb][nb][i];
  }
}

}  // namespace

// Load of Y in global memory kept in program order: with plain loads the
// compiler hoists the rows' loads of the Y T and P passes far enough ahead to
// spill ~4 KB of the stage's registers
__device__ __forceinline__ double2 ld_ordered(const double2* p) {
  double2 v;
  asm volatile("ld.global.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p) : "memory");
  return v;
}
template <bool KYG>
__device__ __forceinline__ double2 ldy(const double2* p) {
  return KYG ? ld_ordered(p) : *p;
}

// KYG: Y in the item's work area of the reflector buffer (ld > kSmemLd);
// KVG: V there too (ld > kVSmemLd)
// OCC: CTAs per SM
template <int MR, bool KYG, bool KVG = false, int OCC = 1>
__global__ void __launch_bounds__(kThr, OCC) sb_kernel(const EigItem* __restrict__ items, double2* __restrict__ hbuf,
                                                    double2* __restrict__ rbuf) {
  const EigItem it = items[blockIdx.x];
  const int ld = it.ld;
  const int tid = threadIdx.x;
  double2* A = hbuf + it.h_off;
  extern __shared__ __align__(16) unsigned char smraw[];
  const int mmax = ld - kNB;
  SbSmem S;
  double2* work = rbuf + it.r_off + band_off(ld);
  S.V = KVG ? work + (size_t)mmax * kNB : reinterpret_cast<double2*>(smraw);
  S.Y = KYG ? work : S.V + (size_t)mmax * kNB;
  S.T = KVG ? reinterpret_cast<double2*>(smraw) : (KYG ? S.V : S.Y) + (size_t)mmax * kNB;
  S.M = S.T + kNB * 17;
  S.P = S.M + kNB * 17;
  S.taus = S.P + kNB * 17;
  // the panel QR's work arrays: inside Y (free until Y = A V is formed;
  // 256 + 32 + 16 MR <= 16 mmax double2 for ld >= 96), or after taus
  S.part = KYG ? S.taus + kNB : S.Y;
  S.rowj = S.part + 2 * 8 * 16;
  S.pvw = S.rowj + 2 * 16;

  for (int c0 = 0; c0 + kNB < ld; c0 += kNB) {
    const int r0 = c0 + kNB, m = ld - r0, Mt = m / kNB;
    panel_qr<MR, !KVG>(A, ld, c0, r0, m, S.V, S.T, S.part, S.rowj, S.pvw, S.M, S.taus, S.P);
    // T into the free upper tile (rows c0.., columns r0..) for the back-transform
    for (int idx = tid; idx < kNB * kNB; idx += kThr) {
      const int i = idx % kNB, j = idx / kNB;
      A[(size_t)(r0 + j) * ld + c0 + i] = S.T[i * 17 + j];
    }
    // ---- Y = A22 V on the tensor cores
    pass_y<KVG>(A, ld, r0, Mt, S.V, S.Y);
    __syncthreads();
    // ---- X = Y T - 1/2 V (T^H V^H Y T) on the tensor cores. X1 = Y T in
    // place: a warp owns 8-row blocks of Y (A fragments: its rows; B: T);
    // the lanes' reads of a block end before its writes (__syncwarp)
    {
      const int lane = tid & 31, wid = tid >> 5, gr = lane >> 2, gk = lane & 3;
      for (int I8 = wid; I8 < 2 * Mt; I8 += kNW) {
        double cr[2][2] = {{0, 0}, {0, 0}}, ci[2][2] = {{0, 0}, {0, 0}};
#pragma unroll
        for (int kb = 0; kb < 4; ++kb) {
          const double2 a = ldy<KYG>(S.Y + pidx(8 * I8 + gr, 4 * kb + gk));
#pragma unroll
          for (int nb = 0; nb < 2; ++nb) cmma(cr[nb], ci[nb], a, S.T[(4 * kb + gk) * 17 + 8 * nb + gr]);
        }
        __syncwarp();
#pragma unroll
        for (int nb = 0; nb < 2; ++nb)
#pragma unroll
          for (int i = 0; i < 2; ++i) S.Y[pidx(8 * I8 + gr, 8 * nb + 2 * gk + i)] = make_double2(cr[nb][i], ci[nb][i]);
      }
      __syncthreads();
      // M = V^H X1: warp w computes the 8 x 8 block (w & 3) of M over one half
      // of the rows (w >> 2); the second half's partials pass through P (free
      // until P = T^H M) and are added by the first half's warps in a fixed
      // order
      {
        const int ib = (wid & 3) >> 1, jb = wid & 1, half = wid >> 2;
        double cr[2] = {0, 0}, ci[2] = {0, 0};
        for (int kb = half * 2 * Mt; kb < (half + 1) * 2 * Mt; ++kb) {
          const int k = 4 * kb + gk;
          const double2 a = cconj(ldy<KVG>(S.V + pidx(k, 8 * ib + gr)));
          const double2 b = ldy<KYG>(S.Y + pidx(k, 8 * jb + gr));
          cmma(cr, ci, a, b);
        }
        const int mi = 8 * ib + gr;
        if (half == 1) {
#pragma unroll
          for (int i = 0; i < 2; ++i) S.P[mi * 17 + 8 * jb + 2 * gk + i] = make_double2(cr[i], ci[i]);
        }
        __syncthreads();
        if (half == 0) {
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const double2 o = S.P[mi * 17 + 8 * jb + 2 * gk + i];
            S.M[mi * 17 + 8 * jb + 2 * gk + i] = make_double2(cr[i] + o.x, ci[i] + o.y);
          }
        }
      }
      __syncthreads();
      {  // P = T^H M
        const int i = tid / kNB, j = tid % kNB;
        double2 sacc = make_double2(0, 0);
        for (int k = 0; k <= i; ++k) sacc = cadd(sacc, cmulc(S.T[k * 17 + i], S.M[k * 17 + j]));
        S.P[i * 17 + j] = sacc;
      }
      __syncthreads();
      // X = X1 - 1/2 V P: each lane updates the entries of its own D fragment
      for (int I8 = wid; I8 < 2 * Mt; I8 += kNW) {
        double cr[2][2] = {{0, 0}, {0, 0}}, ci[2][2] = {{0, 0}, {0, 0}};
#pragma unroll
        for (int kb = 0; kb < 4; ++kb) {
          const double2 a = ldy<KVG>(S.V + pidx(8 * I8 + gr, 4 * kb + gk));
#pragma unroll
          for (int nb = 0; nb < 2; ++nb) cmma(cr[nb], ci[nb], a, S.P[(4 * kb + gk) * 17 + 8 * nb + gr]);
        }
#pragma unroll
        for (int nb = 0; nb < 2; ++nb)
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            double2* y = S.Y + pidx(8 * I8 + gr, 8 * nb + 2 * gk + i);
            const double2 x1 = ldy<KYG>(y);
            *y = make_double2(x1.x - 0.5 * cr[nb][i], x1.y - 0.5 * ci[nb][i]);
          }
      }
    }
    __syncthreads();
    // ---- A22 -= V X^H + X V^H on the tensor cores
    pass_u(A, ld, r0, Mt, S.V, S.Y);
    __syncthreads();
  }
}

// ------------------------------------------------------------------ stage 2
// Band storage Bd[c * kBandLd + d] = A(c + d, c), d = 0..31: the band and the
// bulge (a task reaches d = 31 at most), with kNB zero columns after the last
// one: a task that sticks out of the matrix works on zeros (its reflectors are
// zero there), so that no task checks a row or column.
//
// Task (s, j) (sweep s, step j, first row p = s + 1 + 16 j) applies reflector j
// of the sweep two-sidedly to its diagonal block D = A(p : p+16, p : p+16) and
// from the right to the block E = A(p+16 : p+32, p : p+16) below it; E's first
// column then gives reflector j + 1, applied to E from the left. It touches
// exactly the elements (r, c) with p <= c < p + 16 and c <= r < p + 32, plus
// column s when j = 0, so it meets sweep s - 1 only in that sweep's steps <= j + 1.
//
// Eight pairs of warps, pair = s mod 8, a D warp and an E warp each. Both publish
// their progress in shared-memory words (release) that other warps wait for
// (acquire, bounded by a time limit), in half steps:
//   D  reflector 0 formed (from column s, whose last writers are D(s-1, 0) and
//      the first half of E(s-1, 0)): 2 j + 1 = 1; D(s, j) done: 2 (j + 1)
//   E  E(s, j) H applied, reflector j + 1 formed: 2 j + 1; E(s, j) done: 2 (j + 1)
// D(s, j) needs E(s-1, j) and D(s-1, j+1); E(s, j) needs those and only the first
// half of E(s-1, j+1), of whose block it touches one element, the corner (first
// row and column) that is final then (tests/test_bulge_order.py holds every access of
// every task against these waits). Within a sweep D(s, j) waits for E's
// reflector, and E, before it writes a reflector slot, for D to have left it. No
// barrier of any kind between steps.
//
// Bound by latency: a sweep follows the one before it one and a half E tasks
// behind, so a matrix takes about 1.5 (ld - 1) E tasks, whatever the number of
// pairs. E is therefore kept short: all offsets relative to p are fixed per lane
// (one base address a step), sums are fused multiply-adds, a reflector takes one
// rsqrt and one reciprocal, both halves of the warp keep the first column so that
// its norm takes four shuffles, and the sweep's first reflector is D's work.
// Measured on a B200: 296 matrices of n = 274 2.31 -> 1.50 ms, 148 of n = 570
// (band in global memory) 4.84 -> 3.9 ms, against tasks that waited for whole
// tasks of the sweep before, with a barrier per step and checks of every row and
// column (1770 warp instructions a task, now 1000 with the polls).
constexpr int kBandLd = 2 * kNB;
constexpr int kMaxPairs = 8;             // sweeps in flight: one per pair of warps (a D and an E warp)
constexpr int kProgStride = 128;         // progress word: sweep * 128 + half steps done
// a reflector slot: entries 0..7 at 0, 8..15 at 9 (the two halves of a warp read
// them from different banks), tau at 17
constexpr int kSlot = 18;
__device__ __forceinline__ int vidx(int r) { return r + (r >> 3); }
constexpr long long kWaitNs = 2000000000LL;  // default limit of one wait

__host__ __device__ inline size_t band_double2(int ld) { return (size_t)(ld + kNB) * kBandLd; }
__host__ __device__ inline size_t sbtrd_smem_bytes(int ld, int pairs, bool bg) {
  return sizeof(double2) * ((bg ? 0 : band_double2(ld)) + pairs * 4 * kSlot) + sizeof(int) * (2 * pairs + 4);
}

__device__ __forceinline__ int ld_acquire_shared(const int* p) {
  int v;
  asm volatile("ld.acquire.cta.shared::cta.b32 %0, [%1];"
               : "=r"(v)
               : "r"((unsigned)__cvta_generic_to_shared(p))
               : "memory");
  return v;
}
__device__ __forceinline__ void st_release_shared(int* p, int v) {
  asm volatile("st.release.cta.shared::cta.b32 [%0], %1;" ::"r"((unsigned)__cvta_generic_to_shared(p)), "r"(v)
               : "memory");
}
__device__ __forceinline__ long long global_ns() {
  long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Waits until *flag >= need: kSpin polls at once, then one every ~kPollNs so
// that a waiting warp leaves the issue slots to the warps that work. Gives up,
// and sets *err, after limit_ns, after 2^28 polls, or at once when another warp
// has given up already.
constexpr unsigned kPollNs = 40;
constexpr int kSpin = 1;
__device__ __forceinline__ void wait_progress(const int* flag, int need, int* err, long long limit_ns) {
#pragma unroll 1
  for (int k = 0; k < kSpin; ++k)
    if (ld_acquire_shared(flag) >= need) return;
  if (*reinterpret_cast<volatile int*>(err)) return;
  const long long t0 = global_ns();
  for (int k = 1; k < (1 << 28); ++k) {
    __nanosleep(kPollNs);
    if (ld_acquire_shared(flag) >= need) return;
    if ((k & 63) == 0) {
      if (*reinterpret_cast<volatile int*>(err)) return;
      if (global_ns() - t0 > limit_ns) break;
    }
  }
  atomicExch(err, 1);
}
__device__ __forceinline__ void publish(int* flag, int v, int lane) {
  __syncwarp();
  if (lane == 0) {
    __threadfence_block();
    st_release_shared(flag, v);
  }
}

__device__ __forceinline__ double2 shfl2(double2 v, int src) {
  return make_double2(__shfl_sync(0xffffffffu, v.x, src), __shfl_sync(0xffffffffu, v.y, src));
}
__device__ __forceinline__ void add_halves(double2& v) {
  v.x += __shfl_xor_sync(0xffffffffu, v.x, 16);
  v.y += __shfl_xor_sync(0xffffffffu, v.y, 16);
}

// KBG: the band in the item's work area of the reflector buffer (ld >
// kSmemLd; a CTA-private region, so the same CTA-scope ordering as in shared
// memory applies)
template <int kPairs, bool KBG>
__global__ void __launch_bounds__(64 * kPairs, kMaxPairs / kPairs) sbtrd_kernel(const EigItem* __restrict__ items,
                                                        const double2* __restrict__ hbuf, double2* __restrict__ rbuf) {
  constexpr int kS2Thr = 64 * kPairs, kS2W = kS2Thr / 32;
  const EigItem it = items[blockIdx.x];
  const int ld = it.ld;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const double2* A = hbuf + it.h_off;
  double2* R = rbuf + it.r_off;
  extern __shared__ __align__(16) unsigned char smraw[];
  double2* Bd = KBG ? R + band_off(ld) : reinterpret_cast<double2*>(smraw);
  // [pair][2][kSlot]: v (v_0 = 1), tau of the pair's next steps
  double2* slots = KBG ? reinterpret_cast<double2*>(smraw) : Bd + band_double2(ld);
  double2* wsm = slots + kPairs * 2 * kSlot;                 // [warp][kSlot]: a vector broadcast in the warp
  int* prog_d = reinterpret_cast<int*>(wsm + kS2W * kSlot);  // [pair]: progress of the D and E warps
  int* prog_e = prog_d + kPairs;
  int* err = prog_e + kPairs;                                // a wait gave up
  for (int idx = tid; idx < (ld + kNB) * kBandLd; idx += kS2Thr) {
    const int c = idx / kBandLd, d = idx % kBandLd;
    Bd[idx] = (d <= kNB && c + d < ld) ? A[(size_t)c * ld + c + d] : make_double2(0, 0);
  }
  if (tid < 2 * kPairs) prog_d[tid] = -1;
  if (tid == 0) *err = 0;
  __syncthreads();
  const int i = lane & 15, h = lane >> 4;
  const int pair = wid >> 1;
  // E (bulge) warp, else D (diagonal block) warp: in every other two pairs the roles
  // are swapped, so that each of the four schedulers (warp mod 4) has two E warps
  const bool ewarp = ((wid ^ (pair >> 1)) & 1) != 0;
  double2* wv = wsm + wid * kSlot;
  double2* sl = slots + pair * 2 * kSlot;
  const long long limit = it.wait_ns > 0 ? it.wait_ns : kWaitNs;
  // offsets from Bd + p kBandLd. D element (i, 8h + cc): on or below the diagonal
  // at column 8h + cc, above it the conjugate at column i; up: bit cc set where above
  int doff[8];
  unsigned up = 0;
#pragma unroll
  for (int cc = 0; cc < 8; ++cc) {
    const int c = 8 * h + cc;
    doff[cc] = c <= i ? c * (kBandLd - 1) + i : i * (kBandLd - 1) + c;
    if (c > i) up |= 1u << cc;
  }
  // E element (i, 8h + cc) at e_off + cc (kBandLd - 1); (8h + rr, column i) at t_off + rr, for
  // i = 0 column 1 again: column 0 is final there, and the next sweep may be writing its corner
  const int e_off = 8 * h * (kBandLd - 1) + kNB + i;
  const int t_off = max(i, 1) * (kBandLd - 1) + kNB + 8 * h;
  for (int s = pair; s <= ld - 2; s += kPairs) {
    const int ns = sweep_steps(ld, s), nprev = s > 0 ? sweep_steps(ld, s - 1) : 0;
    const int base = s * kProgStride, pbase = (s - 1) * kProgStride, pp = (s - 1) & (kPairs - 1);
    // this pair's previous sweep is finished
    const int own_done = s >= kPairs ? base - kPairs * kProgStride + 2 * sweep_steps(ld, s - kPairs) : INT_MIN;
    const bool stuck = it.wait_fault && s == 1;
    double2* Rs = R + sweep_first(ld, s) * kNB;
    double2* B = Bd + (size_t)(s + 1) * kBandLd;  // column p
    if (!ewarp) {
      // ---- reflector 0 from column s (rows s + 1 .. s + 16), which becomes
      // (beta, 0, ...): nothing reads it again before the tridiagonal is extracted
      if (s > 0) {
        wait_progress(&prog_e[pp], stuck ? INT_MAX : pbase + 1, err, limit);
        wait_progress(&prog_d[pp], pbase + 2, err, limit);
      }
      wait_progress(&prog_e[pair], own_done, err, limit);
      double2* cs = B - kBandLd + 1;
      const double2 xi = cs[i];
      const double xx = sum16(i >= 1 ? fma(xi.x, xi.x, xi.y * xi.y) : 0.0);
      const Refl Rf = make_refl(cs[0], xx);
      __syncwarp();
      if (h == 0) {
        const double2 v = i == 0 ? make_double2(1, 0) : cmul(xi, Rf.scal);
        sl[vidx(i)] = v;
        if (i == 0) sl[17] = Rf.tau;
        Rs[i] = i == 0 ? Rf.tau : v;
        cs[i] = make_double2(i == 0 ? Rf.beta : 0.0, 0.0);
      }
      publish(&prog_d[pair], base + 1, lane);
    }
    for (int j = 0; j < ns; ++j, B += kNB * kBandLd) {
      const double2* vsrc = sl + (j & 1) * kSlot;
      if (!ewarp) {
        // ---- D <- H^H D H: lane (row i, half h)
        if (s > 0) {
          wait_progress(&prog_e[pp], pbase + 2 * min(j + 1, nprev), err, limit);
          wait_progress(&prog_d[pp], pbase + 2 * min(j + 2, nprev), err, limit);
        }
        if (j > 0) wait_progress(&prog_e[pair], base + 2 * j - 1, err, limit);
        const double2 tau = vsrc[17], vi = vsrc[vidx(i)];
        double2 vc[8], d[8];
#pragma unroll
        for (int cc = 0; cc < 8; ++cc) {
          vc[cc] = vsrc[9 * h + cc];
          d[cc] = B[doff[cc]];
          if (up & (1u << cc)) d[cc].y = -d[cc].y;
        }
        double2 y = make_double2(0, 0), y1 = make_double2(0, 0);
#pragma unroll
        for (int cc = 0; cc < 8; cc += 2) {
          cfma(y, d[cc], vc[cc]);
          cfma(y1, d[cc + 1], vc[cc + 1]);
        }
        y = cadd(y, y1);
        add_halves(y);
        // v^H y = v^H D v is real; w = tau y - 1/2 |tau|^2 (v^H y) v
        const double vy = sum16(fma(vi.x, y.x, vi.y * y.y));
        const double al = -0.5 * fma(tau.x, tau.x, tau.y * tau.y) * vy;
        double2 w = cscale(vi, al);
        cfma(w, tau, y);
        if (h == 0) wv[vidx(i)] = w;
        __syncwarp();
#pragma unroll
        for (int cc = 0; cc < 8; ++cc) {
          cfmsc(d[cc], vi, wv[9 * h + cc]);
          cfmsc(d[cc], w, vc[cc]);
          if (!(up & (1u << cc))) B[doff[cc]] = d[cc];
        }
        publish(&prog_d[pair], base + 2 * (j + 1), lane);
      } else if (j + 1 < ns) {
        // ---- E <- E H, then the next reflector from its first column and
        // E(:, 1:) <- H2^H E(:, 1:); the sweep's last step has no E
        if (s > 0) {
          wait_progress(&prog_d[pp], pbase + 2 * min(j + 2, nprev), err, limit);
          wait_progress(&prog_e[pp], stuck ? INT_MAX : pbase + min(2 * j + 3, 2 * nprev), err, limit);
        }
        // D has formed reflector 0; D has left the slot of reflector j + 1
        wait_progress(&prog_d[pair], base + max(1, 2 * j), err, limit);
        double2* Eb = B + e_off;
        double2 vc[8], e[8];
#pragma unroll
        for (int cc = 0; cc < 8; ++cc) {
          e[cc] = Eb[cc * (kBandLd - 1)];
          vc[cc] = vsrc[9 * h + cc];
        }
        const double2 tau = vsrc[17];
        double2 u = make_double2(0, 0), u1 = make_double2(0, 0);
#pragma unroll
        for (int cc = 0; cc < 8; cc += 2) {
          cfma(u, e[cc], vc[cc]);
          cfma(u1, e[cc + 1], vc[cc + 1]);
        }
        u = cadd(u, u1);
        add_halves(u);
        const double2 tu = cmul(tau, u);  // E(i, c) -= tau u_i conj(v_c)
        cfmsc(e[0], tu, vc[0]);
        // the first column x in both halves
        const double2 x = shfl2(e[0], i);
        const double xx = sum16(i >= 1 ? fma(x.x, x.x, x.y * x.y) : 0.0);
        const Refl Rf = make_refl(shfl2(x, 0), xx);
#pragma unroll
        for (int cc = 1; cc < 8; ++cc) cfmsc(e[cc], tu, vc[cc]);
        double2* nx = sl + ((j + 1) & 1) * kSlot;
        if (h == 0) {
          const double2 v2 = i == 0 ? make_double2(1, 0) : cmul(x, Rf.scal);
          nx[vidx(i)] = v2;
          if (i == 0) nx[17] = Rf.tau;
          Rs[(j + 1) * kNB + i] = i == 0 ? Rf.tau : v2;
          e[0] = make_double2(i == 0 ? Rf.beta : 0.0, 0.0);
        }
#pragma unroll
        for (int cc = 0; cc < 8; ++cc) Eb[cc * (kBandLd - 1)] = e[cc];
        publish(&prog_e[pair], base + 2 * j + 1, lane);
        // lane (column i, rows 8h ..)
        double2* Et = B + t_off;
        double2 col[8], v2r[8];
#pragma unroll
        for (int rr = 0; rr < 8; ++rr) {
          col[rr] = Et[rr];
          v2r[rr] = nx[9 * h + rr];
        }
        double2 z = make_double2(0, 0), z1 = make_double2(0, 0);
#pragma unroll
        for (int rr = 0; rr < 8; rr += 2) {
          cfmac(z, v2r[rr], col[rr]);
          cfmac(z1, v2r[rr + 1], col[rr + 1]);
        }
        z = cadd(z, z1);
        add_halves(z);
        const double2 tz = cmulc(Rf.tau, z);
        if (i > 0) {
#pragma unroll
          for (int rr = 0; rr < 8; ++rr) {
            cfms(col[rr], v2r[rr], tz);
            Et[rr] = col[rr];
          }
        }
        publish(&prog_e[pair], base + 2 * (j + 1), lane);
      } else {
        // both slots of the pair are free when E and D report the sweep finished
        publish(&prog_e[pair], base + 2 * (j + 1), lane);
      }
    }
  }
  __syncthreads();
  // tridiagonal T after the reflectors above: d real, e real (beta); the
  // unused e[ld - 1] carries the wait status (1: a wait gave up)
  double* de = reinterpret_cast<double*>(R + ceil_sum(ld - 1) * kNB);
  for (int c = tid; c < ld; c += kS2Thr) {
    de[c] = Bd[(size_t)c * kBandLd].x;
    de[ld + c] = c + 1 < ld ? Bd[(size_t)c * kBandLd + 1].x : (*err ? 1.0 : 0.0);
  }
}

// --------------------------------------------------------- tridiagonal stage
// Bisection (pmx_trieig.cuh) with 256 threads per matrix, 256 / nval probes per
// eigenvalue and round: bound by the FP64 pipe with two or more CTAs per SM, by the
// row-to-row chain of the Sturm sequence (8 cycles) below. The eigenvectors are a
// kernel of their own, because one thread per vector works there, for which 256
// threads and their registers would leave the SM empty: 64 threads a matrix, with
// the factors and iterates in global memory (in shared memory, one CTA per SM: the
// same up to 148 matrices, 3-5 % slower solver beyond). Measured on a B200 against
// one kernel with divisions in the Sturm chain, one thread per eigenvalue cluster
// and four factor arrays: 296 matrices of n = 274 with 17 vectors 0.67 -> 0.12 +
// 0.21 ms, 148 of n = 570 with 25 vectors 2.37 -> 0.17 + 0.44 ms.
constexpr int kTriThr = 256, kTriVecThr = 64;

inline size_t tri_smem_bytes(int n, int nval) {
  return sizeof(double) * ((size_t)3 * n + 8 + 3 * nval + kTriThr) + sizeof(int) * (kTriThr + 4);
}
inline size_t tri_vec_smem_bytes(int n, int nvec) {
  return sizeof(double) * ((size_t)2 * n + 8 + 2 * nvec) + sizeof(int) * ((size_t)nvec + 8);
}

// T of an item: d [n] and e [n] into shared memory; false when the bulge chase
// gave up a wait (T is incomplete)
__device__ __forceinline__ bool load_tri(const EigItem& it, const double2* rbuf, double* d, double* e) {
  const int n = it.n, ld = it.ld;
  const double* de = reinterpret_cast<const double*>(rbuf + it.r_off + ceil_sum(ld - 1) * kNB);
  for (int c = threadIdx.x; c < n; c += blockDim.x) {
    d[c] = de[c];
    e[c] = c + 1 < n ? de[ld + c] : 0.0;
  }
  __syncthreads();
  return de[2 * ld - 1] == 0.0;
}

__global__ void __launch_bounds__(kTriThr) tri_val_kernel(const EigItem* __restrict__ items,
                                                     const double2* __restrict__ rbuf, double* __restrict__ wbuf,
                                                     int* __restrict__ info) {
  const EigItem it = items[blockIdx.x];
  const int n = it.n, nval = it.nval;
  extern __shared__ __align__(16) unsigned char smraw[];
  double* d = reinterpret_cast<double*>(smraw);
  double* e = d + n;
  double* e2 = e + n;
  double* red = e2 + n;
  double* lam = red + 8;
  double* lo = lam + nval;
  double* hi = lo + nval;
  double* xs = hi + nval;
  int* cnt = reinterpret_cast<int*>(xs + kTriThr);
  if (!load_tri(it, rbuf, d, e)) {
    if (threadIdx.x == 0) info[blockIdx.x] = 3;
    return;
  }
  const TriWork tw{d, e, e2, red, lam, lo, hi, xs, cnt, nullptr, nullptr};
  const int status = tri_eigvals(tw, n, nval, wbuf + it.w_off, it.bisect_cap);
  if (threadIdx.x == 0) info[blockIdx.x] = status;
}

__global__ void __launch_bounds__(kTriVecThr) tri_vec_kernel(const EigItem* __restrict__ items,
                                                        const double2* __restrict__ rbuf,
                                                        const double* __restrict__ wbuf, double2* __restrict__ zbuf,
                                                        double* __restrict__ scratch, const int* __restrict__ info) {
  const EigItem it = items[blockIdx.x];
  const int n = it.n, nvec = it.want_vec ? it.nev : 0, tid = threadIdx.x;
  if (nvec <= 0 || info[blockIdx.x] != 0) return;
  extern __shared__ __align__(16) unsigned char smraw[];
  double* d = reinterpret_cast<double*>(smraw);
  double* e = d + n;
  double* red = e + n;
  double* lam = red + 8;
  double* rn = lam + nvec;
  int* clus = reinterpret_cast<int*>(rn + nvec);
  int* misc = clus + nvec + 1;
  load_tri(it, rbuf, d, e);
  // as tri_eigvals leaves T: its norm, negligible off-diagonals zero
  double tn = 0.0;
  for (int i = tid; i < n; i += kTriVecThr)
    tn = fmax(tn, fabs(d[i]) + (i > 0 ? fabs(e[i - 1]) : 0.0) + (i < n - 1 ? fabs(e[i]) : 0.0));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) tn = fmax(tn, __shfl_xor_sync(0xffffffffu, tn, o));
  if ((tid & 31) == 0) red[tid >> 5] = tn;
  __syncthreads();
  tn = fmax(red[0], red[1]);
  for (int i = tid; i < n - 1; i += kTriVecThr)
    if (fabs(e[i]) <= DBL_EPSILON * (fabs(d[i]) + fabs(d[i + 1]))) e[i] = 0.0;
  for (int k = tid; k < nvec; k += kTriVecThr) lam[k] = wbuf[it.w_off + k];
  if (tid == 0) red[3] = tn;
  __syncthreads();
  const TriWork tw{d, e, nullptr, red, lam, rn, nullptr, nullptr, nullptr, clus, misc};
  tri_eigvecs(tw, n, nvec, zbuf + it.z_off, scratch + it.s_off, blockIdx.x);
}

// ----------------------------------------------------------- back-transform
// Eigenvectors of T -> of the band. The bulge-chasing reflectors (s, j) act on
// rows s + 1 + 16 j .. + 15, and are applied with s descending; reflectors of one
// sweep act on disjoint rows, and (s, j) meets a later sweep's reflectors only at
// steps <= j. So the 16 sweeps of a group can be applied step by step, j
// ascending: block (S, j) = reflectors (S + 15 .. S, j), all inside the window of
// 32 rows from S + 16 j. One warp owns 32 / G vectors and keeps their window in
// registers, a vector's rows r = h (mod G) in the lane (vector, h); between
// blocks the window moves down 16 rows, so a row is read and written once per
// group instead of once per sweep (one CTA-wide barrier per sweep before).
// Everything is private to the warp: no barriers, vectors updated in place in
// global memory (G neighbouring rows of a vector are one contiguous piece), the
// next rows in registers and the next block's reflectors by cp.async meanwhile.
// Bound by the FP64 pipe (8 FMAs per entry of a reflector and vector) with 16
// warps per SM, by the latency of a reflector's sum and update (420 cycles) in
// small batches. G = 4 lanes per vector: where a reflector does not start on a
// multiple of 4, one entry more per lane meets a zero beside the staged reflector
// (19 % of the work; 6 % with G = 2), but twice the warps of G = 2 hide more of
// that latency and 24 vectors fill three warps: 0-4 % faster for 16 and 24 vectors
// on 148-1184 matrices. Measured on a B200 together with panel_back_kernel against
// one CTA per matrix with a barrier per sweep and panel columns on the CUDA cores:
// 296 matrices of n = 274 with 17 vectors 1.25 -> 0.97 ms (1184: 4.9 -> 2.8 ms),
// 148 of n = 570 with 25 vectors 6.1 -> 3.6 ms.
// ADJ applies Q2^H instead (the adjoint's resolvent): groups, steps and reflectors in
// the opposite order, with the conjugate of tau, the window moving up.
constexpr int kBackG = 16;     // sweeps per group
constexpr int kBackLanes = 4;  // lanes per vector

template <bool ADJ>
__global__ void __launch_bounds__(32, 16) band_back_kernel(const EigItem* __restrict__ items,
                                                      const double2* __restrict__ rbuf, double2* __restrict__ zbuf,
                                                      const int* __restrict__ info) {
  const EigItem it = items[blockIdx.x];
  const int n = it.n, ld = it.ld, nvec = it.want_vec ? it.nev : 0;
  constexpr int G = kBackLanes, kVec = 32 / G, kM = 32 / G, kHalf = kM / 2;
  constexpr int kSt = kNB + 2 * (G - 1);  // a staged reflector with its zeros
  const int k0 = blockIdx.y * kVec;
  if (k0 >= nvec || info[blockIdx.x] != 0) return;
  const int lane = threadIdx.x, h = lane % G, k = min(k0 + lane / G, nvec - 1);
  const bool own = k0 + lane / G < nvec;  // spare lanes repeat the last vector and store nothing
  const double2* R = rbuf + it.r_off;
  double2* z = zbuf + it.z_off + (size_t)k * n + h;
  __shared__ double2 sv[2 * kBackG * kSt];  // [2][16][kSt]: reflector entry q at G - 1 + q
  __shared__ double2 st[2 * kBackG];        // [2][16]: tau
  for (int i = lane; i < 2 * kBackG * kSt; i += 32)
    sv[i] = make_double2(i % kSt == G - 1 ? 1.0 : 0.0, 0.0);  // v_0 = 1, zeros on both sides
  __syncwarp();
  // reflectors (S + t, j) into buffer b; those past the end of their sweep as zero
  auto stage = [&](int b, int S, int j) {
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int t = 2 * u + (lane >> 4), q = lane & 15, s = S + t;
      const bool ok = s <= ld - 2 && j < sweep_steps(ld, s);
      const double2* src = R + (ok ? ((size_t)sweep_first(ld, s) + j) * kNB + q : 0);
      double2* dst = q == 0 ? st + b * kBackG + t : sv + (b * kBackG + t) * kSt + G - 1 + q;
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_addr(dst)), "l"(src), "r"(ok ? 16 : 0)
                   : "memory");
    }
    cp_async_commit();
  };
  auto load = [&](int r) { return r + h < n ? z[r] : make_double2(0, 0); };
  const int last = (ld - 2) / kBackG * kBackG;
  for (int g = 0; g <= last; g += kBackG) {
    const int S = ADJ ? g : last - g;
    const int nj = sweep_steps(ld, S);
    double2 w[kM];
    int p0 = ADJ ? S + kNB * (nj - 1) : S;  // first row of the window
    stage(0, S, ADJ ? nj - 1 : 0);
#pragma unroll
    for (int m = 0; m < kM; ++m) w[m] = load(p0 + G * m);
    for (int u = 0; u < nj; ++u, p0 += ADJ ? -kNB : kNB) {
      double2 wn[kHalf];
      if (u + 1 < nj) {
        stage((u + 1) & 1, S, ADJ ? nj - 2 - u : u + 1);
#pragma unroll
        for (int m = 0; m < kHalf; ++m) wn[m] = load(p0 + (ADJ ? -kNB : 2 * kNB) + G * m);
        cp_async_wait<1>();
      } else {
#pragma unroll
        for (int m = 0; m < kHalf; ++m) wn[m] = make_double2(0, 0);
        cp_async_wait<0>();
      }
      __syncwarp();
      const double2* v = sv + (u & 1) * kBackG * kSt + h + G - 1;
      const double2* tv = st + (u & 1) * kBackG;
#pragma unroll
      for (int tt = 0; tt < kBackG; ++tt) {
        // rows t + 1 .. t + 16 of the window: entry q = G m + h - (t + 1)
        const int t = ADJ ? tt : kBackG - 1 - tt;
        constexpr int kE = kNB / G + 1;
        const int m0 = (t + 1) / G, ne = (t + kNB) / G - m0 + 1;
        double2 ve[kE], d0 = make_double2(0, 0), d1 = make_double2(0, 0);
#pragma unroll
        for (int e = 0; e < kE; ++e) {
          if (e < ne) {
            ve[e] = v[t * kSt + G * (m0 + e) - (t + 1)];
            cfmac((e & 1) ? d1 : d0, ve[e], w[m0 + e]);
          }
        }
        double2 d = cadd(d0, d1);
#pragma unroll
        for (int o = 1; o < G; o <<= 1) {
          d.x += __shfl_xor_sync(0xffffffffu, d.x, o);
          d.y += __shfl_xor_sync(0xffffffffu, d.y, o);
        }
        d = ADJ ? cmulc(tv[t], d) : cmul(tv[t], d);
#pragma unroll
        for (int e = 0; e < kE; ++e)
          if (e < ne) cfms(w[m0 + e], ve[e], d);
      }
      __syncwarp();  // the staged reflectors have been read
      // the half of the window that this group is done with
#pragma unroll
      for (int m = 0; m < kHalf; ++m) {
        const int out = ADJ ? m + kHalf : m, r = p0 + G * out;
        if (own && r + h < n) z[r] = w[out];
        if (ADJ) {
          w[m + kHalf] = w[m];
          w[m] = wn[m];
        } else {
          w[m] = w[m + kHalf];
          w[m + kHalf] = wn[m];
        }
      }
    }
#pragma unroll
    for (int m = 0; m < kHalf; ++m) {
      const int out = ADJ ? m + kHalf : m, r = p0 + G * out;
      if (own && r + h < n) z[r] = w[out];
    }
  }
}

// element r of column i of a panel's explicit V (unit diagonal, zeros above;
// below the diagonal the reflectors that stage 1 left in place)
__device__ __forceinline__ double2 panel_v(const double2* __restrict__ vcol, int r, int i) {
  return r > i ? __ldg(vcol + r) : make_double2(r == i ? 1.0 : 0.0, 0.0);
}

// Eigenvectors of the band -> of H: the panels in reverse, Z[r0:] -= V (T (V^H
// Z[r0:])), on the FP64 tensor cores. One CTA per matrix and 8 NB vectors, which
// stay in shared memory; V is read straight from global memory as MMA fragments
// (each value twice per panel, by the CTAs of a matrix from L2). Per panel: V^H Z
// with the rows split over the warps and the partial sums added in a fixed order,
// T times that, and the update of the rows. Two to three CTAs per SM cover the
// three barriers and the load latency of a panel.
template <int NB>
__host__ __device__ constexpr int panel_ldz() { return 8 * NB + 2; }  // row stride free of bank conflicts
template <int NB>
inline size_t panel_back_smem(int ld) {
  return sizeof(double2) * ((size_t)ld * panel_ldz<NB>() + 2 * kNB * panel_ldz<NB>() + kNB * 17 + (kNW / NB) * kNB * 8 * NB);
}

// ADJ applies Q1^H: the panels forward, with T^H.
template <int NB, bool ADJ>
__global__ void __launch_bounds__(kThr, 2) panel_back_kernel(const EigItem* __restrict__ items,
                                                           const double2* __restrict__ hbuf,
                                                           double2* __restrict__ zbuf, const int* __restrict__ info) {
  const EigItem it = items[blockIdx.x];
  const int n = it.n, ld = it.ld, nvec = it.want_vec ? it.nev : 0;
  constexpr int kVec = 8 * NB, kLdz = panel_ldz<NB>(), kKG = kNW / NB;
  const int k0 = blockIdx.y * kVec;
  if (k0 >= nvec || info[blockIdx.x] != 0) return;
  const int nv = min(kVec, nvec - k0);
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, gr = lane >> 2, gk = lane & 3;
  const double2* A = hbuf + it.h_off;
  double2* zg = zbuf + it.z_off + (size_t)k0 * n;
  extern __shared__ __align__(16) unsigned char smraw[];
  double2* Z = reinterpret_cast<double2*>(smraw);  // [ld][kLdz]
  double2* W = Z + (size_t)ld * kLdz;              // [16][kLdz] V^H Z
  double2* W2 = W + kNB * kLdz;                    // [16][kLdz] T V^H Z
  double2* T = W2 + kNB * kLdz;                    // [16][17]
  double2* red = T + kNB * 17;                     // [kKG][16][kVec] partial sums
  for (int idx = tid; idx < ld * kVec; idx += kThr) {
    const int k = idx / ld, r = idx % ld;
    Z[r * kLdz + k] = k < nv && r < n ? zg[(size_t)k * n + r] : make_double2(0, 0);
  }
  const int nb = wid % NB, kg = wid / NB;  // this warp's vectors and share of the rows in V^H Z
  for (int pc = 0; pc <= ld - 2 * kNB; pc += kNB) {
    const int c0 = ADJ ? pc : ld - 2 * kNB - pc;
    const int r0 = c0 + kNB, m = ld - r0;
    const double2* Vp = A + (size_t)c0 * ld + r0;  // column i at Vp + i ld
    if (tid < kNB * kNB) {
      const int i = tid % kNB, j = tid / kNB;
      T[i * 17 + j] = __ldg(A + (size_t)(r0 + j) * ld + c0 + i);
    }
    __syncthreads();  // Z of the last panel (or the load), T
    {
      double cr[2][2] = {{0, 0}, {0, 0}}, ci[2][2] = {{0, 0}, {0, 0}};
      const double2* va = Vp + (size_t)gr * ld;
      const double2* vb = va + (size_t)8 * ld;
      const double2* zb = Z + (size_t)r0 * kLdz + 8 * nb + gr;
#pragma unroll 4
      for (int ks = kg; ks < m / 4; ks += kKG) {
        const int r = 4 * ks + gk;
        const double2 a0 = cconj(ks < 4 ? panel_v(va, r, gr) : __ldg(va + r));
        const double2 a1 = cconj(ks < 4 ? panel_v(vb, r, gr + 8) : __ldg(vb + r));
        const double2 b = zb[r * kLdz];
        cmma(cr[0], ci[0], a0, b);
        cmma(cr[1], ci[1], a1, b);
      }
#pragma unroll
      for (int x = 0; x < 2; ++x)
#pragma unroll
        for (int y = 0; y < 2; ++y)
          red[((kg * kNB) + 8 * x + gr) * kVec + 8 * nb + 2 * gk + y] = make_double2(cr[x][y], ci[x][y]);
    }
    __syncthreads();
    for (int idx = tid; idx < kNB * kVec; idx += kThr) {
      const int i = idx / kVec, k = idx % kVec;
      double2 s = red[i * kVec + k];
#pragma unroll
      for (int g = 1; g < kKG; ++g) s = cadd(s, red[(g * kNB + i) * kVec + k]);
      W[i * kLdz + k] = s;
    }
    __syncthreads();
    for (int idx = tid; idx < kNB * kVec; idx += kThr) {  // T upper triangular
      const int i = idx / kVec, k = idx % kVec;
      double2 s = make_double2(0, 0);
      if (ADJ)
        for (int q = 0; q <= i; ++q) cfmac(s, T[q * 17 + i], W[q * kLdz + k]);
      else
        for (int q = i; q < kNB; ++q) cfma(s, T[i * 17 + q], W[q * kLdz + k]);
      W2[i * kLdz + k] = s;
    }
    __syncthreads();
    double2 bw[4][NB];
#pragma unroll
    for (int kb = 0; kb < 4; ++kb)
#pragma unroll
      for (int x = 0; x < NB; ++x) {
        const double2 t = W2[(4 * kb + gk) * kLdz + 8 * x + gr];
        bw[kb][x] = make_double2(-t.x, -t.y);
      }
#pragma unroll 2
    for (int I = wid; I < m / 8; I += kNW) {
      const int r = 8 * I + gr;
      double2 a[4];
#pragma unroll
      for (int kb = 0; kb < 4; ++kb) {
        const double2* vc = Vp + (size_t)(4 * kb + gk) * ld;
        a[kb] = I < 2 ? panel_v(vc, r, 4 * kb + gk) : __ldg(vc + r);
      }
#pragma unroll
      for (int x = 0; x < NB; ++x) {
        double2* zp = Z + (size_t)(r0 + r) * kLdz + 8 * x + 2 * gk;
        const double2 z0 = zp[0], z1 = zp[1];
        double cr[2] = {z0.x, z1.x}, ci[2] = {z0.y, z1.y};
#pragma unroll
        for (int kb = 0; kb < 4; ++kb) cmma(cr, ci, a[kb], bw[kb][x]);
        zp[0] = make_double2(cr[0], ci[0]);
        zp[1] = make_double2(cr[1], ci[1]);
      }
    }
  }
  __syncthreads();
  for (int idx = tid; idx < nv * n; idx += kThr) {
    const int k = idx / n, r = idx % n;
    zg[(size_t)k * n + r] = Z[r * kLdz + k];
  }
}

template <int NB, bool ADJ>
cudaError_t launch_panel_back(const EigItem* items, int nitems, int ld, int max_nvec, const double2* hbuf,
                              double2* zbuf, const int* info, cudaStream_t st) {
  const size_t sm = panel_back_smem<NB>(ld);
  const cudaError_t e =
      cudaFuncSetAttribute(panel_back_kernel<NB, ADJ>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  if (e != cudaSuccess) return e;
  panel_back_kernel<NB, ADJ><<<dim3(nitems, (max_nvec + 8 * NB - 1) / (8 * NB)), kThr, sm, st>>>(items, hbuf, zbuf,
                                                                                              info);
  return cudaGetLastError();
}

// Q (or Q^H) on the vectors of every item
template <bool ADJ>
cudaError_t apply_q(const EigItem* items, int nitems, int ld, int max_nvec, const double2* hbuf, const double2* rbuf,
                    double2* zbuf, const int* info, cudaStream_t st) {
  constexpr int kVec = 32 / kBackLanes;
  const auto band = [&]() {
    band_back_kernel<ADJ><<<dim3(nitems, (max_nvec + kVec - 1) / kVec), 32, 0, st>>>(items, rbuf, zbuf, info);
    return cudaGetLastError();
  };
  // 16 vectors a CTA while two CTAs share an SM (ld <= 304), else 8
  const auto panels = [&]() {
    return max_nvec > 8 && panel_back_smem<2>(ld) <= 112 * 1024
               ? launch_panel_back<2, ADJ>(items, nitems, ld, max_nvec, hbuf, zbuf, info, st)
               : launch_panel_back<1, ADJ>(items, nitems, ld, max_nvec, hbuf, zbuf, info, st);
  };
  const cudaError_t e = ADJ ? panels() : band();
  return e != cudaSuccess ? e : (ADJ ? band() : panels());
}

// x <- -(T - lam_k)^-1 x for the complex vectors of every item, in place; eigenvalue
// lam_k of item b at lam[w_off + k]. Two threads per vector (real and imaginary
// part) share one factorisation.
constexpr int kShiftThr = 128;
__global__ void __launch_bounds__(kShiftThr) tri_shift_kernel(const EigItem* __restrict__ items,
                                                         const double2* __restrict__ rbuf,
                                                         const double* __restrict__ lam, double2* __restrict__ zbuf,
                                                         double* __restrict__ scratch) {
  const EigItem it = items[blockIdx.x];
  const int n = it.n, nvec = it.nev, tid = threadIdx.x;
  extern __shared__ __align__(16) unsigned char smraw[];
  double* d = reinterpret_cast<double*>(smraw);
  double* e = d + n;
  __shared__ double red[kShiftThr / 32];
  load_tri(it, rbuf, d, e);
  double tn = 0.0;
  for (int i = tid; i < n; i += kShiftThr)
    tn = fmax(tn, fabs(d[i]) + (i > 0 ? fabs(e[i - 1]) : 0.0) + (i < n - 1 ? fabs(e[i]) : 0.0));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) tn = fmax(tn, __shfl_xor_sync(0xffffffffu, tn, o));
  if ((tid & 31) == 0) red[tid >> 5] = tn;
  __syncthreads();
  tn = fmax(fmax(red[0], red[1]), fmax(red[2], red[3]));
  for (int i = tid; i < n - 1; i += kShiftThr)
    if (fabs(e[i]) <= DBL_EPSILON * (fabs(d[i]) + fabs(d[i + 1]))) e[i] = 0.0;
  __syncthreads();
  const double tiny = fmax(DBL_EPSILON * tn, 1e-290);
  const int ldv = tri_ldv(nvec);
  double* F = scratch + it.s_off;
  double* I0 = F + (size_t)n * ldv;
  for (int k = tid; k < nvec; k += kShiftThr) tri_factor(d, e, n, lam[it.w_off + k], tiny, F + k, I0 + k, ldv);
  __syncthreads();
  for (int x = tid; x < 2 * nvec; x += kShiftThr) {
    const int k = x >> 1;
    double* xb = reinterpret_cast<double*>(zbuf + it.z_off + (size_t)k * n) + (x & 1);
    tri_factored_solve(d, e, lam[it.w_off + k], F + k, I0 + k, ldv, n, xb, 2, -1.0);
  }
}

// ------------------------------------------------------------------- host
int heev2_ld(int n) { return (n + kNB - 1) / kNB * kNB; }

bool heev2_supported(int max_n) { return heev2_ld(max_n) >= 96 && heev2_ld(max_n) <= kMaxLd; }

size_t heev2_rbuf_double2(int ld, int launch_ld) {
  return (size_t)band_off(ld) + (launch_ld > kSmemLd ? band_double2(ld) : 0);
}

cudaError_t launch_heev2(const EigItem* items, int nitems, int max_n, int max_nval, int max_nvec, double2* hbuf,
                         double* wbuf, double2* zbuf, double* scratch, double2* rbuf, int* info, cudaStream_t st) {
  if (nitems <= 0) return cudaSuccess;
  if (!heev2_supported(max_n)) return cudaErrorInvalidValue;
  const int ld = heev2_ld(max_n);
  cudaError_t e;
  const int mr = sb_rows(ld);
  const bool big = ld > kSmemLd;  // Y and the band in the reflector buffer's work areas
  const size_t s1 = sb_smem_bytes(ld, mr, big, ld > kVSmemLd);
  // up to kSmallLd two CTAs per SM, although 128 registers spill a little, once there
  // are more matrices than SMs
  auto sb = mr == 9    ? (nitems > 148 ? sb_kernel<9, false, false, 2> : sb_kernel<9, false>)
            : mr == 17 ? sb_kernel<17, false>
            : mr == 25 ? sb_kernel<25, false>
            : mr == 36 ? sb_kernel<36, true>
            : mr == 49 ? sb_kernel<49, true>
                       : sb_kernel<75, true, true>;
  e = cudaFuncSetAttribute(sb, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)s1);
  if (e != cudaSuccess) return e;
  sb<<<nitems, kThr, s1, st>>>(items, hbuf, rbuf);
  // small matrices have at most ten steps a sweep, which four pairs of warps keep up
  // with: two CTAs per SM then, once there are more matrices than SMs
  // (measured with both: 1025 matrices of n = 113 3.89 -> 3.17 ms, 433 1.77 -> 1.57;
  // 122 with one CTA per SM 0.71, with the two-CTA kernels 0.77)
  const int pairs = ld <= kSmallLd && nitems > 148 ? 4 : kMaxPairs;
  const size_t s2 = sbtrd_smem_bytes(ld, pairs, big);
  auto tr = big ? sbtrd_kernel<8, true> : (pairs == 4 ? sbtrd_kernel<4, false> : sbtrd_kernel<8, false>);
  e = cudaFuncSetAttribute(tr, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)s2);
  if (e != cudaSuccess) return e;
  tr<<<nitems, 64 * pairs, s2, st>>>(items, hbuf, rbuf);
  const size_t s3 = tri_smem_bytes(max_n, max_nval);
  e = cudaFuncSetAttribute(tri_val_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)s3);
  if (e != cudaSuccess) return e;
  tri_val_kernel<<<nitems, kTriThr, s3, st>>>(items, rbuf, wbuf, info);
  if (max_nvec > 0) {
    const size_t s5 = tri_vec_smem_bytes(max_n, max_nvec);
    e = cudaFuncSetAttribute(tri_vec_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)s5);
    if (e != cudaSuccess) return e;
    tri_vec_kernel<<<nitems, kTriVecThr, s5, st>>>(items, rbuf, wbuf, zbuf, scratch, info);
  }
  e = cudaGetLastError();
  if (max_nvec > 0 && e == cudaSuccess) {
    e = apply_q<false>(items, nitems, ld, max_nvec, hbuf, rbuf, zbuf, info, st);
  }
  return e;
}

cudaError_t launch_heev2_resolvent(const EigItem* items, int nitems, int max_n, int max_nvec, const double2* hbuf,
                                   const double2* rbuf, const double* lam, double2* zbuf, double* scratch,
                                   const int* info, cudaStream_t st) {
  if (nitems <= 0 || max_nvec <= 0) return cudaSuccess;
  const int ld = heev2_ld(max_n);
  cudaError_t e = apply_q<true>(items, nitems, ld, max_nvec, hbuf, rbuf, zbuf, info, st);
  if (e != cudaSuccess) return e;
  tri_shift_kernel<<<nitems, kShiftThr, sizeof(double) * 2 * max_n, st>>>(items, rbuf, lam, zbuf, scratch);
  e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  return apply_q<false>(items, nitems, ld, max_nvec, hbuf, rbuf, zbuf, info, st);
}

}  // namespace dev
}  // namespace pmx
