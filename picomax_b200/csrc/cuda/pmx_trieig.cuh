// Eigenpairs of a real symmetric tridiagonal matrix T (diagonal d, off-diagonal
// e) by one CTA: multisection bisection on Sturm counts for the lowest nval
// eigenvalues, then inverse iteration with modified Gram-Schmidt inside
// eigenvalue clusters for the lowest nvec eigenvectors. Shared by the one-stage
// eigensolver (heev_kernel) and the tridiagonal stage of the two-stage one.
//
// LAPACK's dstebz / dstein (the tridiagonal stages behind Eigen's
// SelfAdjointEigenSolver results in the reference, src/pmx_epm.cpp:232) are
// the published methods restated here: Gershgorin interval, bisection on Sturm
// counts to 2 eps |lambda|, inverse iteration from a pseudo-random start.
#pragma once

#include <cfloat>
#include <cmath>

#include <cuda_runtime.h>

#include "pmx_common.cuh"

namespace pmx {
namespace dev {

constexpr int kTriBisectIters = 200;  // cap; multisection converges in ~14 rounds
constexpr int kTriInvIters = 3;

// Number of eigenvalues below x of a T scaled to norm 1 (d, and e2 the squares of
// the off-diagonals): sign changes of the Sturm sequence
//   p_i = (d_i - x) p_{i-1} - e_{i-1}^2 p_{i-2}
// itself, not of its ratios p_i / p_{i-1}: the ratios take a division per row, on
// the chain from row to row (90 cycles), the sequence one FMA (8). It is the exact
// sequence of a T whose entries differ by rounding errors of d - x and e^2, as the
// ratios are. Every 8 rows both running terms are scaled by a power of two, and the
// smaller one raised to 2^-200 of the larger (a change of d by less). In between they
// stay in range: a row grows them by 3 at most, and since d - x is zero or above 2^-100
// and e^2 zero or above 2^-172 (tri_snap, tri_eigvals) a row shrinks them by 1e-30 at
// most, two rows by 1e-52. Without this, a chain of d = x and tiny e ran into
// zeros. A zero counts as
// positive: its neighbours have opposite signs, so exactly one change is seen; only
// after a zero off-diagonal would it wipe out the rest, so with SPLIT (some e2 is
// zero) zeros are replaced by tiny values of the sign opposite to the last one.
template <bool SPLIT>
__device__ __forceinline__ int sturm_count(const double* d, const double* e2, int n, double x) {
  double p0 = 1.0, p1 = d[0] - x;
  if (SPLIT && p1 == 0.0) p1 = -1e-30;
  int c = (unsigned)__double2hiint(p1) >> 31;
  auto row = [&](int i) {
    const double t = e2[i - 1] * p0;
    double p2 = fma(d[i] - x, p1, -t);
    if (SPLIT && p2 == 0.0) p2 = -1e-30 * p1;
    c += (unsigned)(__double2hiint(p2) ^ __double2hiint(p1)) >> 31;
    p0 = p1;
    p1 = p2;
  };
  int i = 1;
  for (; i + 8 <= n; i += 8) {
#pragma unroll
    for (int u = 0; u < 8; ++u) row(i + u);
    // 2^-exponent of the larger one
    const int ex = max((__double2hiint(p0) >> 20) & 0x7ff, (__double2hiint(p1) >> 20) & 0x7ff);
    const double sc = __hiloint2double((2046 - min(max(ex, 1), 2045)) << 20, 0);
    p0 = copysign(fmax(fabs(p0 * sc), 0x1p-200), p0);
    p1 = copysign(fmax(fabs(p1 * sc), 0x1p-200), p1);
  }
  for (; i < n; ++i) row(i);
  return c;
}

// A value of the scaled T or a probe, rounded to a multiple of 2^-97 (if it is above
// 2^-48 it is one of 2^-100 already): far below the bisection's 2^-76.
__device__ __forceinline__ double tri_snap(double v) { return fabs(v) < 0x1p-48 ? (v + 0x1.8p-45) - 0x1.8p-45 : v; }

__device__ __forceinline__ double hash_uniform(unsigned long long a, unsigned long long b) {
  unsigned long long x = a * 0x9E3779B97F4A7C15ull ^ (b + 0x632BE59BD9B4E019ull);
  x ^= x >> 31;
  x *= 0xBF58476D1CE4E5B9ull;
  x ^= x >> 27;
  x *= 0x94D049BB133111EBull;
  x ^= x >> 31;
  return ((double)(x >> 11) * (1.0 / 9007199254740992.0)) * 2.0 - 1.0;  // (-1, 1)
}

// Shared-memory work arrays of the tridiagonal stage.
struct TriWork {
  double* d;     // [n] diagonal
  double* e;     // [n] off-diagonal (e[n-1] unused); negligible entries are zeroed
  double* e2;    // [n] squares of the scaled e
  double* red;   // [8] Gershgorin interval, |T|, T finite, some e2 zero
  double* lam;   // [nval] eigenvalues
  double* lo;    // [nval] bisection brackets
  double* hi;    // [nval]
  double* xs;    // [blockDim.x] multisection probes
  int* cnt;      // [blockDim.x] their Sturm counts
  int* clus;     // [nvec + 1] cluster starts
  int* misc;     // [4]
};

__device__ __forceinline__ int sturm_count(const TriWork& W, int n, double x, bool split) {
  return split ? sturm_count<true>(W.d, W.e2, n, x) : sturm_count<false>(W.d, W.e2, n, x);
}

// Lowest nval eigenvalues of T into lam[] and wout[]. Returns 0, 1 (bisection
// did not converge) or 2 (non-finite eigenvalue). Every thread of the block
// calls it; contains block barriers. blockDim.x must be a multiple of 32.
__device__ inline int tri_eigvals(const TriWork& W, int n, int nval, double* __restrict__ wout, int cap = 0) {
  const int iters = cap > 0 ? cap : kTriBisectIters;
  const int tid = threadIdx.x, nthr = blockDim.x;
  double *d = W.d, *e = W.e, *e2 = W.e2, *red = W.red, *lo = W.lo, *hi = W.hi, *xs = W.xs, *lam = W.lam;
  int* cnt = W.cnt;
  // Gershgorin interval and norm; a non-finite entry of T (fmin/fmax would
  // skip it) fails the matrix
  {
    double glo = DBL_MAX, ghi = -DBL_MAX, tn = 0.0;
    int fin = 1;
    for (int i = tid; i < n; i += nthr) {
      const double el = i > 0 ? fabs(e[i - 1]) : 0.0, er = i < n - 1 ? fabs(e[i]) : 0.0;
      fin &= (isfinite(d[i]) && isfinite(el) && isfinite(er)) ? 1 : 0;
      glo = fmin(glo, d[i] - el - er);
      ghi = fmax(ghi, d[i] + el + er);
      tn = fmax(tn, fabs(d[i]) + el + er);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      glo = fmin(glo, __shfl_xor_sync(0xffffffffu, glo, o));
      ghi = fmax(ghi, __shfl_xor_sync(0xffffffffu, ghi, o));
      tn = fmax(tn, __shfl_xor_sync(0xffffffffu, tn, o));
    }
    // per-warp results pass through xs (3 nthr / 32 <= nthr doubles)
    if ((tid & 31) == 0) {
      xs[3 * (tid >> 5)] = glo;
      xs[3 * (tid >> 5) + 1] = ghi;
      xs[3 * (tid >> 5) + 2] = tn;
    }
    fin = __syncthreads_and(fin);
    if (tid == 0) {
      for (int w = 1; w < nthr / 32; ++w) {
        glo = fmin(glo, xs[3 * w]);
        ghi = fmax(ghi, xs[3 * w + 1]);
        tn = fmax(tn, xs[3 * w + 2]);
      }
      red[0] = glo;
      red[1] = ghi;
      red[3] = tn;
      red[4] = fin;
    }
    __syncthreads();
  }
  const double tnorm = red[3];
  const bool finite_t = red[4] != 0.0;
  // negligible off-diagonals are zero; the counts work on T scaled by a power of two
  const int ex = finite_t && tnorm > 0.0 ? ilogb(tnorm) + 1 : 0;
  int split = 0;
  for (int i = tid; i < n - 1; i += nthr) {
    double v = e[i];
    if (fabs(v) <= DBL_EPSILON * (fabs(d[i]) + fabs(d[i + 1]))) e[i] = v = 0.0;
    v = scalbn(v, -ex);
    e2[i] = fabs(v) < 0x1p-86 ? 0.0 : v * v;
    split |= e2[i] == 0.0;
  }
  split = __syncthreads_or(split);
  for (int i = tid; i < n; i += nthr) d[i] = tri_snap(scalbn(d[i], -ex));
  const double pad = 2.0 * DBL_EPSILON * n + DBL_MIN;
  const double glo = scalbn(red[0], -ex) - pad, ghi = scalbn(red[1], -ex) + pad;
  // brackets end at 2 eps |lambda|, at least 2^-24 eps of the norm
  constexpr double kFloor = DBL_EPSILON / 16777216.0;
  auto tol_of = [&](double l, double h) { return 2.0 * DBL_EPSILON * fmax(fabs(l), fabs(h)) + kFloor; };
  // multisection: G threads per eigenvalue probe G interior points at once
  const int G = nval > 0 ? max(1, nthr / nval) : 1;
  __syncthreads();
  int converged = 0;
  if (nval > nthr) {
    // more eigenvalues than threads: plain bisection, each thread owns the
    // eigenvalues tid, tid + nthr, ...
    for (int k = tid; k < nval; k += nthr) {
      lo[k] = glo;
      hi[k] = ghi;
    }
    for (int iter = 0; iter < iters; ++iter) {
      int done = 1;
      for (int k = tid; k < nval; k += nthr) {
        double l = lo[k], h = hi[k];
        const double tol = tol_of(l, h);
        if (h - l > tol) {
          const double x = tri_snap(l + 0.5 * (h - l));
          if (sturm_count(W, n, x, split) <= k)
            l = x;
          else
            h = x;
          lo[k] = l;
          hi[k] = h;
          done &= (h - l) <= tol ? 1 : 0;
        }
      }
      done = __syncthreads_and(done);
      if (done) {
        converged = 1;
        break;
      }
    }
  }
  for (int iter = 0; iter < iters && !converged && nval <= nthr; ++iter) {
    // the first round's probes cover the whole interval for every eigenvalue
    const int k = tid / G, g = tid % G;
    if (iter == 0) {
      const double x = tri_snap(glo + (ghi - glo) * (double)(tid + 1) / (double)(nthr + 1));
      xs[tid] = x;
      cnt[tid] = sturm_count(W, n, x, split);
    } else if (k < nval) {
      const double l = lo[k], h = hi[k];
      const double x = tri_snap(l + (h - l) * (double)(g + 1) / (double)(G + 1));
      xs[tid] = x;
      cnt[tid] = sturm_count(W, n, x, split);
    }
    __syncthreads();
    int done = 1;
    if (tid < nval) {
      const int kk = tid;
      double l = iter == 0 ? glo : lo[kk], h = iter == 0 ? ghi : hi[kk];
      const double tol = tol_of(l, h);
      const int t0 = iter == 0 ? 0 : kk * G, t1 = iter == 0 ? nthr : kk * G + G;
      if (iter == 0 || h - l > tol) {
        for (int t = t0; t < t1; ++t) {
          if (cnt[t] <= kk)
            l = fmax(l, xs[t]);
          else
            h = fmin(h, xs[t]);
        }
        lo[kk] = l;
        hi[kk] = h;
        done = (h - l) <= tol;
      }
    }
    done = __syncthreads_and(done);
    if (done) {
      converged = 1;
      break;
    }
  }
  int finite = 1;
  for (int k = tid; k < nval; k += nthr) {
    lam[k] = scalbn(0.5 * (lo[k] + hi[k]), ex);
    wout[k] = lam[k];
    finite &= isfinite(lam[k]) ? 1 : 0;
  }
  for (int i = tid; i < n; i += nthr) d[i] = scalbn(d[i], ex);
  finite = __syncthreads_and(finite);
  return !(finite && finite_t) ? 2 : (!converged ? 1 : 0);
}

// LU factors of T - lam I with partial pivoting for repeated solves: per row i
// the multiplier f (its lowest mantissa bit set when rows i and i + 1 were
// swapped, a change of one unit in the last place of f) and 1 / pivot, at
// [i * st]. U's two super-diagonals follow from f, d and e (tri_factored_solve).
// Pivots are kept at or above `tiny` (eps |T|): the eigenvalues of a cluster may be
// equal, and a solve that amplified one of its directions by far more than the others
// would leave the cluster's iterates parallel (graded T: no orthogonality, or NaN).
__device__ inline void tri_factor(const double* __restrict__ d, const double* __restrict__ e, int n, double lam,
                                  double tiny, double* __restrict__ F, double* __restrict__ I0, int st) {
  double a = d[0] - lam;          // current pivot-row diagonal
  double c = n > 1 ? e[0] : 0.0;  // current pivot-row super-diagonal
  for (int i = 0; i < n - 1; ++i) {
    const double b = e[i], dn = d[i + 1] - lam, en = i + 1 < n - 1 ? e[i + 1] : 0.0;
    const size_t o = (size_t)i * st;
    if (fabs(a) >= fabs(b) || fabs(b) < tiny) {
      if (fabs(a) < tiny) a = copysign(tiny, a);
      const double ia = 1.0 / a, f = b * ia;
      F[o] = __longlong_as_double(__double_as_longlong(f) & ~1ll);
      I0[o] = ia;
      a = dn - f * c;
      c = en;
    } else {  // swap rows i and i + 1
      const double ib = 1.0 / b, f = a * ib;
      F[o] = __longlong_as_double(__double_as_longlong(f) | 1ll);
      I0[o] = ib;
      a = c - f * dn;
      c = -f * en;
    }
  }
  if (fabs(a) < tiny) a = copysign(tiny, a);
  I0[(size_t)(n - 1) * st] = 1.0 / a;
}

__device__ __forceinline__ bool tri_swapped(double f) { return (__double_as_longlong(f) & 1ll) != 0; }

// Solves (T - lam I) x = scale b in place with the factors of tri_factor: x (b on
// entry) at xb[i * xs]; returns |x|^2. Division-free; the loads of eight rows run
// ahead of the recurrences (the next eight while these are worked on).
__device__ inline double tri_factored_solve(const double* __restrict__ d, const double* __restrict__ e, double lam,
                                            const double* __restrict__ F, const double* __restrict__ I0, int st, int n,
                                            double* __restrict__ xb, int xs, double scale) {
  constexpr int kB = 8;
  double xc = scale * xb[0];
  {
    double xv[kB], fv[kB], xn[kB], fn[kB];
    auto load = [&](int i0, double (&x)[kB], double (&f)[kB]) {
#pragma unroll
      for (int u = 0; u < kB; ++u) {
        const int i = i0 + u;
        x[u] = i + 1 < n ? xb[(size_t)(i + 1) * xs] : 0.0;
        f[u] = i + 1 < n ? F[(size_t)i * st] : 0.0;
      }
    };
    load(0, xv, fv);
    for (int i0 = 0; i0 < n - 1; i0 += kB) {
      load(i0 + kB, xn, fn);
#pragma unroll
      for (int u = 0; u < kB; ++u) {
        const int i = i0 + u;
        if (i + 1 < n) {
          const double xi = scale * xv[u];
          const bool sw = tri_swapped(fv[u]);
          const double piv = sw ? xi : xc, oth = sw ? xc : xi;
          xb[(size_t)i * xs] = piv;
          xc = fma(-fv[u], piv, oth);
        }
        xv[u] = xn[u];
        fv[u] = fn[u];
      }
    }
  }
  double x1 = xc * I0[(size_t)(n - 1) * st], x2 = 0.0;  // rows i + 1, i + 2
  xb[(size_t)(n - 1) * xs] = x1;
  double s = x1 * x1;
  double yv[kB], iv[kB], fv[kB], yn[kB], in[kB], fn[kB];
  auto load = [&](int i0, double (&y)[kB], double (&p)[kB], double (&f)[kB]) {
#pragma unroll
    for (int u = 0; u < kB; ++u) {
      const int i = i0 - u;
      y[u] = i >= 0 ? xb[(size_t)i * xs] : 0.0;
      p[u] = i >= 0 ? I0[(size_t)i * st] : 0.0;
      f[u] = i >= 1 ? F[(size_t)(i - 1) * st] : 0.0;  // of the row above
    }
  };
  double fi = n > 1 ? F[(size_t)(n - 2) * st] : 0.0;  // of row i
  load(n - 2, yv, iv, fv);
  for (int i0 = n - 2; i0 >= 0; i0 -= kB) {
    load(i0 - kB, yn, in, fn);
#pragma unroll
    for (int u = 0; u < kB; ++u) {
      const int i = i0 - u;
      if (i >= 0) {
        // U's row: swapped (d_{i+1} - lam, e_{i+1}); else (c_i, 0) with c_i = e_i, or
        // -f_{i-1} e_i where row i - 1 was swapped
        const bool sw = tri_swapped(fi);
        const double c = tri_swapped(fv[u]) ? -fv[u] * e[i] : e[i];
        const double u1 = sw ? d[i + 1] - lam : c, u2 = sw && i + 1 < n - 1 ? e[i + 1] : 0.0;
        const double xi = fma(-u1, x1, fma(-u2, x2, yv[u])) * iv[u];
        xb[(size_t)i * xs] = xi;
        s = fma(xi, xi, s);
        x2 = x1;
        x1 = xi;
        fi = fv[u];
      }
      yv[u] = yn[u];
      iv[u] = in[u];
      fv[u] = fn[u];
    }
  }
  return s;
}

// vectors of the inverse iteration side by side: an odd number, so that the rows of
// one vector lie in different banks (at most 4 n nvec doubles for the three arrays)
__host__ __device__ __forceinline__ int tri_ldv(int nvec) { return nvec >= 3 ? (nvec | 1) : nvec; }

// Lowest nvec eigenvectors of T (after tri_eigvals) as real vectors in the
// real parts of z[k * n + i] (imaginary parts zero). One thread per eigenvector:
// one LU factorisation of T - lam I, then kTriInvIters division-free solves from
// a pseudo-random start; after each, the vectors of a cluster of eigenvalues
// closer than 1e-5 |T| are orthogonalised (modified Gram-Schmidt) by one warp.
// The factors and iterates are in `scratch` (3 n tri_ldv(nvec) doubles). `seed`
// makes the start vectors differ per matrix. Every thread of the block calls it.
__device__ inline void tri_eigvecs(const TriWork& W, int n, int nvec, double2* __restrict__ z,
                                   double* __restrict__ scratch, unsigned long long seed) {
  const int tid = threadIdx.x, nthr = blockDim.x, lane = tid & 31, wid = tid >> 5;
  const double* d = W.d;
  const double* e = W.e;
  const double* lam = W.lam;
  double* rn = W.lo;  // 1 / norm of the iterates (the brackets are done with)
  const double tnorm = W.red[3];
  if (tid == 0) {
    int nc = 0;
    const double gap = 1e-5 * tnorm;
    for (int k = 0; k < nvec; ++k)
      if (k == 0 || lam[k] - lam[k - 1] > gap) W.clus[nc++] = k;
    W.clus[nc] = nvec;
    W.misc[0] = nc;
  }
  const int ldv = tri_ldv(nvec);
  double* F = scratch;
  double* I0 = F + (size_t)n * ldv;
  double* X = I0 + (size_t)n * ldv;
  const double tiny = fmax(DBL_EPSILON * tnorm, 1e-290);  // its reciprocal is finite for T = 0 too
  // 1 / |x| of vector k, robust where |x|^2 leaves the FP64 range
  auto inv_norm = [&](int k, double s) {
    if (s > 1e-290 && s < 1e290) return 1.0 / sqrt(s);
    double mx = 0.0;
    for (int i = 0; i < n; ++i) mx = fmax(mx, fabs(X[(size_t)i * ldv + k]));
    if (!(mx > 0.0) || !isfinite(mx)) mx = 1.0;
    s = 0.0;
    for (int i = 0; i < n; ++i) {
      const double v = X[(size_t)i * ldv + k] / mx;
      s += v * v;
    }
    return 1.0 / (mx * sqrt(s));
  };
  for (int k = tid; k < nvec; k += nthr) {
    tri_factor(d, e, n, lam[k], tiny, F + k, I0 + k, ldv);
    for (int i = 0; i < n; ++i) X[(size_t)i * ldv + k] = hash_uniform((seed << 20) + k, i);
    rn[k] = 1.0;
  }
  __syncthreads();
  const int ncl = W.misc[0];
  for (int iter = 0; iter < kTriInvIters; ++iter) {
    for (int k = tid; k < nvec; k += nthr)
      rn[k] = inv_norm(k, tri_factored_solve(d, e, lam[k], F + k, I0 + k, ldv, n, X + k, ldv, rn[k]));
    __syncthreads();
    for (int cl = wid; cl < ncl; cl += nthr / 32) {
      const int c0 = W.clus[cl], c1 = W.clus[cl + 1];
      if (c1 - c0 < 2) continue;
      for (int k = c0; k < c1; ++k) {
        const double r = rn[k];
        for (int i = lane; i < n; i += 32) X[(size_t)i * ldv + k] *= r;
        double s = 1.0;
        for (int kp = c0; kp < k; ++kp) {
          s = 0.0;
          for (int i = lane; i < n; i += 32) s = fma(X[(size_t)i * ldv + kp], X[(size_t)i * ldv + k], s);
          s = -rn[kp] * rn[kp] * warp_sum(s);
          for (int i = lane; i < n; i += 32)
            X[(size_t)i * ldv + k] = fma(s, X[(size_t)i * ldv + kp], X[(size_t)i * ldv + k]);
        }
        s = 0.0;
        for (int i = lane; i < n; i += 32) s = fma(X[(size_t)i * ldv + k], X[(size_t)i * ldv + k], s);
        s = warp_sum(s);
        __syncwarp();
        if (lane == 0) rn[k] = inv_norm(k, s);
        __syncwarp();
      }
    }
    __syncthreads();
  }
  for (int idx = tid; idx < nvec * n; idx += nthr) {
    const int k = idx / n, i = idx - k * n;
    z[idx] = make_double2(X[(size_t)i * ldv + k] * rn[k], 0.0);
  }
  __syncthreads();
}

}  // namespace dev
}  // namespace pmx
