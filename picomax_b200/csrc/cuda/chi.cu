// Stage 2 kernels, FP64 path: overlaps, delta-weighted contraction, scaling and
// the Kramers-Kronig transform of chi_tensor (src/pmx_chi.cpp:319-713) and
// chi_LL (src/pmx_chi_copy.cpp:320-676).
//
// Layouts
//   eigenvectors: z[item][s][row], rows interleaved (G0 up, G0 down, ...) with SOC,
//                 plain G order without SOC (spatial states, spectrum doubled).
//   M[t][a][ch]:  overlap of transition t (sorted), a = 3 m + i (i: L, T+, T-),
//                 ch = channel (1 for epsLL and spin-free epsij, 4 for epsij with
//                 SOC: up, down, updown, downup as in src/pmx_chi.cpp:534-544).
//   acc[2][9][np][nf]: Re then Im accumulators per (i, j, pair(m, n<=m), f),
//                 pair(m, n) = m(m+1)/2 + n, which is the .dat order for one q.
#include <cfloat>
#include <cmath>

#include "pmx_chi.hpp"
#include "pmx_common.cuh"

namespace pmx {
namespace dev {

// ------------------------------------------------------------------- overlaps
// One CTA per (k, conduction chunk, valence chunk), the chunks' eigenvectors
// staged in shared memory (rows padded by 16 bytes). Each thread owns one
// (m, c, v) task at a time (pairs fastest, so a warp shares m and its loci
// row) and sums over the plane waves p with loci[m][p] != -1, accumulating
// the moments sum_p conj(c(p)) v(loci p) {1, G_p.x, G_p.y, G_p.z} per spin
// channel in registers: no cross-lane reductions. The
// orbital current u_i^H (G_p + k + q/2 + G_m/2) and the SOC current
// u_i^H v_soc(G_m) (src/pmx_chi.cpp:203-266, constant over p because
// G_loci - G_p = G_m) are then applied to the moments.
__global__ void __launch_bounds__(256) overlap_kernel(OverlapArgs a) {
  const int k = blockIdx.x;
  const int ncd = a.ncd[k], nvd = a.nvd[k];
  // blockIdx.y = (conduction chunk) + ncc * (valence chunk)
  const int ncc = (a.ncd_max + a.cchunk - 1) / a.cchunk;
  const int c_lo = (blockIdx.y % ncc) * a.cchunk;
  const int c_hi = min(ncd, c_lo + a.cchunk);
  const int v_lo = (blockIdx.y / ncc) * a.vchunk;
  const int v_hi = min(nvd, v_lo + a.vchunk);
  if (c_lo >= c_hi || v_lo >= v_hi) return;
  const int nvl = v_hi - v_lo;
  const int n = a.n, npw = a.npw, ldn = n + 1;
  extern __shared__ __align__(16) unsigned char smraw[];
  double2* sc = reinterpret_cast<double2*>(smraw);           // [cchunk][ldn]
  double2* sv = sc + (size_t)a.cchunk * ldn;                  // [vchunk][ldn]
  double* sg = reinterpret_cast<double*>(sv + (size_t)a.vchunk * ldn);  // [npw][3]
  const int tid = threadIdx.x;
  for (int c = c_lo; c < c_hi; ++c) {
    const double2* src = a.zk + ((size_t)k * a.nev + a.cidx[a.cbase[k] + c]) * n;
    for (int r = tid; r < n; r += blockDim.x) sc[(size_t)(c - c_lo) * ldn + r] = src[r];
  }
  for (int v = v_lo; v < v_hi; ++v) {
    const double2* src = a.zq + ((size_t)k * a.nev + a.vidx[a.vbase[k] + v]) * n;
    for (int r = tid; r < n; r += blockDim.x) sv[(size_t)(v - v_lo) * ldn + r] = src[r];
  }
  for (int r = tid; r < 3 * npw; r += blockDim.x) sg[r] = a.G[r];
  __syncthreads();
  const double kx = a.kpts[3 * k], ky = a.kpts[3 * k + 1], kz = a.kpts[3 * k + 2];
  const int npair = (c_hi - c_lo) * nvl;
  const int A = 3 * a.neps;
  const int ntask = a.neps * npair;
  for (int task = tid; task < ntask; task += blockDim.x) {
    const int m = task / npair, pr = task - m * npair;
    const int cl = pr / nvl, v = v_lo + pr % nvl;
    const long long dst = a.dest[a.blkoff[k] + (long long)(c_lo + cl) * nvd + v];
    if (dst < 0) continue;
    const int* loci = a.loci + (size_t)m * npw;
    const double2* cvec = sc + (size_t)cl * ldn;
    const double2* vvec = sv + (size_t)(v - v_lo) * ldn;
    // moments: [0..3] spin-summed or up-up, [4..7] down-down, [8] up-down, [9] down-up
    double2 mo[10];
#pragma unroll
    for (int q = 0; q < 10; ++q) mo[q] = make_double2(0, 0);
    for (int p = 0; p < npw; ++p) {
      const int lp = loci[p];
      if (lp < 0) continue;
      const double gx = sg[3 * p], gy = sg[3 * p + 1], gz = sg[3 * p + 2];
      if (!a.soc) {
        const double2 s = cmulc(cvec[p], vvec[lp]);
        mo[0] = cadd(mo[0], s);
        mo[1] = cadd(mo[1], cscale(s, gx));
        mo[2] = cadd(mo[2], cscale(s, gy));
        mo[3] = cadd(mo[3], cscale(s, gz));
      } else {
        const double2 cu = cvec[2 * p], cd = cvec[2 * p + 1];
        const double2 vu = vvec[2 * lp], vd = vvec[2 * lp + 1];
        const double2 uu = cmulc(cu, vu), dd = cmulc(cd, vd);
        if (a.nch == 4) {
          mo[0] = cadd(mo[0], uu);
          mo[1] = cadd(mo[1], cscale(uu, gx));
          mo[2] = cadd(mo[2], cscale(uu, gy));
          mo[3] = cadd(mo[3], cscale(uu, gz));
          mo[4] = cadd(mo[4], dd);
          mo[5] = cadd(mo[5], cscale(dd, gx));
          mo[6] = cadd(mo[6], cscale(dd, gy));
          mo[7] = cadd(mo[7], cscale(dd, gz));
          mo[8] = cadd(mo[8], cmulc(cu, vd));
          mo[9] = cadd(mo[9], cmulc(cd, vu));
        } else {
          const double2 s = cadd(uu, dd);
          mo[0] = cadd(mo[0], s);
          mo[1] = cadd(mo[1], cscale(s, gx));
          mo[2] = cadd(mo[2], cscale(s, gy));
          mo[3] = cadd(mo[3], cscale(s, gz));
        }
      }
    }
    // w = k + q/2 + G_m/2, as in (G_p + K + Q/2 + G_m/2) at src/pmx_chi.cpp:535
    const double wx = (kx + a.q[0] / 2) + a.G[3 * m] / 2;
    const double wy = (ky + a.q[1] / 2) + a.G[3 * m + 1] / 2;
    const double wz = (kz + a.q[2] / 2) + a.G[3 * m + 2] / 2;
    double2* out = a.M + ((size_t)dst * A + 3 * m) * a.nch;
#pragma unroll 1
    for (int i = 0; i < 3; ++i) {
      const double2* u = a.uvec + ((size_t)m * 3 + i) * 3;  // u_i of q+G_m
      const double2 s = a.ssoc[m * 3 + i];                  // u_i^H v_soc(G_m)
      // orbital current of a moment set: sum_x conj(u_x) (M_x + w_x M_0)
      auto orb = [&](const double2* mm) {
        double2 r = cmulc(u[0], cadd(mm[1], cscale(mm[0], wx)));
        r = cadd(r, cmulc(u[1], cadd(mm[2], cscale(mm[0], wy))));
        r = cadd(r, cmulc(u[2], cadd(mm[3], cscale(mm[0], wz))));
        return r;
      };
      if (a.mode == 1) {  // epsLL: L = density, T = u.(v_orb + v_soc)
        out[(size_t)i * a.nch] = i == 0 ? mo[0] : cadd(orb(mo), cmul(s, mo[0]));
      } else if (a.nch == 1) {  // epsij without SOC: single channel, orbital current
        out[(size_t)i * a.nch] = orb(mo);
      } else {  // epsij with SOC: up, down, updown, downup
        double2* o = out + (size_t)i * 4;
        o[0] = orb(mo);
        o[1] = orb(mo + 4);
        o[2] = cmul(s, mo[8]);
        o[3] = cmul(s, mo[9]);
      }
    }
  }
}

cudaError_t launch_overlap(const OverlapArgs& a, int nk, cudaStream_t st) {
  if (nk <= 0) return cudaSuccess;
  if (a.cchunk < 1 || a.vchunk < 1) return cudaErrorInvalidValue;
  const size_t smem = overlap_smem_bytes(a.cchunk, a.vchunk, a.n, a.npw);
  cudaError_t err = cudaFuncSetAttribute(overlap_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (err != cudaSuccess) return err;
  const int ncc = (a.ncd_max + a.cchunk - 1) / a.cchunk, nvc = (a.nvd_max + a.vchunk - 1) / a.vchunk;
  dim3 grid(nk, ncc * nvc);
  overlap_kernel<<<grid, 256, smem, st>>>(a);
  return cudaGetLastError();
}

size_t overlap_smem_bytes(int cchunk, int vchunk, int n, int npw) {
  return ((size_t)cchunk + vchunk) * (n + 1) * sizeof(double2) + (size_t)3 * npw * sizeof(double);
}

bool overlap_tiles(int ncd_max, int nvd_max, int n, int npw, int& cchunk, int& vchunk) {
  const size_t lim = 200 * 1024;
  vchunk = std::max(1, nvd_max);
  cchunk = std::max(1, ncd_max);
  while (cchunk > 1 && overlap_smem_bytes(cchunk, vchunk, n, npw) > lim) --cchunk;
  while (vchunk > 1 && overlap_smem_bytes(cchunk, vchunk, n, npw) > lim) --vchunk;
  return overlap_smem_bytes(cchunk, vchunk, n, npw) <= lim;
}

int overlap_tile_candidates(int ncd_max, int nvd_max, int n, int npw, int* cc, int* vc, int maxc) {
  int c0 = 1, v0 = 1;
  if (!overlap_tiles(ncd_max, nvd_max, n, npw, c0, v0) || maxc < 1) return 0;
  const int cs[2] = {c0, (c0 + 1) / 2}, vs[2] = {v0, (v0 + 1) / 2};
  int cnt = 0;
  for (int i = 0; i < 2; ++i)
    for (int j = 0; j < 2; ++j) {
      bool dup = false;
      for (int q = 0; q < cnt; ++q) dup = dup || (cc[q] == cs[i] && vc[q] == vs[j]);
      if (!dup && cnt < maxc) {
        cc[cnt] = cs[i];
        vc[cnt] = vs[j];
        ++cnt;
      }
    }
  return cnt;
}

// ------------------------------------------------------------ broadening
// src/pmx_chi.cpp:90-164; delta model 0 gauss, 1 lorentz, 2 triangle, 3 rect.
__device__ __forceinline__ double broaden(int model, double eps, double x) {
  switch (model) {
    case 0:
      return exp(-0.5 * x * x / (eps * eps)) / (eps * sqrt(2.0 * 3.14159265358979323846));
    case 1:
      return eps / 3.14159265358979323846 / (eps * eps + x * x);
    case 2:
      return fabs(x) < 0.5 * eps ? 4.0 / eps * (0.5 - fabs(x) / eps) : 0.0;
    default:
      return fabs(x) < 0.5 * eps ? 1.0 / eps : 0.0;
  }
}

// ---------------------------- FP64 contraction with the principal-value term
// (epsLL and epsxyz with kk = 0): the sums of contract64.cu over all transitions
// (src/pmx_chi_copy.cpp:546-575), and with them the principal-value sums of
// src/pmx_chi_copy.cpp:597-615, whose weights depend on the block (i, j) of a
// pair, so that they are not one more matrix product. One CTA computes a 12x12
// block of (a, b) = (3m+i, 3n+j) pairs for 64 frequencies.
namespace {
constexpr int kMB = 4;              // m per block
constexpr int kAB = 3 * kMB;        // a (or b) per block
constexpr int kPairs = kAB * kAB;   // 144
constexpr int kFT = 64;             // frequencies per tile
constexpr int kTK = 16;             // transitions per chunk
constexpr int kCThreads = 256;
}  // namespace

__device__ __forceinline__ void tile_of(int id, int& ta, int& tb) {
  // lower-triangular enumeration: id -> (ta >= tb)
  int r = (int)((sqrt(8.0 * id + 1.0) - 1.0) * 0.5);
  while ((r + 1) * (r + 2) / 2 <= id) ++r;
  while (r * (r + 1) / 2 > id) --r;
  ta = r;
  tb = id - r * (r + 1) / 2;
}

__global__ void __launch_bounds__(kCThreads) contract_pv_kernel(ContractArgs a) {
  int ta, tb;
  tile_of(blockIdx.x, ta, tb);
  const int f_lo = blockIdx.y * kFT;
  const int2 tr = a.trange[blockIdx.y];
  const int A = 3 * a.neps;
  const int a0 = ta * kAB, b0 = tb * kAB;
  extern __shared__ __align__(16) unsigned char smraw[];
  typedef double2 MTile[kAB];
  typedef double PRow[kTK + 1];
  typedef double WTile[kTK][kFT];
  MTile* sMa = reinterpret_cast<MTile*>(smraw);
  MTile* sMb = sMa + kTK;
  PRow* sP1 = reinterpret_cast<PRow*>(sMb + kTK);
  PRow* sP2 = sP1 + kPairs;
  WTile* sW = reinterpret_cast<WTile*>(sP2 + kPairs);
  double* sw = reinterpret_cast<double*>(sW + 4);
  double* sde = sw + kTK;
  const int tid = threadIdx.x;
  const int pg = tid / 16, fg = tid % 16;
  double acc1[9][4], acc2[9][4];  // 1: Im (reO), 2: Re (-imO)
  double pv1[9][4], pv2[9][4];
#pragma unroll
  for (int u = 0; u < 9; ++u)
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      acc1[u][q] = 0;
      acc2[u][q] = 0;
      pv1[u][q] = 0;
      pv2[u][q] = 0;
    }
  int pclass[9];
#pragma unroll
  for (int u = 0; u < 9; ++u) {
    const int pp = pg * 9 + u;
    const int i = (pp / kAB) % 3, j = (pp % kAB) % 3;
    pclass[u] = a.pvclass ? a.pvclass : ((i == 0 && j == 0) ? 1 : ((i == 0 || j == 0) ? 2 : 3));
  }
  for (int t0 = tr.x; t0 < tr.y; t0 += kTK) {
    const int nt = min(kTK, tr.y - t0);
    // stage M of the chunk
    for (int idx = tid; idx < kTK * kAB; idx += kCThreads) {
      const int t = idx / kAB, aa = idx % kAB;
      double2 va = make_double2(0, 0), vb = make_double2(0, 0);
      if (t < nt) {
        const size_t base = (size_t)(t0 + t) * A;
        if (a0 + aa < A) va = a.M[base + a0 + aa];
        if (b0 + aa < A) vb = a.M[base + b0 + aa];
      }
      sMa[t][aa] = va;
      sMb[t][aa] = vb;
    }
    if (tid < kTK) {
      const int t = tid;
      sw[t] = t < nt ? a.wgt[t0 + t] : 0.0;
      sde[t] = t < nt ? a.dE[t0 + t] : 0.0;
    }
    __syncthreads();
    // pair products P1 = w reO, P2 = -w imO
    for (int idx = tid; idx < kPairs * kTK; idx += kCThreads) {
      const int pp = idx / kTK, t = idx % kTK;
      const int ia = pp / kAB, ib = pp % kAB;
      const double2 o = cmulc(sMb[t][ib], sMa[t][ia]);  // a conj(b)
      sP1[pp][t] = sw[t] * o.x;
      sP2[pp][t] = -sw[t] * o.y;
    }
    // weights
    for (int idx = tid; idx < kTK * kFT; idx += kCThreads) {
      const int t = idx / kFT, fl = idx % kFT;
      const int f = f_lo + fl;
      double wv = 0.0;
      const double om = a.dfreq * f;
      const bool ok = t < nt && f < a.nf;
      if (ok) wv = broaden(a.delta, a.eps, sde[t] - om);
      sW[0][t][fl] = wv;
      const double de = sde[t];
      const double den = de * de - om * om;
      sW[1][t][fl] = ok ? de / den : 0.0;          // LL
      sW[2][t][fl] = ok ? 1.0 / den : 0.0;         // LT
      sW[3][t][fl] = ok ? 1.0 / de / den : 0.0;    // TT
    }
    __syncthreads();
    for (int t = 0; t < nt; ++t) {
      double wv[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) wv[q] = sW[0][t][fg + 16 * q];
#pragma unroll
      for (int u = 0; u < 9; ++u) {
        const double p1 = sP1[pg * 9 + u][t], p2 = sP2[pg * 9 + u][t];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          acc1[u][q] = fma(p1, wv[q], acc1[u][q]);
          acc2[u][q] = fma(p2, wv[q], acc2[u][q]);
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const double g = sW[pclass[u]][t][fg + 16 * q];
          pv1[u][q] = fma(p1, g, pv1[u][q]);   // Re2 += w Re(O) g
          pv2[u][q] = fma(-p2, g, pv2[u][q]);  // Im2 += w Im(O) g
        }
      }
    }
    __syncthreads();
  }
  // store
  const size_t blk = (size_t)9 * a.np * a.nf;
#pragma unroll
  for (int u = 0; u < 9; ++u) {
    const int pp = pg * 9 + u;
    const int ia = pp / kAB, ib = pp % kAB;
    const int av = a0 + ia, bv = b0 + ib;
    const int m = av / 3, i = av % 3, nn = bv / 3, j = bv % 3;
    if (m >= a.neps || nn >= a.neps || nn > m) continue;
    const size_t row = ((size_t)(i * 3 + j) * a.np + (size_t)m * (m + 1) / 2 + nn) * a.nf;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int f = f_lo + fg + 16 * q;
      if (f >= a.nf) continue;
      a.acc[row + f] = acc2[u][q];        // Re part
      a.acc[blk + row + f] = acc1[u][q];  // Im part
      a.acc_pv[row + f] = pv1[u][q];
      a.acc_pv[blk + row + f] = pv2[u][q];
    }
  }
}

cudaError_t launch_contract_pv(const ContractArgs& a, cudaStream_t st) {
  const int nmb = (a.neps + kMB - 1) / kMB;
  const int ntiles = nmb * (nmb + 1) / 2;
  const int nft = (a.nf + kFT - 1) / kFT;
  dim3 grid(ntiles, nft);
  if (a.nch != 1 || !a.acc_pv) return cudaErrorInvalidValue;
  const size_t sm = (size_t)2 * kTK * kAB * sizeof(double2) + (size_t)2 * kPairs * (kTK + 1) * sizeof(double) +
                    (size_t)4 * kTK * kFT * sizeof(double) + (size_t)2 * kTK * sizeof(double);
  const cudaError_t err =
      cudaFuncSetAttribute(contract_pv_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  if (err != cudaSuccess) return err;
  contract_pv_kernel<<<grid, kCThreads, sm, st>>>(a);
  return cudaGetLastError();
}

// ---------------------------------------------------------------- scaling
// epsij: chi = SCALEFACTOR acc / w_f^2 with 1/w_0^2 := 0 (src/pmx_chi.cpp:559-563, :631-634).
// epsLL: chi = pi acc * class factor (src/pmx_chi_copy.cpp:579-596), f = 0 gives 0,
//        plus 2 * PV * class factor when kk = 0 (:597-615).
// One CTA per row (i, j, pair) of the Re or Im block: its factors are found once and
// the row is a stream. Bound by HBM: 15930 rows x 2000 frequencies (1 GB) in 0.24 ms
// on a B200; with the row's indices and factors per element it took 0.53 ms.
__global__ void __launch_bounds__(256) scale_kernel(ScaleArgs s) {
  const int row = blockIdx.x;
  const int pair = row % s.np, ij = row / s.np;
  const int i = ij / 3, j = ij % 3;
  int m = (int)((sqrt(8.0 * pair + 1.0) - 1.0) * 0.5);
  while ((m + 1) * (m + 2) / 2 <= pair) ++m;
  while (m * (m + 1) / 2 > pair) --m;
  const int n = pair - m * (m + 1) / 2;
  const size_t o = ((size_t)blockIdx.y * 9 * s.np + row) * s.nf;
  // class of the row: 0 sf_ll / (q_m q_n), 1 sf_lt / q_m, 2 sf_lt / q_n, 3 sf_tt; the
  // first factor of 1 falls with w, that of 3 with w^2
  const double qm = s.mode == 0 ? 1.0 : s.qgn[m], qn = s.mode == 0 ? 1.0 : s.qgn[n];
  // epsxyz: every block scales as TT (src/pmx_chi_copy.cpp:1093, :1272-1281)
  const int cls = s.mode == 2 ? 3 : (i == 0 ? (j == 0 ? 0 : 1) : (j == 0 ? 2 : 3));
  const double f2 = cls == 0 ? s.sf_ll / (qm * qn) : (cls == 1 ? s.sf_lt / qm : (cls == 2 ? s.sf_lt / qn : s.sf_tt));
  for (int f = threadIdx.x; f < s.nf; f += blockDim.x) {
    const double w = s.dfreq * f;
    double v = s.acc[o + f];
    if (s.mode == 0) {
      const double inv = f == 0 ? 0.0 : 1.0 / (w * w);
      v = s.sf * (v * inv);
    } else {
      double f1 = f2;
      if (f == 0)
        f1 = 0.0;
      else if (cls == 1)
        f1 = s.sf_lt / (qm * w);
      else if (cls == 3)
        f1 = s.sf_tt / (w * w);
      v = 3.14159265358979323846 * (v * f1);
      if (s.acc_pv) v += 2.0 * (s.acc_pv[o + f] * f2);
    }
    s.out[o + f] = v;
  }
}

cudaError_t launch_scale(const ScaleArgs& s, cudaStream_t st) {
  scale_kernel<<<dim3(9 * s.np, 2), 256, 0, st>>>(s);
  return cudaGetLastError();
}

// ------------------------------------------------------- Kramers-Kronig
// src/pmx_chi.cpp:272-309: Re_f += ds sum_{s!=f} w_s Im_s/(w_s^2-w_f^2),
// Im_f += ds sum_{s!=f} w_s Re0_s/(w_s^2-w_f^2), ds = 2 dw / pi, both from the
// values before the transform. As a GEMM: Y = X K^T with X = [Im; Re] rows and
// K generated on the fly, then chi += ds Y (swapped halves).
namespace {
constexpr int kKT = 64, kKK = 16;
}

__global__ void __launch_bounds__(256) kk_kernel(const double* __restrict__ chi, double* __restrict__ out,
                                                 int rows, int nf, double dfreq) {
  // chi: [2][rows][nf] (Re block then Im block); out same layout.
  const int r0 = blockIdx.x * kKT, f0 = blockIdx.y * kKT;
  __shared__ double sX[kKK][kKT + 1];
  __shared__ double sK[kKK][kKT + 1];
  const int tid = threadIdx.x, tr = tid / 16, tc = tid % 16;
  double acc[4][4];
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b) acc[a][b] = 0;
  const size_t blk = (size_t)rows * nf;
  // logical row r in [0, 2 rows): r < rows -> source Im row r (updates Re), else source Re row
  for (int s0 = 0; s0 < nf; s0 += kKK) {
    for (int idx = tid; idx < kKK * kKT; idx += 256) {
      const int ss = idx / kKT, rr = idx % kKT;
      const int r = r0 + rr, s = s0 + ss;
      double x = 0.0;
      if (r < 2 * rows && s < nf) {
        const size_t src = r < rows ? blk + (size_t)r * nf + s : (size_t)(r - rows) * nf + s;
        x = chi[src];
      }
      sX[ss][rr] = x;
      const int f = f0 + rr;
      double kv = 0.0;
      if (s < nf && f < nf && s != f) {
        const double ws = dfreq * s, wf = dfreq * f;
        kv = ws / (ws * ws - wf * wf);
      }
      sK[ss][rr] = kv;
    }
    __syncthreads();
#pragma unroll
    for (int ss = 0; ss < kKK; ++ss) {
      double xa[4], kb[4];
#pragma unroll
      for (int a = 0; a < 4; ++a) xa[a] = sX[ss][tr + 16 * a];
#pragma unroll
      for (int b = 0; b < 4; ++b) kb[b] = sK[ss][tc + 16 * b];
#pragma unroll
      for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) acc[a][b] = fma(xa[a], kb[b], acc[a][b]);
    }
    __syncthreads();
  }
  const double ds = dfreq * 2.0 / 3.14159265358979323846;
#pragma unroll
  for (int a = 0; a < 4; ++a) {
    const int r = r0 + tr + 16 * a;
    if (r >= 2 * rows) continue;
    const size_t dst = r < rows ? (size_t)r * nf : blk + (size_t)(r - rows) * nf;
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      const int f = f0 + tc + 16 * b;
      if (f >= nf) continue;
      out[dst + f] = chi[dst + f] + ds * acc[a][b];
    }
  }
}

cudaError_t launch_kk(const double* chi, double* out, int rows, int nf, double dfreq, cudaStream_t st) {
  dim3 grid((2 * rows + kKT - 1) / kKT, (nf + kKT - 1) / kKT);
  kk_kernel<<<grid, 256, 0, st>>>(chi, out, rows, nf, dfreq);
  return cudaGetLastError();
}

}  // namespace dev
}  // namespace pmx

namespace pmx {
namespace dev {

// ------------------------------------------------------------ macroscopic eps
// eps_M(q, w) = 1 / [eps^-1]_00 with eps_mn = delta_mn + chi^LL_mn and the
// n > m half filled by conj(eps_nm), as in the reference's post-processing
// (include/matlab_wrapper/+picomax/+eps/macroscopic.m:13-29, :79). With vector 0
// last, Gaussian elimination of eps x = e_0 with partial pivoting ends in
// u x_0 = y, so that eps_M = 1 / x_0 = u / y without a back substitution; y is 1
// (u is the Schur complement of eps[1:, 1:]) until row 0 itself becomes a pivot,
// which it must where eps[1:, 1:] is near-singular (a pole of eps_M, at which the
// loss function is regular; at the pole itself y = 0 and eps_M is infinite). From
// then on the right-hand side is one more column, kept where that pivot's column
// was. One CTA per (q, w), the matrix in shared memory, lanes over columns and
// warps over rows: bound by the latency of
// the n steps, so that several CTAs share an SM (four of 59 vectors; four warps of
// one CTA had a matrix each before, with a serial back substitution). Measured on a
// B200, 2000 frequencies: 59 vectors 2.06 -> 0.60 ms, 27 vectors 0.138 -> 0.091 ms, 15
// vectors 0.058 -> 0.047 ms.
__global__ void __launch_bounds__(128) epsm_kernel(const double* __restrict__ re, const double* __restrict__ im,
                                                   int neps, int nf, double2* __restrict__ out) {
  extern __shared__ __align__(16) unsigned char smraw[];
  double2* E = reinterpret_cast<double2*>(smraw);  // [n][n], row and column m at (m + n - 1) % n
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int job = blockIdx.x, q = job / nf, f = job % nf;
  const int n = neps, np = n * (n + 1) / 2;
  // chi LL block: [i=0][j=0][q][pair][f]
  for (int r = wid; r < n; r += nw)
    for (int c = lane; c <= r; c += 32) {
      const size_t o = ((size_t)q * np + (size_t)r * (r + 1) / 2 + c) * nf + f;
      double2 v = make_double2(re[o], im[o]);
      const int ri = r == 0 ? n - 1 : r - 1, ci = c == 0 ? n - 1 : c - 1;
      if (r == c) v.x += 1.0;
      E[ri * n + ci] = v;
      if (r != c) E[ci * n + ri] = cconj(v);  // eps_nm = conj(eps_mn) above the diagonal
    }
  __syncthreads();
  int rhs = -1;  // column of the right-hand side, once row 0 (the last row) has been a pivot
  for (int k = 0; k < n - 1; ++k) {
    // pivot among rows k .. n - 1, the same search in every warp
    double best = -1.0;
    int bi = k;
    for (int r = k + lane; r < n; r += 32) {
      const double2 v = E[r * n + k];
      const double a = v.x * v.x + v.y * v.y;
      if (a > best) {
        best = a;
        bi = r;
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const double ob = __shfl_xor_sync(0xffffffffu, best, o);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      if (ob > best || (ob == best && oi < bi)) {
        best = ob;
        bi = oi;
      }
    }
    if (bi != k) {
      __syncthreads();  // every warp has searched
      for (int c = k + threadIdx.x; c <= n; c += blockDim.x) {
        const int cc = c < n ? c : rhs;
        if (cc < 0) continue;
        const double2 t = E[k * n + cc];
        E[k * n + cc] = E[bi * n + cc];
        E[bi * n + cc] = t;
      }
      __syncthreads();
    }
    const bool row0 = rhs < 0 && bi == n - 1;  // row 0 with its right-hand side 1, the others' still 0
    const double2 p = E[k * n + k];
    const double pd = p.x * p.x + p.y * p.y;
    const double2 inv = make_double2(p.x / pd, -p.y / pd);
    for (int r = k + 1 + wid; r < n; r += nw) {
      const double2 fct = cmul(E[r * n + k], inv);
      for (int c = k + 1 + lane; c < n; c += 32) E[r * n + c] = csub(E[r * n + c], cmul(fct, E[k * n + c]));
      if (rhs >= 0 && lane == 0) E[r * n + rhs] = csub(E[r * n + rhs], cmul(fct, E[k * n + rhs]));
      if (row0) {
        __syncwarp();  // the lanes have read the factor from there
        if (lane == 0) E[r * n + k] = make_double2(-fct.x, -fct.y);
      }
    }
    if (row0) rhs = k;
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    double2 u = E[n * n - 1];
    if (rhs >= 0) {
      const double2 y = E[(n - 1) * n + rhs];
      const double m = fmax(fabs(y.x), fabs(y.y));
      if (y.x == 0.0 && y.y == 0.0 && (u.x != 0.0 || u.y != 0.0)) {
        u = make_double2(INFINITY, 0.0);
      } else {
        const double2 ys = make_double2(y.x / m, y.y / m);
        const double d = m * (ys.x * ys.x + ys.y * ys.y);
        u = cmulc(ys, u);
        u = make_double2(u.x / d, u.y / d);
      }
    }
    out[job] = u;
  }
}

cudaError_t launch_epsm(const double* re, const double* im, int neps, int nq, int nf, double2* out, cudaStream_t st) {
  if (neps > 64 || neps < 1) return cudaErrorInvalidValue;
  const size_t smem = (size_t)neps * neps * sizeof(double2);
  cudaError_t e = cudaFuncSetAttribute(epsm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  // warps per matrix: one row pass of the lanes per warp up to 32 vectors
  const int thr = neps <= 16 ? 32 : (neps <= 32 ? 64 : 128);
  epsm_kernel<<<nq * nf, thr, smem, st>>>(re, im, neps, nf, out);
  return cudaGetLastError();
}

// Electron energy-loss function L(q, w) = -Im(1 / eps_M(q, w)) (the quantity
// the macroscopic dielectric function of macroscopic.m, :13-29 and :79, is
// taken for in EELS), and per q the loss peak: the plasmon. One warp per q:
// argmax of L over frequencies f >= fmin (ties to the lower f), then the
// vertex of the parabola through the peak and its two neighbours.
__global__ void __launch_bounds__(128) loss_kernel(const double2* __restrict__ epsm, int nq, int nf, int fmin,
                                                   double dfreq, double* __restrict__ loss,
                                                   double* __restrict__ peak) {
  const int lane = threadIdx.x & 31;
  const int q = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (q >= nq) return;
  const double2* e = epsm + (size_t)q * nf;
  double* L = loss + (size_t)q * nf;
  double best = -1.0;
  int bi = -1;
  for (int f = lane; f < nf; f += 32) {
    const double2 v = e[f];
    const double d = v.x * v.x + v.y * v.y;
    const double l = d > 0.0 ? v.y / d : 0.0;  // -Im(1/eps) = Im(eps) / |eps|^2
    L[f] = l;
    if (f >= fmin && (l > best || bi < 0)) {
      best = l;
      bi = f;
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    const double ob = __shfl_xor_sync(0xffffffffu, best, o);
    const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
    if (oi >= 0 && (bi < 0 || ob > best || (ob == best && oi < bi))) {
      best = ob;
      bi = oi;
    }
  }
  __syncwarp();
  if (lane == 0) {
    double w = bi >= 0 ? bi * dfreq : 0.0, h = bi >= 0 ? best : 0.0;
    if (bi > 0 && bi + 1 < nf) {
      const double ym = L[bi - 1], y0 = L[bi], yp = L[bi + 1];
      const double den = ym - 2.0 * y0 + yp;
      if (den < 0.0) {
        const double t = 0.5 * (ym - yp) / den;  // in (-1/2, 1/2) at a strict maximum
        w = (bi + t) * dfreq;
        h = y0 - 0.25 * (ym - yp) * t;
      }
    }
    peak[2 * q] = w;
    peak[2 * q + 1] = h;
  }
}

cudaError_t launch_loss(const double2* epsm, int nq, int nf, int fmin, double dfreq, double* loss, double* peak,
                        cudaStream_t st) {
  if (nq <= 0 || nf <= 0) return cudaSuccess;
  loss_kernel<<<(nq + 3) / 4, 128, 0, st>>>(epsm, nq, nf, fmin, dfreq, loss, peak);
  return cudaGetLastError();
}

}  // namespace dev
}  // namespace pmx
