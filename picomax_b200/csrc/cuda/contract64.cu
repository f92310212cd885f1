// FP64 chi contraction on the FP64 tensor cores:
//   acc_im[p, f] = sum_t w_t reO_t(p) delta(dE_t - w_f),
//   acc_re[p, f] = -sum_t w_t imO_t(p) delta(dE_t - w_f)
// over the transitions whose window covers f (src/pmx_chi.cpp:573-627), or over
// those whose line shape is not zero there (src/pmx_chi_copy.cpp:546-575).
//
// One CTA: rows = 81 pairs (a, b) of a 9 x 9 block (3 local-field vectors x 3
// directions on each side) as P1 = w reO and P2 = -w imO (162 rows, padded to
// 21 row tiles of 8), columns = 64 frequencies, depth = 16 transitions a chunk.
// Bound by the FP64 pipe. The products and the line shape are formed once per
// chunk in shared memory and multiplied with mma.sync m8n8k4: one instruction
// does the work of eight FMAs per lane from one 8-byte load per operand, where
// register-tiled FMAs took 22 loads per 72. 9 x 9 blocks end on whole
// local-field vectors, so only diagonal blocks hold unused pairs (7 % of the
// rows at 27 vectors, 12 x 12 blocks 14 %). 192 threads with 56 accumulators
// each: two CTAs share an SM, one forms its next chunk while the other
// multiplies; one barrier per chunk (products and line shape double-buffered,
// the next chunk's overlaps by cp.async meanwhile). The line shape, an exp() or a
// division per entry that every pair block would repeat, is tabulated once per
// launch where three blocks or more share it and the table stays within 4 GB.
// Measured on a B200 against 12 x 12 FMA tiles that also ran over the frequencies
// where epsLL's line shape is zero: GaAs + spin-orbit epsij (216 k, 27 vectors,
// 2000 frequencies) 18.2 -> 4.36 ms, wurtzite epsLL (144 k, 59 vectors) 249.7 ->
// 26.9 ms, silicon epsLL (512 k, 15 vectors) 7.70 -> 0.87 ms (without the table 6.1,
// 38.1, 1.20 ms); 16.6 and 22 TFLOP/s in the window on the first two (DGEMM 35.5).
#include <algorithm>
#include <cfloat>
#include <cmath>

#include "pmx_chi.hpp"
#include "pmx_common.cuh"
#include "pmx_dmma.cuh"

namespace pmx {
namespace dev {

namespace {

constexpr int kMB = 3;                 // local-field vectors per block side
constexpr int kAB = 3 * kMB;           // rows of overlaps per side
constexpr int kPairs = kAB * kAB;      // 81
constexpr int kRowTiles = 21;          // 8-row tiles: 2 * 81 rows padded to 168
constexpr int kRows = 8 * kRowTiles;
constexpr int kFT = 64;                // frequencies per CTA
constexpr int kTK = 16;                // transitions per chunk
constexpr int kThr = 192;              // 3 row groups x 2 column groups of warps
constexpr int kWM = 7, kWN = 4;        // 8 x 8 tiles per warp
constexpr int kPLd = kTK + 4;          // row strides that keep the fragment loads free of bank conflicts
constexpr int kWLd = kFT + 4;
constexpr int kMaxSplit = 8;
constexpr size_t kMaxTable = (size_t)4 << 30;  // largest table of line shapes

__device__ __forceinline__ void cp_async16_zfill(void* smem, const void* gmem, bool ok) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_addr(smem)), "l"(gmem), "r"(ok ? 16 : 0)
               : "memory");
}

// lower-triangular enumeration of the blocks: id -> (ta >= tb)
__device__ __forceinline__ void block_of(int id, int& ta, int& tb) {
  int r = (int)((sqrt(8.0 * id + 1.0) - 1.0) * 0.5);
  while ((r + 1) * (r + 2) / 2 <= id) ++r;
  while (r * (r + 1) / 2 > id) --r;
  ta = r;
  tb = id - r * (r + 1) / 2;
}

// line shapes of src/pmx_chi.cpp:90-164 with the constants of the Gaussian hoisted
struct Line {
  int model;
  double eps, norm, arg;
  __device__ __forceinline__ double operator()(double x) const {
    switch (model) {
      case 0:
        return norm * exp(arg * (x * x));
      case 1:
        return norm / (arg + x * x);
      case 2:
        return fabs(x) < 0.5 * eps ? 4.0 / eps * (0.5 - fabs(x) / eps) : 0.0;
      default:
        return fabs(x) < 0.5 * eps ? 1.0 / eps : 0.0;
    }
  }
};
__device__ __forceinline__ Line make_line(int model, double eps) {
  Line l{model, eps, 0.0, 0.0};
  if (model == 0) {
    l.norm = 1.0 / (eps * sqrt(2.0 * 3.14159265358979323846));
    l.arg = -0.5 / (eps * eps);
  } else if (model == 1) {
    l.norm = eps / 3.14159265358979323846;
    l.arg = eps * eps;
  }
  return l;
}

// W chunks (kTK transitions x kFT frequencies, row-major) per frequency tile: how
// many before tile ft, in wofs[ft]
__global__ void __launch_bounds__(1024) chunk_offsets_kernel(const int2* __restrict__ trange, int nft,
                                                             long long* __restrict__ wofs) {
  __shared__ long long sums[1024];
  long long base = 0;
  for (int f0 = 0; f0 < nft; f0 += 1024) {
    const int ft = f0 + threadIdx.x;
    const long long c = ft < nft ? (trange[ft].y - trange[ft].x + kTK - 1) / kTK : 0;
    sums[threadIdx.x] = c;
    __syncthreads();
    for (int o = 1; o < 1024; o <<= 1) {
      const long long v = threadIdx.x >= o ? sums[threadIdx.x - o] : 0;
      __syncthreads();
      sums[threadIdx.x] += v;
      __syncthreads();
    }
    if (ft < nft) wofs[ft] = base + sums[threadIdx.x] - c;
    base += sums[1023];
    __syncthreads();
  }
}

// The line shape of every chunk, once for all pair blocks
__global__ void __launch_bounds__(256) wtab_kernel(ContractArgs a, const long long* __restrict__ wofs,
                                                   double* __restrict__ wtab) {
  const int ft = blockIdx.y, f_lo = ft * kFT;
  const int2 tr = a.trange[ft];
  const int nc = (tr.y - tr.x + kTK - 1) / kTK;
  const Line line = make_line(a.delta, a.eps);
  for (int c = blockIdx.x; c < nc; c += gridDim.x) {
    double* out = wtab + (wofs[ft] + c) * (kTK * kFT);
    for (int idx = threadIdx.x; idx < kTK * kFT; idx += 256) {
      const int t = tr.x + c * kTK + idx / kFT, f = f_lo + idx % kFT;
      double v = 0.0;
      if (t < tr.y && f < a.nf && (a.window < 0 || abs(f - a.f0[t]) <= a.window)) v = line(a.dE[t] - a.dfreq * f);
      out[idx] = v;
    }
  }
}

template <int NCH>
constexpr size_t smem_bytes() {
  return sizeof(double2) * 2 * 2 * kAB * NCH * kTK + sizeof(double) * 2 * (kRows * kPLd + kTK * kWLd);
}

// element (e, t) of the staged overlaps, e = (side * 9 + a) * NCH + channel: the
// XOR spreads both the copies (consecutive e) and the reads (consecutive t) over
// the banks
__device__ __forceinline__ int midx(int e, int t) { return e * kTK + (t ^ (e & (kTK - 1))); }

}  // namespace

// WT: the line shape comes from wtab (chunk c of frequency tile ft at wofs[ft] + c),
// else it is formed here
template <int NCH, bool WT>
__global__ void __launch_bounds__(kThr, 2) contract64_kernel(ContractArgs a, const double* __restrict__ wtab,
                                                           const long long* __restrict__ wofs,
                                                           double* __restrict__ part) {
  int ta, tb;
  block_of(blockIdx.x, ta, tb);
  const int f_lo = blockIdx.y * kFT;
  const int A = 3 * a.neps;
  const int a0 = ta * kAB, b0 = tb * kAB;
  int2 tr = a.trange[blockIdx.y];
  const double* wsrc = WT ? wtab + wofs[blockIdx.y] * (kTK * kFT) : nullptr;
  if (gridDim.z > 1) {  // this CTA's share of the chunks
    const int nc = (tr.y - tr.x + kTK - 1) / kTK, per = (nc + gridDim.z - 1) / gridDim.z;
    const int t0 = tr.x + (int)blockIdx.z * per * kTK;
    if (WT) wsrc += (size_t)blockIdx.z * per * (kTK * kFT);
    tr = make_int2(min(t0, tr.y), min(t0 + per * kTK, tr.y));
  }
  constexpr int kElems = 2 * kAB * NCH;  // overlaps per transition
  extern __shared__ __align__(16) unsigned char smraw[];
  double2* sM = reinterpret_cast<double2*>(smraw);                       // [2][kElems][kTK]
  double* sP = reinterpret_cast<double*>(sM + 2 * kElems * kTK);         // [2][kRows][kPLd]
  double* sW = sP + 2 * kRows * kPLd;                                    // [2][kTK][kWLd]
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int gr = lane >> 2, gk = lane & 3;
  const int wm = wid % 3, wn = wid / 3;
  const Line line = make_line(a.delta, a.eps);
  double acc[kWM][kWN][2];
#pragma unroll
  for (int i = 0; i < kWM; ++i)
#pragma unroll
    for (int j = 0; j < kWN; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
  for (int idx = tid; idx < 2 * (kRows - 2 * kPairs) * kPLd; idx += kThr) {  // padding rows
    const int b = idx / ((kRows - 2 * kPairs) * kPLd), r = idx % ((kRows - 2 * kPairs) * kPLd);
    sP[b * kRows * kPLd + 2 * kPairs * kPLd + r] = 0.0;
  }
  // overlap e of the block is always copied by the same threads, kTPh transitions apart
  constexpr int kTPh = kThr / kElems;
  const int se = tid % kElems, st0 = tid / kElems;
  const int side = se / (kAB * NCH), sr = se - side * (kAB * NCH), sab = (side ? b0 : a0) + sr / NCH;
  const double2* ssrc = a.M + (size_t)min(sab, A - 1) * NCH + sr % NCH;
  auto stage_m = [&](int buf, int t0) {
    if (st0 < kTPh) {
      double2* dst = sM + buf * kElems * kTK;
#pragma unroll
      for (int t = st0; t < kTK; t += kTPh) {
        const bool ok = t0 + t < tr.y && sab < A;
        cp_async16_zfill(dst + midx(se, t), ssrc + (size_t)(ok ? t0 + t : 0) * A * NCH, ok);
      }
    }
    cp_async_commit();
  };
  auto stage_w = [&](int buf, int t0) {
    const double* src = wsrc + (size_t)((t0 - tr.x) / kTK) * (kTK * kFT);
    for (int idx = tid; idx < kTK * kFT / 2; idx += kThr)
      cp_async16(sW + buf * kTK * kWLd + (idx / (kFT / 2)) * kWLd + 2 * (idx % (kFT / 2)), src + 2 * idx);
    cp_async_commit();
  };
  // pair products: thread (transition pt, row pa of the block), nine pairs
  const int pt = tid & (kTK - 1), pa = tid / kTK;
  auto weight = [&](int t0) { return pa < kAB && t0 + pt < tr.y ? a.wgt[t0 + pt] : 0.0; };
  double w = weight(tr.x);
  if (tr.x < tr.y) {
    stage_m(0, tr.x);
    if (WT) stage_w(0, tr.x);
  }
  cp_async_wait<0>();
  __syncthreads();
  int buf = 0;
  for (int t0 = tr.x; t0 < tr.y; t0 += kTK, buf ^= 1) {
    if (t0 + kTK < tr.y) stage_m(buf ^ 1, t0 + kTK);
    double* P = sP + buf * kRows * kPLd;
    double* W = sW + buf * kTK * kWLd;
    const double wnext = weight(t0 + kTK);
    if (pa < kAB) {
      const double2* m = sM + buf * kElems * kTK;
      double2 va[NCH];
#pragma unroll
      for (int ch = 0; ch < NCH; ++ch) va[ch] = cscale(m[midx(pa * NCH + ch, pt)], w);
      const double2 sa = NCH == 1 ? va[0] : cadd(va[0], va[1 % NCH]);
      const double2 xa = cadd(va[2 % NCH], va[3 % NCH]);
      double* P1 = P + pa * kAB * kPLd + pt;
#pragma unroll
      for (int ib = 0; ib < kAB; ++ib) {
        double2 vb[NCH];
#pragma unroll
        for (int ch = 0; ch < NCH; ++ch) vb[ch] = m[midx((kAB + ib) * NCH + ch, pt)];
        double re, im;  // w reO, -w imO of a conj(b)
        if (NCH == 1) {
          re = va[0].x * vb[0].x + va[0].y * vb[0].y;
          im = va[0].x * vb[0].y - va[0].y * vb[0].x;
        } else {
          // up, down, updown, downup (src/pmx_chi.cpp:596-606): with S = up + down
          // and X = updown + downup, reO = Re(S_a S_b*) - Re(X_a X_b*);
          // imO = Im(up up* + down down* - updown updown* - downup downup*)
          const double2 sb = cadd(vb[0], vb[1 % NCH]), xb = cadd(vb[2 % NCH], vb[3 % NCH]);
          re = (sa.x * sb.x + sa.y * sb.y) - (xa.x * xb.x + xa.y * xb.y);
          im = (va[0].x * vb[0].y - va[0].y * vb[0].x) + (va[1 % NCH].x * vb[1 % NCH].y - va[1 % NCH].y * vb[1 % NCH].x) -
               (va[2 % NCH].x * vb[2 % NCH].y - va[2 % NCH].y * vb[2 % NCH].x) -
               (va[3 % NCH].x * vb[3 % NCH].y - va[3 % NCH].y * vb[3 % NCH].x);
        }
        P1[ib * kPLd] = re;
        P1[(kPairs + ib) * kPLd] = im;
      }
    }
    w = wnext;
    if (!WT) {  // line shape inside each transition's window
      for (int idx = tid; idx < kTK * kFT; idx += kThr) {
        const int t = idx / kFT, fl = idx % kFT, f = f_lo + fl;
        double v = 0.0;
        if (t0 + t < tr.y && f < a.nf && (a.window < 0 || abs(f - a.f0[t0 + t]) <= a.window))
          v = line(a.dE[t0 + t] - a.dfreq * f);
        W[t * kWLd + fl] = v;
      }
    }
    cp_async_wait<0>();
    __syncthreads();
    // every warp has left the previous chunk's products: its line-shape buffer is free
    if (WT && t0 + kTK < tr.y) stage_w(buf ^ 1, t0 + kTK);
    // ---- multiply. No barrier after it: the next chunk's products go into the other
    // buffer, and the barrier after them comes before this one is written again
    const double* Pa = P + (8 * kWM * wm + gr) * kPLd + gk;
    const double* Wb = W + gk * kWLd + 8 * kWN * wn + gr;
#pragma unroll
    for (int kk = 0; kk < kTK / 4; ++kk) {
      double av[kWM], bv[kWN];
#pragma unroll
      for (int i = 0; i < kWM; ++i) av[i] = Pa[8 * i * kPLd + 4 * kk];
#pragma unroll
      for (int j = 0; j < kWN; ++j) bv[j] = Wb[4 * kk * kWLd + 8 * j];
#pragma unroll
      for (int i = 0; i < kWM; ++i)
#pragma unroll
        for (int j = 0; j < kWN; ++j) dmma(acc[i][j][0], acc[i][j][1], av[i], bv[j]);
    }
  }
  // ---- store: rows 0..80 are the Im part (reO), 81..161 the Re part
  const size_t blk = (size_t)9 * a.np * a.nf;
  double* out = gridDim.z > 1 ? part + (size_t)blockIdx.z * 2 * blk : a.acc;
#pragma unroll
  for (int i = 0; i < kWM; ++i) {
    const int row = 8 * (kWM * wm + i) + gr;
    const int pp = row < kPairs ? row : row - kPairs;
    if (row >= 2 * kPairs) continue;
    const int av = a0 + pp / kAB, bv = b0 + pp % kAB;
    const int m = av / 3, ii = av % 3, nn = bv / 3, jj = bv % 3;
    if (m >= a.neps || nn > m) continue;
    double* o = out + (row < kPairs ? blk : 0) + ((size_t)(ii * 3 + jj) * a.np + (size_t)m * (m + 1) / 2 + nn) * a.nf;
#pragma unroll
    for (int j = 0; j < kWN; ++j) {
      const int f = f_lo + 8 * (kWN * wn + j) + 2 * gk;
      if (f < a.nf) o[f] = acc[i][j][0];
      if (f + 1 < a.nf) o[f + 1] = acc[i][j][1];
    }
  }
}

// the shares' sums in share order
__global__ void __launch_bounds__(256) contract64_sum_kernel(const double* __restrict__ part, double* __restrict__ acc,
                                                             size_t vals, int split) {
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < vals; i += (size_t)gridDim.x * blockDim.x) {
    double s = part[i];
    for (int z = 1; z < split; ++z) s += part[(size_t)z * vals + i];
    acc[i] = s;
  }
}

namespace {
int grid_blocks(const ContractArgs& a) {
  const int nb = (a.neps + kMB - 1) / kMB;
  return nb * (nb + 1) / 2;
}
}  // namespace

// Shares of the transitions per tile: few tiles (few local-field vectors or
// frequencies) leave SMs idle, so that their transitions are cut until about two
// waves of two CTAs per SM run, each with 8 chunks or more.
int contract64_split(const ContractArgs& a, long long T) {
  if (a.one_share) return 1;
  const long long ctas = (long long)grid_blocks(a) * ((a.nf + kFT - 1) / kFT);
  const long long want = (4 * 148 + ctas - 1) / std::max(1LL, ctas);
  return (int)std::max(1LL, std::min({want, (long long)kMaxSplit, T / (8 * kTK)}));
}

namespace {
size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }
size_t part_bytes(const ContractArgs& a, long long T) {
  const int z = contract64_split(a, T);
  return z > 1 ? align256(sizeof(double) * 2 * 9 * (size_t)a.np * a.nf * z) : 0;
}
// upper bound of the chunks of all frequency tiles: a window touches at most
// (2 window + 1 + 62) / 64 + 1 of them
size_t wtab_bytes(const ContractArgs& a, long long T) {
  const long long nft = (a.nf + kFT - 1) / kFT;
  const long long span = a.window < 0 ? nft : std::min<long long>(nft, (2LL * a.window + kFT) / kFT + 2);
  const long long chunks = (T * span + kTK - 1) / kTK + nft;
  return align256(sizeof(long long) * nft) + sizeof(double) * kTK * kFT * (size_t)chunks;
}
}  // namespace

// The shares' partial sums, and with `table` the line shapes: worth it where several
// pair blocks share them
size_t contract64_workspace_bytes(const ContractArgs& a, long long T, bool table) {
  return part_bytes(a, T) + (table ? wtab_bytes(a, T) : 0);
}
bool contract64_wants_table(const ContractArgs& a, long long T) {
  return grid_blocks(a) >= 3 && wtab_bytes(a, T) <= kMaxTable;
}

cudaError_t launch_contract64(const ContractArgs& a, long long T, void* ws, bool table, int& nlaunch,
                              cudaStream_t st) {
  const int split = contract64_split(a, T);
  const int nft = (a.nf + kFT - 1) / kFT;
  double* part = reinterpret_cast<double*>(ws);
  long long* wofs = reinterpret_cast<long long*>(reinterpret_cast<unsigned char*>(ws) + part_bytes(a, T));
  double* wtab = reinterpret_cast<double*>(reinterpret_cast<unsigned char*>(wofs) + align256(sizeof(long long) * nft));
  nlaunch = 1;
  if (table) {
    chunk_offsets_kernel<<<1, 1024, 0, st>>>(a.trange, nft, wofs);
    wtab_kernel<<<dim3((unsigned)std::min<long long>(std::max(1LL, T / kTK), 1024), nft), 256, 0, st>>>(a, wofs, wtab);
    nlaunch += 2;
  }
  const dim3 grid(grid_blocks(a), nft, split);
  auto kernel = a.nch == 1 ? (table ? contract64_kernel<1, true> : contract64_kernel<1, false>)
                           : (table ? contract64_kernel<4, true> : contract64_kernel<4, false>);
  const size_t sm = a.nch == 1 ? smem_bytes<1>() : smem_bytes<4>();
  const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  if (e != cudaSuccess) return e;
  kernel<<<grid, kThr, sm, st>>>(a, wtab, wofs, part);
  if (split > 1) {
    contract64_sum_kernel<<<592, 256, 0, st>>>(part, a.acc, (size_t)2 * 9 * a.np * a.nf, split);
    ++nlaunch;
  }
  return cudaGetLastError();
}

int contract_ftile() { return kFT; }

}  // namespace dev
}  // namespace pmx
