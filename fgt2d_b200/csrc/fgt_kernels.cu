// CUDA stages of the plane-wave FGT for sm_100a.
//
// (a) form     : per leaf, Hermite coefficients of its sources and the
//                Hermite -> plane-wave transform (g2dformhc_vec + g2dh2pw_real_vec,
//                g3dformhc_vec + g3dh2pw_real_vec), or the direct tensor-product
//                exponential sum (g3dformpwc_vec) where the reference uses it.
// (b) shifts   : diagonal plane-wave translations (g2dshiftpw_vec,
//                g2dcopypwexp_vec): mp -> loc over the plane-wave list here; merge
//                up to the cut level and split down to the leaves are parts of
//                the transforms (fgt_sep.cu, fgt_sep3d.cu).
// (c) eval     : per leaf, plane wave -> Taylor (g2dpw2local_real_vec) and
//                Taylor evaluation (g2dlevalp_vec), or direct plane-wave
//                evaluation (g2dpwevalp_vec) on the levels the reference picks.
// (d) direct   : near-field Gaussian sum with the reference cutoff
//                (g2d_directcp_vec / g3d_directcp_vec), target-centric.
//
// Expansions are complex FP64 in the reference layouts: 2D pw(npw/2, npw),
// 3D pw(npw, npw, npw/2), one block of nexp per (box slot, density).
#include <cuda_runtime.h>

#include <algorithm>
#include <chrono>
#include <exception>
#include <cstdio>
#include <cstdlib>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <mutex>
#include <type_traits>

#include "fgt_device.hpp"
#include "fgt_kcommon.cuh"
#include "fgt_sep.hpp"

namespace fgtb {

namespace {

// ------------------------------------------------------------ sort / unsort
// Tree order: out row i = in row perm[i] (dreorderf, fmmcommon2d.f:3-26);
// coordinates and charges of a point move together.
__global__ void k_gather_pts(const double* __restrict__ x, const double* __restrict__ q,
                             double* __restrict__ xs, double* __restrict__ qs,
                             const int* __restrict__ perm, int n, int dim, int nd, int vec) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const long long p = perm[i];
    if (x == nullptr) {
    } else if (dim == 2 && vec) {
      reinterpret_cast<double2*>(xs)[i] = reinterpret_cast<const double2*>(x)[p];
    } else {
      for (int d = 0; d < dim; d++) xs[(long long)i * dim + d] = x[p * dim + d];
    }
    if (q)
      for (int c = 0; c < nd; c++) qs[(long long)i * nd + c] = q[p * nd + c];
  }
}
// mp -> loc translation rows from their 1D factors (pw_translation_matrices):
// row s = (ox+1) + 3 (oy+1) [+ 9 (oz+1)], entry e = prod_d (o_d = 0 ? 1 :
// o_d > 0 ? w1 : conj(w1)) at e's node along d.  Products are formed left to
// right without contraction, (ac - bd, ad + bc).
__device__ __forceinline__ double2 cmul_rn(double2 a, double2 b) {
  return make_double2(__dsub_rn(__dmul_rn(a.x, b.x), __dmul_rn(a.y, b.y)),
                      __dadd_rn(__dmul_rn(a.x, b.y), __dmul_rn(a.y, b.x)));
}
__global__ void k_shift_tables(int dim, int npw, int nexp, const double2* __restrict__ w1,
                               double2* __restrict__ wsh) {
  const int n2 = npw / 2, total = (dim == 2 ? 9 : 27) * nexp;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
    const int s = i / nexp, e = i - s * nexp;
    const int node[3] = {dim == 2 ? e % n2 : e % npw, dim == 2 ? e / n2 : (e / npw) % npw, e / (npw * npw)};
    const int o[3] = {s % 3 - 1, (s / 3) % 3 - 1, s / 9 - 1};
    double2 f = make_double2(1.0, 0.0);
    for (int d = 0; d < dim; d++) {
      double2 v = o[d] == 0 ? make_double2(1.0, 0.0) : w1[node[d]];
      if (o[d] < 0) v.y = -v.y;
      f = cmul_rn(f, v);
    }
    wsh[i] = f;
  }
}

// *bad = 1 when any of x[0, n) is not finite
__global__ void k_all_finite(const double* __restrict__ x, size_t n, int* __restrict__ bad) {
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    if (!isfinite(x[i])) *bad = 1;
}
// qs[i] = q[perm[i]] for one density (the charges of every execute): four
// independent random reads in flight per thread
__global__ void __launch_bounds__(256) k_gather1(const double* __restrict__ q, const int* __restrict__ perm, int n,
                                                 double* __restrict__ qs) {
  const int stride = gridDim.x * blockDim.x;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += 4 * stride) {
    int p[4];
    double v[4];
#pragma unroll
    for (int u = 0; u < 4; u++) p[u] = i + u * stride < n ? perm[i + u * stride] : -1;
#pragma unroll
    for (int u = 0; u < 4; u++) v[u] = p[u] >= 0 ? q[p[u]] : 0.0;
#pragma unroll
    for (int u = 0; u < 4; u++)
      if (p[u] >= 0) qs[i + u * stride] = v[u];
  }
}
// inv[perm[i]] = i
__global__ void k_invperm(const int* __restrict__ perm, int n, int* __restrict__ inv) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) inv[perm[i]] = i;
}
// Caller order: out row j = in row iperm[j] (dreorderi / dreorderiv,
// fmmcommon2d.f:29-90), written as a gather so the stores stay coalesced.  A
// sorted row holds the potentials, gradients and Hessians of a point (w0, w1,
// w2 values); each goes to its own array (null: skipped).  A thread per value,
// so a row's random read is one access for all three (an array at a time, the
// rows of 3e5 + 1e5 points with Hessians took 27 us, 15 us this way).
__global__ void __launch_bounds__(256) k_unsort(const double* __restrict__ in, const int* __restrict__ iperm, int n,
                                                int w0, int w1, int w2, double* __restrict__ o0,
                                                double* __restrict__ o1, double* __restrict__ o2) {
  const unsigned w = w0 + w1 + w2;
  const long long total = (long long)n * w;
  for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < total;
       t += (long long)gridDim.x * blockDim.x) {
    const long long j = total < (1LL << 31) ? (unsigned)t / w : t / w;
    const int e = (int)(t - j * w);
    const double v = in[(long long)iperm[j] * w + e];
    if (e < w0) {
      if (o0) o0[j * w0 + e] = v;
    } else if (e < w0 + w1) {
      if (o1) o1[j * w1 + e - w0] = v;
    } else if (o2) {
      o2[j * w2 + e - w0 - w1] = v;
    }
  }
}

// ------------------------------------------------------------ (a) form, 2D on FP64 MMA
// Hermite block of a leaf, H[j][k] = sum_t q_t x_t^j y_t^k (g2dformhc_vec,
// g2drouts.f:100-168, without the 1/sqrt(j! k!) factors, which the
// Hermite -> plane-wave table carries), on the FP64 tensor cores: mma.sync.m8n8k4.f64 takes
// four sources per step (K = 4) into NT x NT tiles of 8 x 8 (P <= 8 NT).
// Fragment layout (PTX ISA, m8n8k4 .f64): A element (row = lane/4, col =
// lane%4), B element (row = lane%4, col = lane/4), accumulator pair (row =
// lane/4, col = 2 (lane%4) + i).  The powers x^j and q y^j of a block of 32
// sources are built once per source (one lane each) in a per-warp
// shared-memory stage laid out [j][source] with a row stride of 36 doubles, so
// each fragment load is two conflict-free wavefronts.  Four warps split the
// leaf's sources; their tiles are summed in shared memory and the P x P block
// goes to the leaf's slot of the Hermite buffer.
// With dipoles (DIP) the source derivative enters as a second column per
// source (g2dformhd_vec / g2dformhcd_vec, g2drouts.f:173-338; in the
// unnormalised powers here d/dX x^j = j dsq x^(j-1)):
//   column 0: X = x^j,               Y = q y^k + v2 k dsq y^(k-1)
//   column 1: X = v1 j dsq x^(j-1),  Y = y^k
// (v = dipstr * n), so a block of 32 columns holds 16 sources.
// WARP: a task per warp instead of per CTA, for leaves of few sources (two
// blocks of columns or less per leaf left half of the CTA's warps idle and the
// other half waiting for the final sum): 3e5 sources, 19 a leaf, order 21, 69 ->
// 25 us; 1e5, 52 a leaf, order 30, 47 -> 16; dipoles of two densities, 2e5
// sources, 26 a leaf, 133 -> 57.
template <int NT, bool DIP, bool WARP>
__global__ void __launch_bounds__(128) k_form2d_mma(KP k, const FormTask* __restrict__ tasks, int ntask,
                                                    const long long* __restrict__ hoff,
                                                    double* __restrict__ hbuf) {
  constexpr int PP = 8 * NT, SW = 36, WS = 2 * PP * SW;  // per-warp staging [2][PP][SW]
  const int task = WARP ? blockIdx.x * 4 + (threadIdx.x >> 5) : blockIdx.x;
  if (WARP && task >= ntask) return;  // no CTA-wide barrier on this path
  const FormTask T = tasks[task];
  const int ind = blockIdx.y;
  const int Pn = T.p + 1;
  // the CTA's PP x PP block of H (orders beyond PP take several)
  const int nb = (Pn + PP - 1) / PP, jb = PP * (blockIdx.z / nb), kb = PP * (blockIdx.z % nb);
  extern __shared__ double smf[];
  double* stg = smf;                                          // [4][WS]
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const double cx = k.centers[2 * T.box], cy = k.centers[2 * T.box + 1];
  const int j0 = lane >> 2, tl = lane & 3;
  double* X = stg + warp * WS;  // X[j][s] = x_s^j, Y[j][s] = q_s y_s^j
  double* Y = X + PP * SW;
  double c[2][NT][NT][2];
#pragma unroll
  for (int h = 0; h < 2; h++)
#pragma unroll
    for (int a = 0; a < NT; a++)
#pragma unroll
      for (int b = 0; b < NT; b++) c[h][a][b][0] = c[h][a][b][1] = 0.0;
  // each warp takes blocks of 32 sources in turn: every lane builds the
  // powers of one source in shared memory, then the warp runs up to eight
  // K = 4 steps of the FP64 MMA over the block, alternating two accumulator
  // sets so consecutive steps are independent
  constexpr int SPB = DIP ? 16 : 32;  // sources per 32-column block
  for (int base = WARP ? 0 : SPB * warp; base < T.n; base += WARP ? SPB : 4 * SPB) {
    const int sl = DIP ? lane >> 1 : lane;
    double x = 0.0, y = 0.0, q = 0.0, v[2] = {0.0, 0.0};
    if (base + sl < T.n) {
      const int i = T.s0 + base + sl;
      const double2 pt = reinterpret_cast<const double2*>(k.src)[i];
      x = (pt.x - cx) * k.dsq;
      y = (pt.y - cy) * k.dsq;
      if (DIP) {
        q = src_charge(k, i, ind);
        src_dipole<2>(k, i, ind, v);
      } else {
        q = k.chg[(size_t)i * k.nd + ind];
      }
    }
    if (!DIP) {
      double xp = 1.0, yp = q;
      for (int j = 0; j < jb; j++) xp *= x;
      for (int j = 0; j < kb; j++) yp *= y;
#pragma unroll
      for (int j = 0; j < PP; j++) {
        X[j * SW + lane] = xp;
        Y[j * SW + lane] = yp;
        xp *= x;
        yp *= y;
      }
    } else {
      // column (lane & 1): powers and their derivatives, one pass
      const bool c1 = lane & 1;
      const double ax = c1 ? 0.0 : 1.0, bx = c1 ? v[0] * k.dsq : 0.0;
      const double ay = c1 ? 1.0 : q, by = c1 ? 0.0 : v[1] * k.dsq;
      double xp = 1.0, yp = 1.0, xm = 0.0, ym = 0.0;  // x^j, j x^(j-1)
      for (int j = 0; j < jb; j++) {
        xm = fma(xm, x, xp);
        xp *= x;
      }
      for (int j = 0; j < kb; j++) {
        ym = fma(ym, y, yp);
        yp *= y;
      }
#pragma unroll
      for (int j = 0; j < PP; j++) {
        X[j * SW + lane] = fma(ax, xp, bx * xm);
        Y[j * SW + lane] = fma(ay, yp, by * ym);
        xm = fma(xm, x, xp);  // (j+1) x^j = j x^(j-1) x + x^j
        ym = fma(ym, y, yp);
        xp *= x;
        yp *= y;
      }
    }
    __syncwarp();
    const int ncol = DIP ? 2 * min(SPB, T.n - base) : T.n - base;
    const int nst = min(8, (ncol + 3) >> 2);
    for (int st = 0; st < nst; st += 2) {
#pragma unroll
      for (int h = 0; h < 2; h++) {
        if (st + h < nst) {
          const int col = 4 * (st + h) + tl;
          double av[NT], bv[NT];
#pragma unroll
          for (int a = 0; a < NT; a++) {
            av[a] = X[(8 * a + j0) * SW + col];
            bv[a] = Y[(8 * a + j0) * SW + col];
          }
#pragma unroll
          for (int a = 0; a < NT; a++)
#pragma unroll
            for (int b = 0; b < NT; b++) dmma_884(c[h][a][b][0], c[h][a][b][1], av[a], bv[b]);
        }
      }
    }
    __syncwarp();
  }
  // tile (a, b) holds H'[j = 8a + lane/4][k = 8b + 2 (lane%4) + i]; each warp
  // writes its sum into its own staging area, then the four are added and
  // the leaf's P x P block is stored row-major (x power j, y power k)
  double* hb = hbuf + hoff[task] + (size_t)ind * Pn * Pn;
  if (WARP) {
#pragma unroll
    for (int a = 0; a < NT; a++)
#pragma unroll
      for (int b = 0; b < NT; b++)
#pragma unroll
        for (int i = 0; i < 2; i++) {
          const int j = jb + 8 * a + j0, kk = kb + 8 * b + 2 * tl + i;
          if (j < Pn && kk < Pn) hb[j * Pn + kk] = c[0][a][b][i] + c[1][a][b][i];
        }
    return;
  }
  double* part = X;
#pragma unroll
  for (int a = 0; a < NT; a++)
#pragma unroll
    for (int b = 0; b < NT; b++)
#pragma unroll
      for (int i = 0; i < 2; i++)
        part[(8 * a + j0) + PP * (8 * b + 2 * tl + i)] = c[0][a][b][i] + c[1][a][b][i];
  __syncthreads();
  const int nj = min(PP, Pn - jb), nk = min(PP, Pn - kb);
  for (int e = threadIdx.x; e < nj * nk; e += 128) {
    const int j = e / nk, kk = e - j * nk, f = j + PP * kk;
    hb[(jb + j) * Pn + kb + kk] = stg[f] + stg[WS + f] + stg[2 * WS + f] + stg[3 * WS + f];
  }
}

// A leaf's partial Hermite blocks (one after the other, n of them) added into
// the first: 32 coefficients per CTA, eight threads each with every eighth
// block (a thread alone waits for hundreds of loads in a row: 37 us instead of
// 5 at 586 blocks), added in a fixed order.  In 2D all leaves of several
// blocks; in 3D those of more than SUM_BLOCKS3D, since k_up_z adds blocks as it
// reads them, 1.7 us each in a row but beside the other columns, and the launch
// costs 4 to 7 (one leaf of 595 blocks among 1e6 sources, order 7 and 13: 1764
// and 4303 us added there, 854 and 3189 here; of 126, 6e4 sources: 197 and 330,
// 107 and 297; of 21: 109 and 302, 97 and 306; blob leaves of 9 to 16, forces:
// 1720 and 1728).
constexpr int SUM_BLOCKS3D = 32;
__global__ void __launch_bounds__(256) k_sum_blocks(const BlockSum* __restrict__ sums, int nd,
                                                    double* __restrict__ hbuf) {
  __shared__ double part[8][32];
  const BlockSum S = sums[blockIdx.x];
  const int len = S.len * nd, x = threadIdx.x & 31, w = threadIdx.x >> 5;
  double* h = hbuf + S.off;
  for (int e0 = 32 * blockIdx.y; e0 < len; e0 += 32 * gridDim.y) {
    double a = 0.0;
    if (e0 + x < len) {
#pragma unroll 4
      for (int b = w; b < S.n; b += 8) a += h[(size_t)b * len + e0 + x];
    }
    part[w][x] = a;
    __syncthreads();
    if (w == 0 && e0 + x < len) {
#pragma unroll
      for (int i = 1; i < 8; i++) a += part[i][x];
      h[e0 + x] = a;
    }
    __syncthreads();
  }
}

// ------------------------------------------------------------ (a) form, 3D
// One CTA per chunk of at most form_chunk sources of a leaf accumulates the chunk's
// Hermite block H[j + P (k + P l)] (g3dformhc_vec, g3drouts.f:109-192) and
// writes it to its slot of the partial buffer; fgt_sep3d.cu sums a leaf's
// blocks in chunk order and takes them to the cut level's expansions.

// The chunk's Hermite block on the FP64 tensor cores: H[j][(k, l)] =
// sum_t x_t^j (q_t y_t^k z_t^l) (with the 1/sqrt(j!) factors, g3dformhc_vec,
// g3drouts.f:109-192) is one product with M = j (MT tiles of 8), N = the
// P^2 pairs (k, l) and K = the sources, four per mma.m8n8k4 step.  A column
// tile is four k by two l: its B fragment is y^k q z^l, one multiply of a y
// fragment that serves every l of the warp and a z fragment that serves every
// k, so a step of KQ x NLP tiles loads KQ + NLP + MT operands for MT KQ NLP
// products, each load one or two wavefronts (rows of 44 doubles; tiles of
// eight consecutive (k, l) straddled rows and conflicted at every order that
// is no multiple of four).  The warps take the l pairs in turn, starting with
// another one in every CTA (warp w always runs on sub-partition w mod 4);
// KQ quads of k per pass over the sources.  Sources are staged 40 at a time
// as power rows (one thread per source and dimension, the next batch's
// coordinates loaded while this one is summed).  The partial block goes to
// the chunk's slot of the Hermite buffer, laid out H[j + P (k + P l)] as
// k_up_z reads it.  Bound by the tensor pipe (16 cycles per product and
// sub-partition).
// Measured (order 13, eps 1e-6): 4e6 sources in leaves of 115, 1.56 ms with
// eight consecutive columns per tile and eight warps, 1.37 ms; 2e6 in leaves
// of 1157, 0.68 -> 0.66 (65% of the pipe, the rest mostly the tail of three
// waves of CTAs); 1.5e5 of order 15, 0.24 -> 0.09; 3e5 of order 19 at eps
// 1e-9, 0.51 -> 0.38.  Orders above 15 take fewer quads per pass: with three,
// 176 registers left eight warps on an SM and cost more than the passes.
// With dipoles (DIP) every source stages three columns (dip3_coef), 13
// sources (39 columns) per batch.
constexpr int FORM3_SB = 40, FORM3_SW = 44;
// quads of k per pass and pairs of l per warp at MT row tiles
__host__ __device__ constexpr int form3_kq(int P) { return P <= 8 ? 2 : P <= 12 ? 3 : P <= 16 ? 4 : P <= 24 ? 2 : 1; }
__host__ __device__ constexpr int form3_nlp(int P) { return P <= 8 ? 1 : P <= 16 ? 2 : P <= 24 ? 3 : 4; }
size_t form3_smem(int Pn) {
  return (size_t)(8 * ((Pn + 7) / 8) + 4 * ((Pn + 3) / 4) + 2 * ((Pn + 1) / 2)) * FORM3_SW * 8;
}

template <int MT, int KQ, int NLP, bool DIP>
__global__ void __launch_bounds__(128) k_form3d_mma(KP k, const FormTask* __restrict__ tasks,
                                                    const FormChunk* __restrict__ chunks,
                                                    double* __restrict__ hbuf, const double* __restrict__ isq) {
  constexpr int SB = FORM3_SB, SW = FORM3_SW;
  constexpr int VC = DIP ? 3 : 1, SBS = SB / VC;  // columns per source, sources per batch
  const FormChunk C = chunks[blockIdx.x];
  const FormTask T = tasks[C.task];
  const int ind = blockIdx.y;
  const int Pn = T.p + 1, P2 = Pn * Pn, P3 = P2 * Pn, nkq = (Pn + 3) / 4, nlp = (Pn + 1) / 2;
  extern __shared__ double sm[];
  double* X = sm;                // [8 MT][SW]
  double* Y = X + 8 * MT * SW;   // [4 nkq][SW]
  double* Z = Y + 4 * nkq * SW;  // [2 nlp][SW], times q
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, r = lane >> 2, c = lane & 3;
  const int lp0 = (warp + blockIdx.x) & 3;  // the warp's l pairs: lp0 + 4 i
  for (int e = tid; e < (8 * MT + 4 * nkq + 2 * nlp) * SW; e += 128) sm[e] = 0.0;  // rows past the order stay zero
  const int d = tid / SB, t = tid - SB * d;  // staging job
  const bool job = tid < 3 * SB;
  double* const row = (d == 0 ? X : d == 1 ? Y : Z) + t;
  const double cen = k.centers[3 * T.box + (job ? d : 0)];
  auto fetch = [&](int c0, double& u, double& q) {
    u = cen;
    q = 0.0;
    if (job && c0 + t < C.n && !DIP) {
      const size_t i = (size_t)C.s0 + c0 + t;
      u = k.src[3 * i + d];
      q = d == 2 ? k.chg[i * k.nd + ind] : 1.0;
    }
  };
  double* out = hbuf + ((size_t)C.hoff * k.nd + (size_t)ind * P3);
  for (int kq0 = 0; kq0 < nkq; kq0 += KQ) {
    double acc[KQ][NLP][MT][2];
#pragma unroll
    for (int g = 0; g < KQ; g++)
#pragma unroll
      for (int i = 0; i < NLP; i++)
#pragma unroll
        for (int mt = 0; mt < MT; mt++) acc[g][i][mt][0] = acc[g][i][mt][1] = 0.0;
    double un, qn;
    fetch(0, un, qn);
    for (int c0 = 0; c0 < C.n; c0 += SBS) {
      const int m = VC * min(SBS, C.n - c0);
      __syncthreads();
      if (job) {
        if (!DIP) {
          const double v = (un - cen) * k.dsq;
          double w = qn;
          row[0] = w;
#pragma unroll 4
          for (int j = 1; j < Pn; j++) {
            w *= v * __ldg(isq + j);
            row[j * SW] = w;
          }
        } else {
          double v = 0.0, a = 0.0, b = 0.0;
          if (t < m) {
            const int i = C.s0 + c0 + t / VC;
            v = (k.src[(size_t)3 * i + d] - cen) * k.dsq;
            double dv[3];
            src_dipole<3>(k, i, ind, dv);
            dip3_coef(t % VC, d, src_charge(k, i, ind), dv, a, b);
          }
          dip_row(row, SW, Pn, v, a, b, k.dsq, isq);
        }
      }
      fetch(c0 + SBS, un, qn);
      __syncthreads();
      const int nst = (m + 3) >> 2;
      const double* xp = X + r * SW + c;
      const double* yp = Y + (4 * kq0 + (r & 3)) * SW + c;
      const double* zp = Z + (2 * lp0 + (r >> 2)) * SW + c;
      for (int st = 0; st < nst; st++) {
        double a[MT], y[KQ], z[NLP];
#pragma unroll
        for (int mt = 0; mt < MT; mt++) a[mt] = xp[8 * mt * SW + 4 * st];
#pragma unroll
        for (int g = 0; g < KQ; g++) y[g] = kq0 + g < nkq ? yp[4 * g * SW + 4 * st] : 0.0;
#pragma unroll
        for (int i = 0; i < NLP; i++) {
          if (lp0 + 4 * i < nlp) {
            z[i] = zp[8 * i * SW + 4 * st];
#pragma unroll
            for (int g = 0; g < KQ; g++)
              if (kq0 + g < nkq) {
                const double b = y[g] * z[i];
#pragma unroll
                for (int mt = 0; mt < MT; mt++) dmma_884(acc[g][i][mt][0], acc[g][i][mt][1], a[mt], b);
              }
          }
        }
      }
    }
    // the lane's columns 2 c, 2 c + 1 of a tile: k = 4 (kq0 + g) + (2 c & 3) + {0, 1}, l = 2 (lp0 + 4 i) + c / 2
#pragma unroll
    for (int g = 0; g < KQ; g++)
#pragma unroll
      for (int i = 0; i < NLP; i++) {
        const int kk = 4 * (kq0 + g) + ((2 * c) & 3), l = 2 * (lp0 + 4 * i) + (c >> 1);
#pragma unroll
        for (int mt = 0; mt < MT; mt++) {
          const int j = 8 * mt + r;
          if (j < Pn && l < Pn) {
            if (kk < Pn) out[j + Pn * (kk + Pn * l)] = acc[g][i][mt][0];
            if (kk + 1 < Pn) out[j + Pn * (kk + 1 + Pn * l)] = acc[g][i][mt][1];
          }
        }
      }
  }
}

// ------------------------------------------------------------ (c) eval, 2D Taylor blocks
// FP64 evaluation of a leaf's Taylor block lo[b][a] (P rows of E = P rounded up
// to even, y^b x^a; g2dlevalp/g/h_vec, g2drouts.f:847-1085), orders 24 to 39:
//   pot = sum_b y^b C[b],  C[b] = sum_a x^a lo[b][a],
// the inner sum as a product on the FP64 tensor cores, eight points as rows
// (x^a and, for derivatives, a x^(a-1) and a (a-1) x^(a-2): PGH row sets on
// the same columns), K = a in KS steps of four, the columns b; the lane then
// folds its two columns of its point into the sums with y^b and its
// derivatives.  A warp owns 8 MT points and keeps their row sets in
// registers, the block comes from global memory (L1) straight into the
// fragments; a task has one, two or four warps by its points.
// MMA and FMA have the same FP64 rate and the MMA pads P to 4 and 8; what it
// saves against Horner (below, a thread per point) is the idle threads of
// leaves of a few dozen points and the block's passes through shared memory.
// Both, potentials (with gradients; with Hessians), 1e5 uniform points, eps
// 1e-9, order 30-33, 52 points a task: 21 (41; 70) us here, 35 (65; 98) Horner;
// order 24, 35 points: 45 and 56; but order 18-21, 52 points: 49 (102; 147)
// and 41 (84; 125); 26 points: 38 (85; 112) and 38 (65; 94).  So Horner keeps
// the orders below 24, and the tasks of more than 72 points on average
// (order 24, 67 points: 78 and 82; order 19, 237 points: 45 and 25).
template <int KS, int PGH>
__global__ void __launch_bounds__(128) k_eval2d_mma(KP k, const HornerTask* __restrict__ tasks, int ntask, int per,
                                                    const double* __restrict__ lo_all) {
  constexpr int NC = ncomp<2, PGH>(), MT = PGH == 1 ? 2 : 1;
  const int w = blockIdx.x * 4 + (threadIdx.x >> 5);
  if (w >= ntask * per) return;  // no CTA-wide barrier in this kernel
  const int warp = w & (per - 1);
  const HornerTask T = tasks[w / per];
  const int ind = blockIdx.y, Pn = T.p + 1, E = (Pn + 1) & ~1;
  const int lane = threadIdx.x & 31, r = lane >> 2, c = lane & 3;
  const double* lo = lo_all + T.off + (size_t)ind * Pn * E;
  const double2* pts = reinterpret_cast<const double2*>(T.set ? k.trg : k.src);
  double* out = T.set ? k.pottarg : k.pot;
  const int nc = T.set ? k.nc_t : k.nc_s;
  const double cx = k.centers[2 * T.box], cy = k.centers[2 * T.box + 1];
  for (int p0 = 8 * MT * warp; p0 < T.n; p0 += 8 * MT * per) {
    double x[PGH][MT][KS];  // the lane's row entries a = 4 s + c
    double yb[MT], ym[MT], yl[MT], y8[MT], y1[MT];
#pragma unroll
    for (int i = 0; i < MT; i++) {
      const double2 p = pts[T.i0 + min(p0 + 8 * i + r, T.n - 1)];
      const double u = (p.x - cx) * k.dsq, v = (p.y - cy) * k.dsq;
      const double u2 = u * u, u4 = u2 * u2;
      double q0 = c == 0 ? 1.0 : c == 1 ? u : c == 2 ? u2 : u2 * u;  // u^a
      double q1 = c == 0 ? 0.0 : c == 1 ? 1.0 : c == 2 ? u : u2;     // u^(a-1)
      double q2 = c < 2 ? 0.0 : c == 2 ? 1.0 : u;                    // u^(a-2)
#pragma unroll
      for (int s = 0; s < KS; s++) {
        const int a = 4 * s + c;
        const bool in = a < Pn;
        x[0][i][s] = in ? q0 : 0.0;
        if (PGH >= 2) x[PGH >= 2 ? 1 : 0][i][s] = in ? a * q1 : 0.0;
        if (PGH >= 3) x[PGH >= 3 ? 2 : 0][i][s] = in ? a * (a - 1) * q2 : 0.0;
        q1 = s == 0 && c == 0 ? u2 * u : q1 * u4;
        q2 = s == 0 && c < 2 ? (c == 0 ? u2 : u2 * u) : q2 * u4;
        q0 *= u4;
      }
      // the columns b = 8 nt + 2 c and b + 1: y^b, y^(b-1), y^(b-2)
      const double v2 = v * v, v4 = v2 * v2;
      y1[i] = v;
      y8[i] = v4 * v4;
      yb[i] = c == 0 ? 1.0 : c == 1 ? v2 : c == 2 ? v4 : v4 * v2;
      ym[i] = c == 0 ? 0.0 : c == 1 ? v : c == 2 ? v2 * v : v4 * v;
      yl[i] = c == 0 ? 0.0 : c == 1 ? 1.0 : c == 2 ? v2 : v4;
    }
    double sum[MT][NC];
#pragma unroll
    for (int i = 0; i < MT; i++)
#pragma unroll
      for (int v = 0; v < NC; v++) sum[i][v] = 0.0;
    for (int nt = 0; 8 * nt < Pn; nt++) {
      const double* row = lo + min(8 * nt + r, Pn - 1) * E;
      double b[KS];
#pragma unroll
      for (int s = 0; s < KS; s++) b[s] = row[min(4 * s + c, E - 1)];
      double acc[PGH][MT][2];
#pragma unroll
      for (int g = 0; g < PGH; g++)
#pragma unroll
        for (int i = 0; i < MT; i++) acc[g][i][0] = acc[g][i][1] = 0.0;
#pragma unroll
      for (int s = 0; s < KS; s++)
#pragma unroll
        for (int g = 0; g < PGH; g++)
#pragma unroll
          for (int i = 0; i < MT; i++) dmma_884(acc[g][i][0], acc[g][i][1], x[g][i][s], b[s]);
      const int bb = 8 * nt + 2 * c;
      const double f0 = bb < Pn ? 1.0 : 0.0, f1 = bb + 1 < Pn ? 1.0 : 0.0;  // columns past the block
#pragma unroll
      for (int i = 0; i < MT; i++) {
        const double w0 = f0 * yb[i], w1 = f1 * yb[i] * y1[i];
        sum[i][0] = fma(acc[0][i][0], w0, fma(acc[0][i][1], w1, sum[i][0]));
        if constexpr (PGH >= 2) {
          const double d0 = f0 * bb * ym[i], d1 = f1 * (bb + 1) * yb[i];
          sum[i][1] = fma(acc[1][i][0], w0, fma(acc[1][i][1], w1, sum[i][1]));
          sum[i][2] = fma(acc[0][i][0], d0, fma(acc[0][i][1], d1, sum[i][2]));
          if constexpr (PGH >= 3) {
            const double h0 = f0 * bb * (bb - 1) * yl[i], h1 = f1 * (bb + 1) * bb * ym[i];
            sum[i][3] = fma(acc[2][i][0], w0, fma(acc[2][i][1], w1, sum[i][3]));
            sum[i][4] = fma(acc[1][i][0], d0, fma(acc[1][i][1], d1, sum[i][4]));
            sum[i][5] = fma(acc[0][i][0], h0, fma(acc[0][i][1], h1, sum[i][5]));
          }
        }
        // the next eight columns
        const double v = y1[i], v2 = v * v, v4 = v2 * v2;
        yl[i] = nt == 0 && c == 0 ? v4 * v2 : yl[i] * y8[i];
        ym[i] = nt == 0 && c == 0 ? v4 * v2 * v : ym[i] * y8[i];
        yb[i] *= y8[i];
      }
    }
#pragma unroll
    for (int i = 0; i < MT; i++) {
      const int pt = p0 + 8 * i + r;
#pragma unroll
      for (int v = 0; v < NC; v++) {
        double a = sum[i][v];
        a += __shfl_xor_sync(FULL_MASK, a, 1);
        a += __shfl_xor_sync(FULL_MASK, a, 2);
        if ((v & 3) == c && pt < T.n && v < nc)
          out[((size_t)(T.i0 + pt) * nc + v) * k.nd + ind] += a * (v == 0 ? 1.0 : v < 3 ? k.dsq : k.dsq * k.dsq);
      }
    }
  }
}

// k_eval2d_horner: one CTA (128 threads) per chunk of <= 256 points of an
// evaluation leaf; the leaf's Taylor block (P rows of E = 2 NP2) is staged in
// shared memory and each thread evaluates two points (g2dlevalp_vec,
// g2drouts.f:847-900):
//     pot += sum_k1 y^k1 sum_k2 lo[k1][k2] x^k2,
// Horner in x along each row (coefficient pairs read as double2), then in y.
// Plain FP64 FMAs: on B200 the FP64 FMA pipe and the FP64 MMA share one
// throughput, and Horner at the exact order does P (E - 1) + P FMAs a point
// where the 8 x 8 x 4 MMA pads P up to a multiple of 8 in both dimensions.
// PGH > 1 carries the derivative chains of the Horner sums (hstep, hrow),
// the gradient and Hessian of g2dlevalg_vec / g2dlevalh_vec
// (g2drouts.f:905-1085).
template <int NP2, int PGH>
__global__ void __launch_bounds__(128) k_eval2d_horner(KP k, const HornerTask* __restrict__ tasks,
                                                       const double* __restrict__ lo_all) {
  constexpr int NC = ncomp<2, PGH>();
  const HornerTask T = tasks[blockIdx.x];
  const int ind = blockIdx.y, Pn = T.p + 1;
  extern __shared__ double2 lo2[];  // [Pn][NP2]
  const double2* src = reinterpret_cast<const double2*>(lo_all + T.off + (size_t)ind * Pn * 2 * NP2);
  for (int e = threadIdx.x; e < Pn * NP2; e += blockDim.x) lo2[e] = src[e];
  __syncthreads();
  const double* pts = T.set ? k.trg : k.src;
  double* out = T.set ? k.pottarg : k.pot;
  const int nc = T.set ? k.nc_t : k.nc_s;
  const double cx = k.centers[2 * T.box], cy = k.centers[2 * T.box + 1];
  const int ta = threadIdx.x, tb = threadIdx.x + 128;
  if (ta >= T.n) return;
  const bool two = tb < T.n;
  const double2 pa = reinterpret_cast<const double2*>(pts)[T.i0 + ta];
  const double2 pb = reinterpret_cast<const double2*>(pts)[T.i0 + (two ? tb : ta)];
  const double x0 = (pa.x - cx) * k.dsq, y0 = (pa.y - cy) * k.dsq;
  const double x1 = (pb.x - cx) * k.dsq, y1 = (pb.y - cy) * k.dsq;
  Hor2 a0, a1;
  for (int k1 = Pn - 1; k1 >= 0; k1--) {
    const double2* rw = lo2 + k1 * NP2;
    const double2 ct = rw[NP2 - 1];
    double s0 = ct.y, s1 = ct.y, u0 = 0.0, u1 = 0.0, w0 = 0.0, w1 = 0.0;
    hstep<PGH>(s0, u0, w0, x0, ct.x);
    hstep<PGH>(s1, u1, w1, x1, ct.x);
#pragma unroll
    for (int m = NP2 - 2; m >= 0; m--) {
      const double2 c = rw[m];
      hstep<PGH>(s0, u0, w0, x0, c.y);
      hstep<PGH>(s1, u1, w1, x1, c.y);
      hstep<PGH>(s0, u0, w0, x0, c.x);
      hstep<PGH>(s1, u1, w1, x1, c.x);
    }
    hrow<PGH>(a0, y0, s0, u0, w0);
    hrow<PGH>(a1, y1, s1, u1, w1);
  }
  double v[NC];
  hemit<PGH>(a0, k.dsq, v);
  add_out<NC>(out, T.i0 + ta, k.nd, nc, ind, v);
  if (two) {
    hemit<PGH>(a1, k.dsq, v);
    add_out<NC>(out, T.i0 + tb, k.nd, nc, ind, v);
  }
}

// Orders above 64 (rows longer than 64): the same evaluation with a runtime
// row length.
template <int PGH>
__global__ void __launch_bounds__(128) k_eval2d_horner_any(KP k, const HornerTask* __restrict__ tasks,
                                                           const double* __restrict__ lo_all) {
  constexpr int NC = ncomp<2, PGH>();
  const HornerTask T = tasks[blockIdx.x];
  const int ind = blockIdx.y, Pn = T.p + 1, E = (Pn + 1) & ~1;
  extern __shared__ double lo1[];  // [Pn][E]
  const double* src = lo_all + T.off + (size_t)ind * Pn * E;
  for (int e = threadIdx.x; e < Pn * E; e += blockDim.x) lo1[e] = src[e];
  __syncthreads();
  const double* pts = T.set ? k.trg : k.src;
  double* out = T.set ? k.pottarg : k.pot;
  const int nc = T.set ? k.nc_t : k.nc_s;
  const double cx = k.centers[2 * T.box], cy = k.centers[2 * T.box + 1];
  for (int t = threadIdx.x; t < T.n; t += blockDim.x) {
    const double2 pa = reinterpret_cast<const double2*>(pts)[T.i0 + t];
    double v[NC];
    horner2_rt<PGH>(lo1, E, Pn, (pa.x - cx) * k.dsq, (pa.y - cy) * k.dsq, k.dsq, v);
    add_out<NC>(out, T.i0 + t, k.nd, nc, ind, v);
  }
}

// ------------------------------------------------------------ (c) eval, 3D Taylor blocks
// k_eval3d_horner: one CTA (128 threads) per chunk of <= 256 points of an
// evaluation leaf; the leaf's Taylor block lo[c][b][a] (rows of E = 2 NP2)
// is staged in shared memory and each thread evaluates two points by Horner
// in x along each row, then in y, then in z (g3dlevalp_vec,
// g3drouts.f:1045-1107), plain FP64 FMAs at the exact order.
// Horner over the planes and rows of a staged block for NPT points at once,
// NR rows of a plane in flight (independent x chains: instruction-level
// parallelism for leaves of few points), the rows then folded into the y
// chain in row order: the same operations in the same order per point as
// one row at a time.
template <int NP2, int PGH, int NPT, int NR>
__device__ __forceinline__ void horner3_block(const double2* lo3, int Pn, const double* x, const double* y,
                                              const double* z, Hor3* a) {
  for (int cc = Pn - 1; cc >= 0; cc--) {
    Hor2 q[NPT];
    for (int b = Pn - 1; b >= 0; b -= NR) {
      double s[NR][NPT], u[NR][NPT], w[NR][NPT];
      const double2* rw[NR];
#pragma unroll
      for (int r = 0; r < NR; r++) {
        rw[r] = lo3 + (cc * Pn + (b - r >= 0 ? b - r : b)) * NP2;  // past row 0: a copy, not folded
        const double2 ct = rw[r][NP2 - 1];
#pragma unroll
        for (int p = 0; p < NPT; p++) {
          s[r][p] = ct.y;
          u[r][p] = w[r][p] = 0.0;
          hstep<PGH>(s[r][p], u[r][p], w[r][p], x[p], ct.x);
        }
      }
#pragma unroll
      for (int m = NP2 - 2; m >= 0; m--) {
#pragma unroll
        for (int r = 0; r < NR; r++) {
          const double2 cf = rw[r][m];
#pragma unroll
          for (int p = 0; p < NPT; p++) hstep<PGH>(s[r][p], u[r][p], w[r][p], x[p], cf.y);
#pragma unroll
          for (int p = 0; p < NPT; p++) hstep<PGH>(s[r][p], u[r][p], w[r][p], x[p], cf.x);
        }
      }
#pragma unroll
      for (int r = 0; r < NR; r++)
        if (b - r >= 0)
#pragma unroll
          for (int p = 0; p < NPT; p++) hrow<PGH>(q[p], y[p], s[r][p], u[r][p], w[r][p]);
    }
#pragma unroll
    for (int p = 0; p < NPT; p++) hplane<PGH>(a[p], z[p], q[p]);
  }
}

template <int NP2, int PGH>
__global__ void __launch_bounds__(128) k_eval3d_horner(KP k, const HornerTask* __restrict__ tasks,
                                                       const double* __restrict__ lo_all) {
  constexpr int NC = ncomp<3, PGH>();
  const HornerTask T = tasks[blockIdx.x];
  const int ind = blockIdx.y, Pn = T.p + 1;
  extern __shared__ double2 lo3[];  // [Pn][Pn][NP2]
  const double2* src = reinterpret_cast<const double2*>(lo_all + T.off + (size_t)ind * Pn * Pn * 2 * NP2);
  for (int e = threadIdx.x; e < Pn * Pn * NP2; e += blockDim.x) lo3[e] = src[e];
  __syncthreads();
  const double* pts = T.set ? k.trg : k.src;
  double* out = T.set ? k.pottarg : k.pot;
  const int nc = T.set ? k.nc_t : k.nc_s;
  const double cx = k.centers[3 * T.box], cy = k.centers[3 * T.box + 1], cz = k.centers[3 * T.box + 2];
  const int ta = threadIdx.x, tb = threadIdx.x + 128;
  if (ta >= T.n) return;
  const int pa = T.i0 + ta;
  double v[NC];
  if (T.n <= 128) {
    // one point per thread, four rows in flight
    const double x = (pts[3 * pa] - cx) * k.dsq, y = (pts[3 * pa + 1] - cy) * k.dsq, z = (pts[3 * pa + 2] - cz) * k.dsq;
    Hor3 a[1];
    horner3_block<NP2, PGH, 1, 4>(lo3, Pn, &x, &y, &z, a);
    hemit<PGH>(a[0], k.dsq, v);
    add_out<NC>(out, pa, k.nd, nc, ind, v);
    return;
  }
  // two points per thread, two rows in flight
  const bool two = tb < T.n;
  const int pb = T.i0 + (two ? tb : ta);
  const double x[2] = {(pts[3 * pa] - cx) * k.dsq, (pts[3 * pb] - cx) * k.dsq};
  const double y[2] = {(pts[3 * pa + 1] - cy) * k.dsq, (pts[3 * pb + 1] - cy) * k.dsq};
  const double z[2] = {(pts[3 * pa + 2] - cz) * k.dsq, (pts[3 * pb + 2] - cz) * k.dsq};
  Hor3 a[2];
  horner3_block<NP2, PGH, 2, 2>(lo3, Pn, x, y, z, a);
  hemit<PGH>(a[0], k.dsq, v);
  add_out<NC>(out, pa, k.nd, nc, ind, v);
  if (two) {
    hemit<PGH>(a[1], k.dsq, v);
    add_out<NC>(out, pb, k.nd, nc, ind, v);
  }
}

// 2D plane-wave expansion of a box formed directly from its sources: the
// exact sum that the NUFFT scheme computes with a type-1 NUFFT
// (g2dformpwc_vec, 2d/nufft/src/g2drouts.f:1234-1307),
//   mp[a + n2 b] = sum_s q_s ws_a ws_b exp(-i (t_a x_s + t_b y_s)),
// a over the n2 positive x nodes, b over every y node (positive half first,
// the layout of the plane-wave form and of k_eval2d).  One CTA per (box,
// density); per chunk of FORM_CH sources the first threads build one
// source's factor rows each in shared memory (the phases by the recurrence
// e^{-i t1 x} (e^{-2 i t1 x})^m, the charge folded into the x row), then
// every thread sums its own coefficients over the chunk.
__global__ void __launch_bounds__(256) k_form2d_pw(KP k, const FormTask* __restrict__ tasks) {
  const FormTask T = tasks[blockIdx.x];
  const int ind = blockIdx.y;
  const int npw = k.npw, n2 = k.n2, nexp = k.nexp;
  extern __shared__ double sm[];
  double2* FX = reinterpret_cast<double2*>(sm);  // [FORM_CH][n2]
  double2* FY = FX + FORM_CH * n2;               // [FORM_CH][npw]
  const double cx = k.centers[2 * T.box], cy = k.centers[2 * T.box + 1];
  double2* out = k.mp + ((size_t)T.slot * k.nd + ind) * nexp;
  for (int c0 = 0; c0 < T.n; c0 += FORM_CH) {
    const int m = min(FORM_CH, T.n - c0);
    __syncthreads();
    if (threadIdx.x < m) {
      const int i = T.s0 + c0 + threadIdx.x;
      const double x = (k.src[2 * i] - cx) * k.dsq, y = (k.src[2 * i + 1] - cy) * k.dsq;
      const double q = k.chg[(size_t)i * k.nd + ind];
      double2 ex = cexpi(-k.t1 * x), ey = cexpi(-k.t1 * y);
      const double2 exx = cmul(ex, ex), eyy = cmul(ey, ey);
      double2* fx = FX + threadIdx.x * n2;
      double2* fy = FY + threadIdx.x * npw;
      for (int mm = 0; mm < n2; mm++) {
        const double w = k.ws[mm];  // node (2 mm + 1) t1; the weights are even in t
        fx[mm] = make_double2(ex.x * w * q, ex.y * w * q);
        const double2 b = make_double2(ey.x * w, ey.y * w);
        fy[mm] = b;
        fy[n2 + mm] = make_double2(b.x, -b.y);
        ex = cmul(ex, exx);
        ey = cmul(ey, eyy);
      }
    }
    __syncthreads();
    for (int e = threadIdx.x; e < nexp; e += blockDim.x) {
      const int a = e % n2, b = e / n2;
      double2 acc = make_double2(0.0, 0.0);
      for (int t = 0; t < m; t++) acc = cfma(FX[t * n2 + a], FY[t * npw + b], acc);
      if (c0 == 0) {
        out[e] = acc;
      } else {
        const double2 p = out[e];
        out[e] = make_double2(p.x + acc.x, p.y + acc.y);
      }
    }
  }
  if (T.n == 0)  // no sources: a zero expansion
    for (int e = threadIdx.x; e < nexp; e += blockDim.x) out[e] = make_double2(0.0, 0.0);
}

// ------------------------------------------------------------ (b) shifts
// mp -> loc at the cut level: sum over the plane-wave list plus the box's own
// multipole (g2dshiftpw_vec + g2dcopypwexp_vec, fgt2d.f:1048-1060).  Bound by the
// L1 pipe (94%): an expansion entry and a table entry per coefficient and
// neighbour, out of L2 (70%; DRAM 12%).
__global__ void k_m2l(KP k, const M2LTask* __restrict__ tasks, const M2LNbr* __restrict__ nbr) {
  const M2LTask T = tasks[blockIdx.x];
  const size_t per = (size_t)k.nd * k.nexp;
  for (size_t e = (size_t)blockIdx.y * blockDim.x + threadIdx.x; e < per; e += (size_t)gridDim.y * blockDim.x) {
    const int ee = (int)(e % k.nexp);
    double2 a = make_double2(0.0, 0.0);
    for (int t = T.off; t < T.off + T.cnt; t++) {
      const M2LNbr N = nbr[t];
      a = cfma(k.mp[(size_t)N.mp * per + e], k.wsh[(size_t)N.shift * k.nexp + ee], a);
    }
    if (T.self_mp >= 0) {
      const double2 s = k.mp[(size_t)T.self_mp * per + e];
      a.x += s.x;
      a.y += s.y;
    }
    k.loc[(size_t)T.loc * per + e] = a;
  }
}
// ------------------------------------------------------------ (c) eval, plane-wave route derivatives
// A pair of nodes +t, -t with coefficients A (of e^{itx}) and B (of e^{-itx})
// contributes A w + B conj(w), w = e^{itx}; its x derivatives are
// i t (A w - B conj(w)) and -t^2 (A w + B conj(w)).  PwAcc keeps
//   S0 = sum (A w + B w*),  S1 = sum t (A w - B w*),  S2 = sum t^2 (A w + B w*)
// (the derivative orders the evaluation needs), so that d/dx = i S1 and
// d2/dx2 = -S2 (the ww1x / ww1xx factors of g2dpwevalg_vec / g2dpwevalh_vec,
// g2drouts.f:1973-2200, and g3dpwevalg/h_vec, g3drouts.f:2369-2660).
template <int ORD>
struct PwAcc {
  double2 s[ORD + 1];
  __device__ __forceinline__ PwAcc() {
#pragma unroll
    for (int i = 0; i <= ORD; i++) s[i] = make_double2(0.0, 0.0);
  }
  // add A w + B conj(w) at node t
  __device__ __forceinline__ void add(double2 A, double2 B, double2 w, double t) {
    if (ORD == 0) {  // the potential alone: two complex FMAs
      s[0] = cfmac(B, w, cfma(A, w, s[0]));
      return;
    }
    const double2 p = cmul(A, w), m = cmulc(B, w);  // A w, B conj(w)
    const double2 sp = make_double2(p.x + m.x, p.y + m.y);
    s[0].x += sp.x;
    s[0].y += sp.y;
    if (ORD >= 1) {
      s[1].x = fma(t, p.x - m.x, s[1].x);
      s[1].y = fma(t, p.y - m.y, s[1].y);
    }
    if (ORD >= 2) {
      const double t2 = t * t;
      s[2].x = fma(t2, sp.x, s[2].x);
      s[2].y = fma(t2, sp.y, s[2].y);
    }
  }
};

// ------------------------------------------------------------ (c) eval, 2D plane-wave route
// One CTA per (leaf, point set, density): direct plane-wave sum at every point
// with e^{i t x} built by the recurrence of g2dpwevalp_vec (g2drouts.f:1887-1966),
// on the levels where the reference picks it (nlocal > 50, fgt2d.f:1166).
// The stored half is x > 0; y runs over both signs.  With z_j = sum over x
// nodes of e^{i t_x x} t_x^a (y-sum of derivative order b), the outputs are
//   pot = 2 Re z(0,0), g_x = -2 Im z(1,0), g_y = -2 Im z(0,1),
//   h_xx = -2 Re z(2,0), h_xy = -2 Re z(1,1), h_yy = -2 Re z(0,2)
// times dsq per derivative.
template <int PGH>
__global__ void __launch_bounds__(256) k_eval2d(KP k, const EvalTask* __restrict__ tasks) {
  constexpr int NC = ncomp<2, PGH>(), ORD = PGH - 1;
  const EvalTask T = tasks[blockIdx.x];
  const int ind = blockIdx.y;
  const int n2 = k.n2;
  const double2* L = k.loc + ((size_t)T.slot * k.nd + ind) * k.nexp;
  const double* pts = T.set ? k.trg : k.src;
  double* out = T.set ? k.pottarg : k.pot;
  const int nc = T.set ? k.nc_t : k.nc_s;
  const double cx = k.centers[2 * T.box], cy = k.centers[2 * T.box + 1];
  for (int i = threadIdx.x; i < T.n; i += blockDim.x) {
    const int ip = T.i0 + i;
    const double x = (pts[2 * ip] - cx) * k.dsq, y = (pts[2 * ip + 1] - cy) * k.dsq;
    const double2 ex = cexpi(k.t1 * x), ey = cexpi(k.t1 * y);
    const double2 exx = cmul(ex, ex), eyy = cmul(ey, ey);
    // z[0] = (0,0), z[1] = (1,0), z[2] = (0,1), z[3] = (2,0), z[4] = (1,1), z[5] = (0,2)
    double2 z[NC];
#pragma unroll
    for (int c = 0; c < NC; c++) z[c] = make_double2(0.0, 0.0);
    double2 w1 = ex;
    for (int kx = 0; kx < n2; kx++) {
      const double tx = (2 * kx + 1) * k.t1;
      PwAcc<ORD> sy;
      double2 w2 = ey;
      for (int ky = 0; ky < n2; ky++) {
        sy.add(L[kx + n2 * ky], L[kx + n2 * (ky + n2)], w2, (2 * ky + 1) * k.t1);
        w2 = cmul(w2, eyy);
      }
      const double2 a0 = cmul(sy.s[0], w1);
      z[0].x += a0.x;
      z[0].y += a0.y;
      if (PGH >= 2) {
        const double2 a1 = cmul(sy.s[ORD >= 1 ? 1 : 0], w1);
        z[1].x = fma(tx, a0.x, z[1].x);
        z[1].y = fma(tx, a0.y, z[1].y);
        z[2].x += a1.x;
        z[2].y += a1.y;
        if (PGH >= 3) {
          const double2 a2 = cmul(sy.s[ORD >= 2 ? 2 : 0], w1);
          z[3].x = fma(tx * tx, a0.x, z[3].x);
          z[4].x = fma(tx, a1.x, z[4].x);
          z[5].x += a2.x;
        }
      }
      w1 = cmul(w1, exx);
    }
    double v[NC];
    v[0] = 2.0 * z[0].x;
    if (PGH >= 2) {
      v[1] = -2.0 * z[1].y * k.dsq;
      v[2] = -2.0 * z[2].y * k.dsq;
    }
    if (PGH >= 3) {
      const double d2 = k.dsq * k.dsq;
      v[3] = -2.0 * z[3].x * d2;
      v[4] = -2.0 * z[4].x * d2;
      v[5] = -2.0 * z[5].x * d2;
    }
    add_out<NC>(out, ip, k.nd, nc, ind, v);
  }
}

// ------------------------------------------------------------ (d) near field
// Source list of a near-field task: the concatenation of its source ranges
// (leaves of its list1).  A warp walks it in batches of at most CAP sources:
// ranges are read 32 at a time (one per lane) and prefix-summed with
// shuffles; for the batch starting at b0 each lane maps its slots
// b0 + lane + 32 u to source indices by a binary search over the lanes'
// prefixes, so all loads of a batch can be in flight together (a range at a
// time would serialise one load round trip per range).
// ------------------------------------------------------------ (d) near field, kernels
// One warp per chunk of <= 32 evaluation points (g2d_directcp_vec,
// g2ddirect.f:32-76; g3d_directcp_vec, g3ddirect.f:3-49): the chunk's source
// ranges are staged through the warp's shared memory in batches of 256, and
// g lanes per point (g n <= 32) split the sources of that point.
// pot += q exp(-r^2/delta) when r^2 < dmax, all in FP64; with PGH > 1 the
// gradient and Hessian per pair as g2d_directcg/ch_vec (g2ddirect.f:83-212)
// and g3d_directcg/ch_vec (g3ddirect.f:56-203): with rfac = -2/delta and
// d = target - source, grad += rfac d_i r, hess_ii += (rfac + (rfac d_i)^2) r,
// hess_ij += (rfac d_i)(rfac d_j) r, r = q exp(-|d|^2/delta).
template <int DIM, int PGH>
__device__ __forceinline__ void pair_terms(double* acc, double r, const double* d, double rfac) {
  acc[0] += r;
  if (PGH >= 2) {
    double g[DIM];
#pragma unroll
    for (int i = 0; i < DIM; i++) {
      g[i] = rfac * d[i];
      acc[1 + i] = fma(g[i], r, acc[1 + i]);
    }
    if (PGH >= 3) {
      double* h = acc + 1 + DIM;
      if (DIM == 2) {
        h[0] = fma(fma(g[0], g[0], rfac), r, h[0]);
        h[1] = fma(g[0] * g[1], r, h[1]);
        h[2] = fma(fma(g[1], g[1], rfac), r, h[2]);
      } else {
        h[0] = fma(fma(g[0], g[0], rfac), r, h[0]);
        h[1] = fma(fma(g[1], g[1], rfac), r, h[1]);
        h[2] = fma(fma(g[DIM - 1], g[DIM - 1], rfac), r, h[2]);
        h[3] = fma(g[0] * g[1], r, h[3]);
        h[4] = fma(g[0] * g[DIM - 1], r, h[4]);
        h[5] = fma(g[1] * g[DIM - 1], r, h[5]);
      }
    }
  }
}
// Dipole terms per pair (g2d_directd{p,g,h}_vec, g2ddirect.f:217-420, and
// g3d_directd*_vec, g3ddirect.f:207-435), v = dipstr n, e = exp(-r^2/delta):
// with R = 2/delta, u = R (t - s), rinc = u.v,
//   pot += rinc e,  grad_a += g_a e with g_a = R v_a - rinc u_a,
//   hess_aa += (-R (u_a v_a + rinc) - g_a u_a) e,  hess_ab += (-R u_a v_b - g_a u_b) e.
template <int DIM, int PGH>
__device__ __forceinline__ void dip_terms(double* acc, double e, const double* d, const double* v,
                                          double R) {
  double u[DIM], rinc = 0.0;
#pragma unroll
  for (int a = 0; a < DIM; a++) {
    u[a] = R * d[a];
    rinc = fma(u[a], v[a], rinc);
  }
  acc[0] = fma(rinc, e, acc[0]);
  if (PGH >= 2) {
    double g[DIM];
#pragma unroll
    for (int a = 0; a < DIM; a++) {
      g[a] = fma(R, v[a], -rinc * u[a]);
      acc[1 + a] = fma(g[a], e, acc[1 + a]);
    }
    if (PGH >= 3) {
      double* h = acc + 1 + DIM;
      auto hd = [&](int a) { return -R * (u[a] * v[a] + rinc) - g[a] * u[a]; };
      auto ho = [&](int a, int b) { return -R * u[a] * v[b] - g[a] * u[b]; };
      if (DIM == 2) {
        h[0] = fma(hd(0), e, h[0]);
        h[1] = fma(ho(0, 1), e, h[1]);
        h[2] = fma(hd(1), e, h[2]);
      } else {
        h[0] = fma(hd(0), e, h[0]);
        h[1] = fma(hd(1), e, h[1]);
        h[2] = fma(hd(DIM - 1), e, h[2]);
        h[3] = fma(ho(0, 1), e, h[3]);
        h[4] = fma(ho(0, DIM - 1), e, h[4]);
        h[5] = fma(ho(1, DIM - 1), e, h[5]);
      }
    }
  }
}
// DIP: charges (when present) and dipoles, staged with the dipole vectors;
// 128 sources per batch so the staging stays within static shared memory.
template <int DIM, int PGH, bool DIP>
__global__ void __launch_bounds__(128) k_direct(KP k, const DirTask* __restrict__ tasks, int ntask,
                                                const SrcRange* __restrict__ ranges) {
  constexpr int NC = ncomp<DIM, PGH>();
  constexpr int CAP = DIP ? 128 : 256;  // sources staged per warp and batch
  constexpr int ROWS = DIP ? 2 * DIM + 1 : DIM + 1;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int w = blockIdx.x * 4 + warp;
  __shared__ double ssm[4][ROWS * CAP];
  if (w >= ntask) return;  // whole warp leaves; no block-wide barrier below
  const DirTask T = tasks[w];
  const int ind = blockIdx.y;
  double* sx = ssm[warp];
  double* sy = sx + CAP;
  double* sz = sy + CAP;
  double* sq = sz + (DIM == 3 ? CAP : 0);
  double* sv = sq + CAP;  // [DIM][CAP] dipole vectors (DIP)
  // g lanes per point (g * n <= 32) split the sources of that point
  int g = 1;
  while (g * 2 * T.n <= 32) g *= 2;
  const int tt = lane / g, sub = lane - tt * g;
  const bool act = tt < T.n;
  const double* pts = T.set ? k.trg : k.src;
  double* out = T.set ? k.pottarg : k.pot;
  const int nc = T.set ? k.nc_t : k.nc_s;
  const int ip = T.i0 + (act ? tt : 0);
  const double tx = pts[DIM * ip], ty = pts[DIM * ip + 1];
  const double tz = DIM == 3 ? pts[DIM * ip + 2] : 0.0;
  const double ninv = -1.0 / k.delta, rfac = -2.0 / k.delta;
  double acc[NC];
#pragma unroll
  for (int c = 0; c < NC; c++) acc[c] = 0.0;
  for (int rc = 0; rc < T.cnt; rc += 32) {
    const RangeChunk C = load_range_chunk(ranges, T.off, T.cnt, rc, lane);
    for (int b0 = 0; b0 < C.tot; b0 += CAP) {
      const int m = min(CAP, C.tot - b0);
      int js[CAP / 32];
#pragma unroll
      for (int u = 0; u < CAP / 32; u++) js[u] = range_slot_source(C, b0 + lane + 32 * u);
      __syncwarp();
#pragma unroll
      for (int u = 0; u < CAP / 32; u++) {
        const int t = lane + 32 * u;
        if (t < m) {
          const int j = js[u];
          sx[t] = k.src[DIM * j];
          sy[t] = k.src[DIM * j + 1];
          if (DIM == 3) sz[t] = k.src[DIM * j + 2];
          if (DIP) {
            sq[t] = src_charge(k, j, ind);
            double v[DIM];
            src_dipole<DIM>(k, j, ind, v);
#pragma unroll
            for (int a = 0; a < DIM; a++) sv[a * CAP + t] = v[a];
          } else {
            sq[t] = k.chg[(size_t)j * k.nd + ind];
          }
        }
      }
      __syncwarp();
      if (act) {
#pragma unroll 4
        for (int t = sub; t < m; t += g) {
          const double dx = tx - sx[t], dy = ty - sy[t];
          double rr = fma(dx, dx, dy * dy);
          double dz = 0.0;
          if (DIM == 3) {
            dz = tz - sz[t];
            rr = fma(dz, dz, rr);
          }
          if (rr < k.dmax) {
            if (DIP) {
              const double e = exp(rr * ninv), d[3] = {dx, dy, dz};
              double v[DIM];
#pragma unroll
              for (int a = 0; a < DIM; a++) v[a] = sv[a * CAP + t];
              if (PGH == 1) acc[0] = fma(e, sq[t], acc[0]);
              else pair_terms<DIM, PGH>(acc, e * sq[t], d, rfac);
              dip_terms<DIM, PGH>(acc, e, d, v, -rfac);
            } else if (PGH == 1) {
              acc[0] = fma(exp(rr * ninv), sq[t], acc[0]);
            } else {
              const double d[3] = {dx, dy, dz};
              pair_terms<DIM, PGH>(acc, exp(rr * ninv) * sq[t], d, rfac);
            }
          }
        }
      }
    }
  }
#pragma unroll
  for (int c = 0; c < NC; c++)
    for (int o = 1; o < g; o <<= 1) acc[c] += __shfl_xor_sync(0xffffffffu, acc[c], o);
  if (act && sub == 0) add_out<NC>(out, ip, k.nd, nc, ind, acc);
}

// Scaled coordinates of the mixed near field, once per plan: (x - c) cs with
// c the root box's centre, as an FP32 pair (hi, lo) per dimension.
__global__ void k_mixed_coords(const double* __restrict__ x, int n, int dim, double c0, double c1, double c2,
                               double cs, float* __restrict__ f) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    for (int d = 0; d < dim; d++) {
      const double v = (x[(size_t)dim * i + d] - (d == 0 ? c0 : d == 1 ? c1 : c2)) * cs;
      const float h = (float)v;
      f[(size_t)2 * dim * i + 2 * d] = h;
      f[(size_t)2 * dim * i + 2 * d + 1] = (float)(v - (double)h);
    }
}

// Mixed form of the near field (eps >= 1e-6): the same task structure with
// the pair arithmetic in FP32.  Coordinates are taken relative to the root
// box's centre, scaled by sqrt(log2(e) / delta) and split into a float pair
// (hi, lo) once per plan (k_mixed_coords), so dx = (t_hi - s_hi) + (t_lo -
// s_lo) carries about FP32 relative accuracy in dx itself (the hi parts of
// nearby points subtract exactly; the lo parts hold the rest to 2^-48 of the
// coordinate); the Gaussian is then
// 2^-(dx^2 + dy^2 (+ dz^2)) by ex2.approx.  Each lane holds NTL = 4 targets,
// so a staged source is read from shared memory once for four pairs; g lanes
// per target group (g * groups <= 32) split the sources.  Groups of four
// sources are summed in FP32 per target and added into FP64 accumulators.
// With PGH > 1 the FP32 partials are, per target, sum e q, sum e q d_i and
// (PGH = 3) sum e q d_i d_j in the scaled differences d = (x_t - x_s) cs;
// they become the gradient rfac/cs sum e q d_i and the Hessian
// rfac sum e q + (rfac/cs)^2 sum e q d_i^2 (diagonal), (rfac/cs)^2 sum e q d_i d_j
// in FP64 (the per-pair terms of g2d_directch_vec / g3d_directch_vec).
template <int DIM, int PGH>
__global__ void __launch_bounds__(128) k_direct_mixed(KP k, const DirTask* __restrict__ tasks, int ntask,
                                                      const SrcRange* __restrict__ ranges, double cs,
                                                      float amax) {
  constexpr int CAP = 256, NTL = PGH == 1 ? 4 : PGH == 2 ? 2 : 1;
  constexpr int NC = ncomp<DIM, PGH>();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int w = blockIdx.x * 4 + warp;
  __shared__ float fsm[4][(2 * DIM + 1) * CAP];
  if (w >= ntask) return;  // whole warp leaves; no block-wide barrier below
  const DirTask T = tasks[w];
  const int ind = blockIdx.y;
  float* sh = fsm[warp];           // [DIM][CAP] hi parts
  float* sl = sh + DIM * CAP;      // [DIM][CAP] lo parts
  float* sq = sl + DIM * CAP;      // [CAP] charges
  const int ngr = (T.n + NTL - 1) / NTL;
  int g = 1;
  while (g * 2 * ngr <= 32) g *= 2;
  const int tt = lane / g, sub = lane - tt * g;
  const bool act = tt < ngr;
  double* out = T.set ? k.pottarg : k.pot;
  const int nc = T.set ? k.nc_t : k.nc_s;
  const float* fp = T.set ? k.ftrg : k.fsrc;  // the points' FP32 (hi, lo) coordinates
  float th[NTL][DIM], tl[NTL][DIM];
  double acc[NTL][NC];
#pragma unroll
  for (int v = 0; v < NTL; v++) {
#pragma unroll
    for (int c = 0; c < NC; c++) acc[v][c] = 0.0;
    const int it = min(tt * NTL + v, T.n - 1);
#pragma unroll
    for (int d = 0; d < DIM; d++) {
      th[v][d] = fp[(size_t)2 * DIM * (T.i0 + it) + 2 * d];
      tl[v][d] = fp[(size_t)2 * DIM * (T.i0 + it) + 2 * d + 1];
    }
  }
  for (int rc = 0; rc < T.cnt; rc += 32) {
   const RangeChunk C = load_range_chunk(ranges, T.off, T.cnt, rc, lane);
   for (int b0 = 0; b0 < C.tot; b0 += CAP) {
    const int m = min(CAP, C.tot - b0);
    int js[CAP / 32];
#pragma unroll
    for (int u = 0; u < CAP / 32; u++) js[u] = range_slot_source(C, b0 + lane + 32 * u);
    __syncwarp();
#pragma unroll
    for (int u = 0; u < CAP / 32; u++) {
      const int t = lane + 32 * u;
      if (t < m) {
        const int j = js[u];
#pragma unroll
        for (int d = 0; d < DIM; d++) {
          const float2 hl = reinterpret_cast<const float2*>(k.fsrc)[(size_t)DIM * j + d];
          sh[d * CAP + t] = hl.x;
          sl[d * CAP + t] = hl.y;
        }
        sq[t] = (float)k.chg[(size_t)j * k.nd + ind];
      }
    }
    __syncwarp();
    if (act) {
      for (int t = sub; t < m; t += 4 * g) {
        float part[NTL][NC];
#pragma unroll
        for (int v = 0; v < NTL; v++)
#pragma unroll
          for (int c = 0; c < NC; c++) part[v][c] = 0.0f;
#pragma unroll
        for (int u = 0; u < 4; u++) {
          const int tu = t + u * g;
          if (tu < m) {
            float sH[DIM], sL[DIM];
#pragma unroll
            for (int d = 0; d < DIM; d++) {
              sH[d] = sh[d * CAP + tu];
              sL[d] = sl[d * CAP + tu];
            }
            const float q = sq[tu];
#pragma unroll
            for (int v = 0; v < NTL; v++) {
              float a = 0.0f, dd[DIM];
#pragma unroll
              for (int d = 0; d < DIM; d++) {
                dd[d] = (th[v][d] - sH[d]) + (tl[v][d] - sL[d]);
                a = fmaf(dd[d], dd[d], a);
              }
              const float e = ex2_approx(-a);
              if (PGH == 1) {
                part[v][0] = a < amax ? fmaf(e, q, part[v][0]) : part[v][0];
              } else if (a < amax) {
                const float r = e * q;
                part[v][0] += r;
#pragma unroll
                for (int d = 0; d < DIM; d++) part[v][1 + d] = fmaf(dd[d], r, part[v][1 + d]);
                if (PGH >= 3) {
                  float* h = part[v] + 1 + DIM;
                  if (DIM == 2) {
                    h[0] = fmaf(dd[0] * dd[0], r, h[0]);
                    h[1] = fmaf(dd[0] * dd[1], r, h[1]);
                    h[2] = fmaf(dd[1] * dd[1], r, h[2]);
                  } else {
                    h[0] = fmaf(dd[0] * dd[0], r, h[0]);
                    h[1] = fmaf(dd[1] * dd[1], r, h[1]);
                    h[2] = fmaf(dd[DIM - 1] * dd[DIM - 1], r, h[2]);
                    h[3] = fmaf(dd[0] * dd[1], r, h[3]);
                    h[4] = fmaf(dd[0] * dd[DIM - 1], r, h[4]);
                    h[5] = fmaf(dd[1] * dd[DIM - 1], r, h[5]);
                  }
                }
              }
            }
          }
        }
#pragma unroll
        for (int v = 0; v < NTL; v++)
#pragma unroll
          for (int c = 0; c < NC; c++) acc[v][c] += (double)part[v][c];
      }
    }
   }
  }
#pragma unroll
  for (int v = 0; v < NTL; v++)
#pragma unroll
    for (int c = 0; c < NC; c++)
      for (int o2 = 1; o2 < g; o2 <<= 1) acc[v][c] += __shfl_xor_sync(0xffffffffu, acc[v][c], o2);
  if (act && sub == 0) {
    // scaled sums -> physical: d = dx cs, rfac = -2/delta
    const double rfac = -2.0 / k.delta, c1 = rfac / cs, c2 = c1 * c1;
#pragma unroll
    for (int v = 0; v < NTL; v++) {
      const int it = tt * NTL + v;
      if (it >= T.n) continue;
      double w[NC];
      w[0] = acc[v][0];
      if (PGH >= 2)
#pragma unroll
        for (int d = 0; d < DIM; d++) w[1 + d] = c1 * acc[v][1 + d];
      if (PGH >= 3) {
        const double* h = acc[v] + 1 + DIM;
        double* hw = w + 1 + DIM;
        if (DIM == 2) {
          hw[0] = fma(c2, h[0], rfac * w[0]);
          hw[1] = c2 * h[1];
          hw[2] = fma(c2, h[2], rfac * w[0]);
        } else {
          hw[0] = fma(c2, h[0], rfac * w[0]);
          hw[1] = fma(c2, h[1], rfac * w[0]);
          hw[2] = fma(c2, h[2], rfac * w[0]);
          hw[3] = c2 * h[3];
          hw[4] = c2 * h[4];
          hw[5] = c2 * h[5];
        }
      }
      add_out<NC>(out, T.i0 + it, k.nd, nc, ind, w);
    }
  }
}

// ------------------------------------------------------------ large delta
// local[j + P k (+ P^2 l)] = sum_i q h_j(x) h_k(y) (h_l(z)) with
// h_j(x) = H_j(x) e^{-x^2} / j! (g2dformlc_vec, g2drouts.f:621-681), one
// partial sum per CTA added into the global array.
// Dipoles (g2dformld_vec / g3dformld_vec, g2drouts.f:685-840,
// g3drouts.f:857-1040) add columns with the source derivative of one
// factor, dh_j = -(j+1) dsq h_(j+1): 2D (hx, q hy + v2 dhy), (v1 dhx, hy);
// 3D as dip3_coef with these h and dh.
template <int DIM>
__global__ void __launch_bounds__(256) k_ld_form(KP k, int ns, int p, const double3 c3,
                                                 double* __restrict__ local, double* __restrict__ partial) {
  const double cen[3] = {c3.x, c3.y, c3.z};
  const int Pn = p + 1;
  const int nent = DIM == 2 ? Pn * Pn : Pn * Pn * Pn;
  extern __shared__ double sm[];
  double* hx = sm;                    // [FORM_CH][Pn]
  double* hy = hx + FORM_CH * Pn;
  double* hz = hy + FORM_CH * Pn;
  const int ind = blockIdx.y;
  const int per = (ns + gridDim.x - 1) / gridDim.x;
  const int i0 = blockIdx.x * per, i1 = min(ns, i0 + per);
  const int vc = k.ifdipole ? DIM : 1, chs = FORM_CH / vc;
  for (int e0 = 0; e0 < nent; e0 += 256 * 4) {
    double acc[4] = {0, 0, 0, 0};
    for (int c0 = i0; c0 < i1; c0 += chs) {
      const int m = vc * min(chs, i1 - c0);
      __syncthreads();
      if (threadIdx.x < m) {
        const int i = c0 + threadIdx.x / vc, col = threadIdx.x % vc;
        double v[3];
        for (int d = 0; d < DIM; d++) v[d] = (k.src[DIM * i + d] - cen[d]) * k.dsq;
        if (!k.ifdipole) {
          for (int d = 0; d < DIM; d++) {
            double* h = (d == 0 ? hx : d == 1 ? hy : hz) + threadIdx.x * Pn;
            const double f = exp(-v[d] * v[d]);
            h[0] = f;
            if (Pn > 1) h[1] = 2.0 * v[d] * f;
            for (int j = 1; j < Pn - 1; j++) h[j + 1] = 2.0 * (v[d] * h[j] - h[j - 1]) / (j + 1);
          }
          double* hl = (DIM == 2 ? hy : hz) + threadIdx.x * Pn;
          const double q = k.chg[(size_t)i * k.nd + ind];
          for (int j = 0; j < Pn; j++) hl[j] *= q;
        } else {
          double dv[3] = {0.0, 0.0, 0.0}, a, b;
          src_dipole<DIM>(k, i, ind, dv);
          const double q = src_charge(k, i, ind);
          for (int d = 0; d < DIM; d++) {
            if (DIM == 2) {  // columns (hx, q hy + v2 dhy) and (v1 dhx, hy)
              a = d == 0 ? (col ? 0.0 : 1.0) : (col ? 1.0 : q);
              b = d == 0 ? (col ? dv[0] : 0.0) : (col ? 0.0 : dv[1]);
            } else {
              dip3_coef(col, d, q, dv, a, b);
            }
            // h_0 .. h_Pn by the recurrence, row_j = a h_j - b (j+1) dsq h_(j+1)
            double* row = (d == 0 ? hx : d == 1 ? hy : hz) + threadIdx.x * Pn;
            const double f = exp(-v[d] * v[d]);
            double hm = f, hc = 2.0 * v[d] * f;  // h_j, h_(j+1)
            for (int j = 0; j < Pn; j++) {
              row[j] = fma(a, hm, -b * (j + 1.0) * k.dsq * hc);
              const double hn = 2.0 * (v[d] * hc - hm) / (j + 2);
              hm = hc;
              hc = hn;
            }
          }
        }
      }
      __syncthreads();
      for (int t = 0; t < m; t++) {
#pragma unroll
        for (int s = 0; s < 4; s++) {
          const int e = e0 + threadIdx.x + s * 256;
          if (e < nent) {
            const int a = e % Pn, b = (e / Pn) % Pn, c = e / (Pn * Pn);
            double v = hx[t * Pn + a] * hy[t * Pn + b];
            if (DIM == 3) v *= hz[t * Pn + c];
            acc[s] += v;
          }
        }
      }
    }
#pragma unroll
    for (int s = 0; s < 4; s++) {
      const int e = e0 + threadIdx.x + s * 256;
      if (e >= nent) continue;
      if (partial) partial[((size_t)ind * gridDim.x + blockIdx.x) * nent + e] = acc[s];
      else atomicAdd(local + (size_t)ind * nent + e, acc[s]);
    }
  }
}
// local = sum of the per-CTA partial blocks, in CTA order (deterministic)
__global__ void k_ld_sum(int nent, int nparts, const double* __restrict__ partial, double* __restrict__ local) {
  const int ind = blockIdx.y;
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < nent; e += gridDim.x * blockDim.x) {
    double a = 0.0;
    for (int c = 0; c < nparts; c++) a += partial[((size_t)ind * nparts + c) * nent + e];
    local[(size_t)ind * nent + e] = a;
  }
}
// Taylor evaluation at every point (g2dlevalp/g/h_vec, g3dlevalp/g/h_vec);
// outputs in the caller's layout: pot(nd, n), grad(nd, dim, n), hess(nd, H, n).
template <int DIM, int PGH>
__global__ void k_ld_eval(KP k, int n, const double* __restrict__ pts, double* __restrict__ pot,
                          double* __restrict__ grad, double* __restrict__ hess, int p,
                          const double3 c3, const double* __restrict__ local) {
  const double cen[3] = {c3.x, c3.y, c3.z};
  constexpr int NC = ncomp<DIM, PGH>(), NH = nhess<DIM>();
  const int Pn = p + 1;
  const int nent = DIM == 2 ? Pn * Pn : Pn * Pn * Pn;
  const int ind = blockIdx.y, nd = k.nd;
  const double* lo = local + (size_t)ind * nent;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const double x = (pts[DIM * i] - cen[0]) * k.dsq, y = (pts[DIM * i + 1] - cen[1]) * k.dsq;
    double v[NC];
    if (DIM == 2) horner2_rt<PGH>(lo, Pn, Pn, x, y, k.dsq, v);
    else horner3_rt<PGH>(lo, Pn, Pn, x, y, (pts[DIM * i + 2] - cen[DIM - 1]) * k.dsq, k.dsq, v);
    pot[(size_t)i * nd + ind] = v[0];
    if (PGH >= 2)
#pragma unroll
      for (int d = 0; d < DIM; d++) grad[((size_t)i * DIM + d) * nd + ind] = v[1 + d];
    if (PGH >= 3)
#pragma unroll
      for (int c = 0; c < NH; c++) hess[((size_t)i * NH + c) * nd + ind] = v[1 + DIM + c];
  }
}

// ------------------------------------------------------------ FP64 MMA throughput probe
// Eight independent m8n8k4 f64 accumulator chains per warp, `iters` steps:
// 8 * 256 * iters FMAs per warp.  Used to measure the FP64 tensor-core
// denominator of the 2D form/eval roofline on the running GPU.
__global__ void __launch_bounds__(128) k_probe_dmma(double* out, int iters) {
  double c[8][2];
  const double a = 1.0 + 1e-9 * threadIdx.x, b = 1.0 - 1e-9 * blockIdx.x;
#pragma unroll
  for (int i = 0; i < 8; i++) c[i][0] = c[i][1] = 0.0;
  for (int it = 0; it < iters; it++) {
#pragma unroll
    for (int i = 0; i < 8; i++) dmma_884(c[i][0], c[i][1], a, b);
  }
  double s = 0.0;
#pragma unroll
  for (int i = 0; i < 8; i++) s += c[i][0] + c[i][1];
  if (s == 12345.678) out[0] = s;  // keeps the chains live
}

// ------------------------------------------------------------ host helpers
template <typename T, typename A>
cudaError_t put(char*& cur, T*& dst, const std::vector<T, A>& v, cudaStream_t s) {
  dst = reinterpret_cast<T*>(cur);
  size_t b = (v.size() * sizeof(T) + 255) & ~size_t(255);
  cur += b;
  if (v.empty()) return cudaSuccess;
  return cudaMemcpyAsync(dst, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice, s);
}
template <typename T, typename A>
size_t bytes_of(const std::vector<T, A>& v) {
  return (v.size() * sizeof(T) + 255) & ~size_t(255);
}
size_t al(size_t b) { return (b + 255) & ~size_t(255); }

// Arrays placed one after another in the device arena (as put() does) and
// copied up together: the host data is gathered, by the host threads, into
// a pinned mirror of the arena range, which goes up in one asynchronous copy.
// The mirror belongs to the calling thread and is reused; the caller
// synchronises the stream before the thread stages again.
struct Staged {
  struct Item {
    size_t off, bytes;
    const void* src;
  };
  std::vector<Item> items;
  size_t span = 0;
  template <typename T, typename A>
  void add(char*& cur, T*& dst, const std::vector<T, A>& v) {
    dst = reinterpret_cast<T*>(cur);
    const size_t b = v.size() * sizeof(T);
    if (b) items.push_back({span, b, v.data()});
    span += (b + 255) & ~size_t(255);
    cur += (b + 255) & ~size_t(255);
  }
  cudaError_t upload(char* dev, cudaStream_t s) {
    if (span == 0) return cudaSuccess;
    // A mirror that grows keeps its old buffers until the thread exits:
    // cudaFreeHost waits for the whole device, which would stall this
    // request behind every other stream's work (the server's workers).
    struct Mirror {
      char* p = nullptr;
      size_t cap = 0;
      std::vector<char*> old;
      ~Mirror() {
        if (p) cudaFreeHost(p);
        for (char* q : old) cudaFreeHost(q);
      }
    };
    thread_local Mirror m;
    if (m.cap < span) {
      if (m.p) m.old.push_back(m.p);
      m.p = nullptr;
      const size_t want = std::max(std::max(span + span / 4, 2 * m.cap), (size_t)16 << 20);
      m.cap = 0;
      cudaError_t e = cudaHostAlloc(reinterpret_cast<void**>(&m.p), want, cudaHostAllocPortable);
      if (e != cudaSuccess) {
        m.p = nullptr;
        (void)cudaGetLastError();
        // no pinned memory: the arrays go up one by one from where they are
        for (const Item& it : items) {
          e = cudaMemcpyAsync(dev + it.off, it.src, it.bytes, cudaMemcpyHostToDevice, s);
          if (e != cudaSuccess) return e;
        }
        return cudaSuccess;
      }
      m.cap = want;
    }
    // copy in 1 MB pieces so that large arrays are split over the threads
    // (the mirror's address is taken here: m is the calling thread's own)
    char* const mirror = m.p;
    std::vector<std::pair<size_t, size_t>> pieces;  // (item, piece offset)
    for (size_t i = 0; i < items.size(); i++)
      for (size_t o = 0; o < items[i].bytes; o += (1 << 20)) pieces.push_back({i, o});
#pragma omp parallel for schedule(dynamic, 1) if (span > (4u << 20))
    for (long long q = 0; q < (long long)pieces.size(); q++) {
      const Item& it = items[pieces[q].first];
      const size_t o = pieces[q].second, n = std::min<size_t>(1 << 20, it.bytes - o);
      memcpy(mirror + it.off + o, static_cast<const char*>(it.src) + o, n);
    }
    return cudaMemcpyAsync(dev, mirror, span, cudaMemcpyHostToDevice, s);
  }
};


}  // namespace

#define CK(x)                               \
  do {                                      \
    cudaError_t e_ = (x);                   \
    if (e_ != cudaSuccess) return e_;       \
  } while (0)

// Stable sort of tasks by (route, order): a counting sort (the keys are few
// small integers), linear in the number of tasks.
template <typename Task>
std::vector<Task> route_order_sort(const std::vector<Task>& in) {
  // the tasks come level by level, so runs of one key are long: count and
  // place whole runs (a per-task counter increment is a dependency chain
  // through one memory cell when most tasks share a key)
  auto key = [](const Task& t) { return 4096 * t.route + t.p; };
  std::vector<std::pair<size_t, size_t>> runs;  // [begin, end)
  int kmax = 0;
  for (size_t i = 0; i < in.size();) {
    size_t j = i + 1;
    const int k = key(in[i]);
    while (j < in.size() && key(in[j]) == k) j++;
    runs.push_back({i, j});
    kmax = std::max(kmax, k);
    i = j;
  }
  std::vector<size_t> cnt((size_t)kmax + 2, 0);
  for (const auto& r : runs) cnt[key(in[r.first]) + 1] += r.second - r.first;
  for (size_t i = 1; i < cnt.size(); i++) cnt[i] += cnt[i - 1];
  std::vector<Task> out(in.size());
  for (const auto& r : runs) {
    size_t& at = cnt[key(in[r.first])];
    std::copy(in.begin() + r.first, in.begin() + r.second, out.begin() + at);
    at += r.second - r.first;
  }
  return out;
}
// Two pieces of host work, on two threads of the team where `par`.
template <typename F, typename G>
void beside(bool par, F&& f, G&& g) {
  std::exception_ptr err[2];
#pragma omp parallel for schedule(static, 1) if (par)
  for (int i = 0; i < 2; i++) {
    try {
      if (i == 0) f();
      else g();
    } catch (...) {
      err[i] = std::current_exception();
    }
  }
  for (const std::exception_ptr& e : err)
    if (e) std::rethrow_exception(e);
}
cudaError_t device_pool_setup() {
  // keep freed stream-ordered allocations in the device's default pool
  // instead of returning them at every synchronisation (process-local
  // runtime state, once per device)
  static std::mutex mu;
  static bool done[64] = {false};
  int dev = 0;
  CK(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lk(mu);
  if (dev >= 0 && dev < 64 && !done[dev]) {
    cudaMemPool_t pool;
    CK(cudaDeviceGetDefaultMemPool(&pool, dev));
    uint64_t thr = UINT64_MAX;
    CK(cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &thr));
    done[dev] = true;
  }
  return cudaSuccess;
}

// What changes a plan's arithmetic is chosen by order from the tasks of the
// whole transform (a shard's: of all its ranks).
//
// Formation: sources per partial block (chunk), and in 2D the orders whose
// leaves (or chunks) take a warp each (k_form2d_mma).
struct FormRules {
  int chunk = 1 << 30;
  std::vector<uint8_t> warp;
};
FormRules form_rules(const Params& P, const std::vector<FormTask>& tasks, int sms) {
  FormRules R;
  // sources and tasks by order; the tasks come level by level, so a run of one
  // order is summed in registers
  std::vector<long long> n(P.ntermmax + 1, 0), cnt(P.ntermmax + 1, 0);
  long long nsrc = 0;
  int most = 0;
  for (size_t i = 0; i < tasks.size();) {
    const int p = tasks[i].p;
    long long sum = 0, num = 0;
    for (; i < tasks.size() && tasks[i].p == p; i++)
      if (tasks[i].route == ROUTE_HERMITE) {
        sum += tasks[i].n;
        num++;
        most = std::max(most, tasks[i].n);
      }
    nsrc += sum;
    n[p] += sum;
    cnt[p] += num;
  }
  // Sources per partial block: at most 4096, fewer (whole batches of the
  // kernel) where that leaves SMs without a CTA
  if (P.dim == 3) {
    const int batch = P.ifdipole ? FORM3_SB / 3 : FORM3_SB;
    R.chunk = (int)std::min<long long>(4096 / batch, std::max<long long>(6, nsrc / (8LL * sms * batch))) * batch;
    return R;
  }
  // 2D: about eight chunks per SM of at least 512 sources, whole passes of
  // the kernels' four warps (four leaves of 75000 sources in four CTAs took
  // 0.76 ms of a 0.80 ms execute, 0.02 of 0.08 cut up)
  R.chunk = (int)std::max<long long>(512, (nsrc / (8LL * sms) + 255) / 256 * 256);
  // leaves (or chunks) of about two blocks of source columns or less, a warp each
  if (most > R.chunk)
    for (const FormTask& f : tasks)
      if (f.route == ROUTE_HERMITE && f.n > R.chunk) cnt[f.p] += (f.n + R.chunk - 1) / R.chunk - 1;
  R.warp.resize(n.size());
  for (size_t p = 0; p < n.size(); p++) R.warp[p] = n[p] * (P.ifdipole ? 2 : 1) <= 80 * cnt[p];
  return R;
}
// Taylor evaluation: the orders evaluated from blocks (the others from the
// columns, 3D) and, in 2D, the warps per task of k_eval2d_mma (0: Horner).
struct EvalRules {
  std::vector<uint8_t> blocks, per;
};
EvalRules eval_rules(const Params& P, const std::vector<int>& nlocal, const std::vector<EvalTask>& tasks, int pgh) {
  EvalRules R;
  const int np = P.ntermmax + 1, n2 = P.npw / 2;
  R.blocks.assign(np, P.dim == 2);
  R.per.assign(np, 0);
  if (P.dim == 2) {
    // k_eval2d_mma where it is the faster one (its comment), with as many
    // warps per task as have points
    bool some = false;  // a level of such an order
    for (int l = std::max(P.npwlevel, 0); l <= P.nlevels; l++) some = some || (nlocal[l] >= 24 && nlocal[l] < 40);
    if (!some) return R;
    std::vector<long long> n(np, 0), cnt(np, 0);
    for (size_t i = 0; i < tasks.size();) {
      const int p = tasks[i].p;
      long long sum = 0, num = 0;
      for (; i < tasks.size() && tasks[i].p == p; i++)
        if (tasks[i].route == ROUTE_TAYLOR) {
          sum += tasks[i].n;
          num += tasks[i].n <= 256 ? 1 : (tasks[i].n + 255) / 256;
        }
      n[p] += sum;
      cnt[p] += num;
    }
    const long long tile = pgh <= 1 ? 16 : 8;
    for (int p = 24; p < std::min(40, np); p++)
      if (n[p] <= 72 * cnt[p]) R.per[p] = n[p] > 3 * tile * cnt[p] ? 4 : n[p] > tile * cnt[p] ? 2 : 1;
    return R;
  }
  // Multiply-adds on the FP64 pipe of the two ways, each with what its
  // kernels lose beside them (measured, 3D, eps 1e-6 and 1e-9): a leaf's
  // block costs P^3 (n2 + 44) (44: its two passes over memory) and its
  // points 2 P^3 per 32 begun; the column way 1.5 * 2 n2 P^2 per 8 points
  // begun.  Mixed potentials up to order 15 are evaluated on the BF16
  // tensor cores from the blocks; rows above 30 coefficients have no
  // block evaluation.
  std::vector<long long> leaves(np, 0), n32(np, 0), n8(np, 0);
  for (size_t t = 0; t < tasks.size();) {
    const int p = tasks[t].p;
    long long num = 0, m32 = 0, m8 = 0;
    for (; t < tasks.size() && tasks[t].p == p; t++) {
      const EvalTask& e = tasks[t];
      if (e.route != ROUTE_TAYLOR) continue;
      num += t == 0 || tasks[t - 1].box != e.box;  // a leaf's tasks are consecutive
      m32 += (e.n + 31) / 32;
      m8 += (e.n + 7) / 8;
    }
    leaves[p] += num;
    n32[p] += 32 * m32;
    n8[p] += 8 * m8;
  }
  for (int p = 0; p < np; p++) {
    const double Pn = p + 1, P3 = Pn * Pn * Pn;
    const double cb = P3 * (n2 + 44) * leaves[p] + 2.0 * P3 * pgh * n32[p];
    const double cc = 3.0 * n2 * Pn * Pn * pgh * n8[p];
    R.blocks[p] = Pn <= 30 && ((Pn <= 16 && pgh == 1 && !P.ifdipole) || cb < cc);
  }
  return R;
}

cudaError_t device_plan_create(const HostPlan& H, DevicePlan& D, const int* d_isrc, const int* d_itarg,
                               cudaStream_t pst, size_t* size_only) {
  const auto tnow = [] {
    return std::chrono::duration<double>(std::chrono::steady_clock::now().time_since_epoch()).count();
  };
  const double tin = tnow();
  double tp[4];
  int np_ = 0;
  D = DevicePlan();
  D.P = H.P;
  const Params& P = H.P;
  D.nboxes = H.tree.nboxes;
  D.nch = 1 << P.dim;
  int dev = 0;
  CK(cudaGetDevice(&dev));
  CK(cudaDeviceGetAttribute(&D.sm_count, cudaDevAttrMultiProcessorCount, dev));
  double tq[4];
  int nq = 0;
  tq[nq++] = tnow();
  // order form and eval tasks by route so each kernel gets a contiguous range
  // (then by order; stable)
  std::vector<FormTask> form;
  std::vector<EvalTask> ev;
  beside(H.form.size() > 2048, [&] { form = route_order_sort(H.form); }, [&] { ev = route_order_sort(H.eval); });
  D.nform = (int)form.size();
  for (auto& f : form) {
    (f.route == ROUTE_PW ? D.form_pw_n : D.form_hermite_n)++;
    if (f.route == ROUTE_HERMITE) D.form_pmax = std::max(D.form_pmax, f.p);
  }
  D.neval = (int)ev.size();
  for (auto& e : ev) {
    (e.route == ROUTE_PW ? D.eval_pw_n : D.eval_taylor_n)++;
    if (e.route == ROUTE_TAYLOR) D.eval_pmax = std::max(D.eval_pmax, e.p);
    else D.eval_pw_max = std::max(D.eval_pw_max, e.n);
  }
  // Plane-wave scheme: the Hermite leaves in the order of the columns (and
  // slabs) of their cut-level boxes, and the leaves formed from exponential sums
  const int lcut = std::max(P.npwlevel, 0);
  const bool sep = P.scheme == 0 && !P.all_direct;
  if (sep)  // the plane-wave route evaluates the cut-level box's expansion about its centre
    for (int t = D.eval_taylor_n; t < D.neval; t++)
      while (H.tree.level[ev[t].box] > lcut) ev[t].box = H.tree.parent[ev[t].box];
  SepLists up;
  std::vector<BlockSum> sums;   // leaves of several partial blocks
  std::vector<PwFormTask> pwf;  // 3D boxes formed from exponential sums
  std::vector<SrcRange> pwf_src;
  std::vector<double> sep_ph;
  size_t hbuf_doubles = 0;  // the leaves' (partial) Hermite blocks
  std::vector<std::pair<int, int>> run;  // a leaf's Taylor tasks, by its number in the list below
  SepRows sep_rows;
  uvector<SepItem> sep_items;  // every leaf at or below the cut level, in the order of the lists
  std::vector<int> sep_order_of;   // order by depth below the cut level
  if (sep) {
    const Tree& tr = H.tree;
    // the leaves that a form or a Taylor task needs, those of the form tasks
    // first, with their Taylor tasks [run.first, run.second) (a leaf's are
    // consecutive)
    uvector<int> num(tr.nboxes);
#pragma omp parallel for schedule(static) if (tr.nboxes > 16384)
    for (int b = 0; b < tr.nboxes; b++) num[b] = -1;
    std::vector<int> boxes(D.nform);
    boxes.reserve(D.nform + D.eval_taylor_n);
    for (int i = 0; i < D.nform; i++) {
      num[form[i].box] = i;
      boxes[i] = form[i].box;
    }
    run.resize(D.nform + D.eval_taylor_n, {0, 0});
    for (int t = 0, u; t < D.eval_taylor_n; t = u) {
      const int b = ev[t].box;
      for (u = t + 1; u < D.eval_taylor_n && ev[u].box == b;) u++;
      if (num[b] < 0) {
        num[b] = (int)boxes.size();
        boxes.push_back(b);
      }
      run[num[b]] = {t, u};
    }
    for (int l = lcut; l <= P.nlevels; l++) sep_order_of.push_back(H.nlocal[l]);
    sep_order(tr, lcut, boxes, sep_rank(sep_order_of), sep_items, sep_rows);
    sep_phases(H, sep_rows, tr.boxsize[lcut], sep_ph);
  }
  std::vector<long long> form_hoff;
  // Taylor evaluation: point chunks of <= 256 that read a leaf's block
  std::vector<HornerTask> horner;
  size_t lo_doubles = 0;
  // The Taylor leaves in the order of the columns (and slabs) of their
  // cut-level boxes, in 3D each order group either with Taylor blocks or
  // evaluated from the columns
  SepLists dn;
  std::vector<ColTask> ctask;
  uvector<SepItem> dn_items;
  std::vector<long long> first;   // first task of every item
  FormRules frules;
  EvalRules erules;
  long long nh = 0, nct = 0;
  double eval_flops = 0.0;  // per density, without the way down
  const int pgh = std::max(1, std::max(P.ifpgh, P.ifpghtarg)), cp = sep_col_points(pgh);
  auto build_up = [&] {
    const int* mp_slot = H.mp_slot.data() + H.tree.lfirst[lcut];
    const std::vector<FormTask> in(form.begin(), form.begin() + D.form_hermite_n);
    uvector<SepItem> items(D.form_hermite_n), pw;
    std::vector<SepLeaf> leaf(D.form_hermite_n);
    std::vector<int> box(D.form_hermite_n);
    int ni = 0;
    long long hoff = 0;
    frules = form_rules(P, H.form_of_all.empty() ? H.form : H.form_of_all, D.sm_count);
    D.form_chunk = frules.chunk;
    const int chunk = D.form_chunk;
    for (const SepItem& s : sep_items) {
      const int i = s.num;
      if (i >= D.nform) continue;
      if (i >= D.form_hermite_n) {
        pw.push_back(s);
        continue;
      }
      const FormTask& f = form[ni] = in[i];
      const int n = f.n <= chunk ? 1 : (f.n + chunk - 1) / chunk;
      items[ni] = s;
      box[ni] = s.box;
      const int len = (f.p + 1) * (f.p + 1) * (P.dim == 3 ? f.p + 1 : 1);
      const bool sum = n > (P.dim == 2 ? 1 : SUM_BLOCKS3D);
      leaf[ni++] = {hoff, 0, sum ? 1 : n};
      if (sum) sums.push_back({hoff * P.nd, len, n});
      hoff += (long long)n * len;
    }
    hbuf_doubles = (size_t)hoff * P.nd;
    // the boxes formed from exponential sums; `add` where leaves below add to them
    std::stable_sort(pw.begin(), pw.end(), [](const SepItem& a, const SepItem& b) { return a.root < b.root; });
    std::vector<int> has;  // the roots of the other leaves
    if (!pw.empty()) {
      for (const SepItem& s : items) has.push_back(s.root);
      std::sort(has.begin(), has.end());
    }
    for (size_t i = 0; i < pw.size(); i++) {
      const FormTask& f = form[pw[i].num];
      const int r = pw[i].root;
      if (i == 0 || pw[i - 1].root != r)
        pwf.push_back({H.tree.lfirst[lcut] + r, mp_slot[r], (int)pwf_src.size(), 0,
                       std::binary_search(has.begin(), has.end(), r)});
      pwf_src.push_back({f.s0, f.n});
      pwf.back().cnt++;
    }
    D.up_box.swap(box);
    D.up_leaf = leaf;
    sep_lists(P.dim, items, sep_rows, leaf, sep_order_of, mp_slot, -1, P.npw, up);
    // 2D: the source chunks as tasks of their own, each with its partial block
    if (P.dim == 2 && sums.empty()) {
      std::vector<long long> off(form.size());
      for (size_t t = 0; t < off.size(); t++) off[t] = D.up_leaf[t].off * P.nd;
      form_hoff.swap(off);
    } else if (P.dim == 2) {
      std::vector<FormTask> ch;
      ch.reserve(form.size());
      for (int t = 0; t < D.form_hermite_n; t++) {
        const FormTask& f = form[t];
        const long long P2 = (long long)(f.p + 1) * (f.p + 1);
        for (int c = 0, b = 0; c < f.n; c += D.form_chunk, b++) {
          FormTask g = f;
          g.s0 = f.s0 + c;
          g.n = std::min(D.form_chunk, f.n - c);
          ch.push_back(g);
          form_hoff.push_back((D.up_leaf[t].off + b * P2) * P.nd);
        }
      }
      form.swap(ch);
      D.form_hermite_n = (int)form.size();
    }
  };
  auto build_down = [&] {
    uvector<SepItem> items(sep_items.size());
    int ni = 0;
    for (const SepItem& s : sep_items)
      if (run[s.num].second > 0) items[ni++] = s;
    items.resize(ni);
    erules = eval_rules(P, H.nlocal, H.eval_of_all.empty() ? H.eval : H.eval_of_all, pgh);
    const std::vector<uint8_t>& blocks = erules.blocks;
    std::vector<long long> len(sep_order_of.size());  // doubles of a block, by depth
    for (size_t d = 0; d < len.size(); d++) {
      const long long p = sep_order_of[d], Pn = p + 1, E = (Pn + 1) & ~1LL;
      len[d] = blocks[p] ? P.nd * Pn * E * (P.dim == 3 ? Pn : 1) : 0;
    }
    std::vector<SepLeaf> leaf(ni);
    long long lo = 0;
    for (int i = 0; i < ni; i++) {
      leaf[i] = {lo, 0, 1};
      lo += len[items[i].d];
    }
    lo_doubles = (size_t)lo;
    sep_lists(P.dim, items, sep_rows, leaf, sep_order_of, H.loc_slot.data() + H.tree.lfirst[lcut], -1, P.npw, dn);
    // first task of every item, the groups' ranges; the tasks below
    std::vector<long long> at0(ni);
    for (SepGroup& G : dn.groups) {
      G.blocks = blocks[G.p];
      const int step = G.blocks ? 256 : cp;
      const long long t0 = G.blocks ? nh : nct;
      long long n = 0, at = t0;
      const int i0 = dn.cols[G.cbeg].beg, i1 = dn.cols[G.cend - 1].beg + dn.cols[G.cend - 1].cnt;
      for (int i = i0; i < i1; i++) {
        const std::pair<int, int> r = run[items[i].num];
        at0[i] = at;
        for (int t = r.first; t < r.second; t++) {
          at += ev[t].n <= step ? 1 : (ev[t].n + step - 1) / step;
          n += ev[t].n;
        }
      }
      const double Pn = G.p + 1, n2 = P.npw / 2;
      // a block's Horner sums; from a column the z sums and the product with them
      eval_flops += 2.0 * pgh * n * (G.blocks ? std::pow(Pn, P.dim) : 2.0 * n2 * Pn * (Pn + 1.0));
      (G.blocks ? nh : nct) = at;
      (G.blocks ? D.horner_groups : D.ctask_groups).push_back({G.p, (int)t0, (int)at});
      if (G.blocks) D.horner_groups.back().per = erules.per[G.p];
    }
    dn_items.swap(items);
    first.swap(at0);
  };
  if (sep) beside(sep_items.size() > 2048, build_up, build_down);
  if (P.dim == 3 && P.scheme == 1)  // the NUFFT scheme: every box by itself
    for (const FormTask& f : form) {
      pwf.push_back({f.box, f.slot, (int)pwf_src.size(), 1, 0});
      pwf_src.push_back({f.s0, f.n});
    }
  tq[nq++] = tnow();
  // launch groups of equal order among the Hermite form tasks
  for (int t = 0; t < D.form_hermite_n;) {
    int u = t;
    while (u < D.form_hermite_n && form[u].p == form[t].p) u++;
    D.form_groups.push_back({form[t].p, t, u});
    if (P.dim == 2 && sep) D.form_groups.back().warp = frules.warp[form[t].p];
    t = u;
  }

  // dominant form group (most sources) for the per-kernel roofline of the bench
  if (P.dim == 2) {
    long long best = -1;
    for (size_t gi = 0; gi < D.form_groups.size(); gi++) {
      const OrderGroup& G = D.form_groups[gi];
      long long n = 0;
      for (int t = G.beg; t < G.end; t++) n += form[t].n;
      const double Pn = G.p + 1;
      D.group_flops.push_back(2.0 * (double)n * Pn * Pn * P.nd);
      D.group_alg_flops.push_back(4.0 * (double)n * P.npw * P.npw * P.nd);
      if (n > best) { best = n; D.dom_form_group = (int)gi; }
    }
  }
  tp[np_++] = tnow();
  if (sep) {
    const uvector<SepItem>& items = dn_items;
    horner.resize(nh);
    ctask.resize(nct);
    const int ncol = (int)dn.cols.size();
#pragma omp parallel for schedule(static) if (ncol > 1024)
    for (int c = 0; c < ncol; c++)
      for (int l = dn.cols[c].beg; l < dn.cols[c].beg + dn.cols[c].cnt; l++) {
        const std::pair<int, int> r = run[items[l].num];
        long long at = first[l];
        for (int t = r.first; t < r.second; t++) {
          const EvalTask& e = ev[t];
          if (erules.blocks[e.p])
            for (int q = 0; q < e.n; q += 256)
              horner[at++] = {e.box, e.set, e.i0 + q, std::min(256, e.n - q), e.p, dn.leaves[l].off};
          else
            for (int q = 0; q < e.n; q += cp)
              ctask[at++] = {e.box, e.set, e.i0 + q, std::min(cp, e.n - q), dn.leaves[l].row, e.p + 1, dn.cols[c].off};
        }
      }
  }
  tp[np_++] = tnow();
  D.nm2l = (int)H.m2l.size();
  D.ndir = (int)(H.dnear.mem ? H.dnear.ndir : (long long)H.dir.size());
  D.nmp = H.nmp;
  D.nloc = H.nloc;
  D.direct_pairs = H.direct_pairs;
  D.form_sources = H.form_sources;
  D.eval_points = H.eval_points;
  tp[np_++] = tnow();
  // 3D: source chunks and their partial Hermite blocks
  std::vector<FormChunk> fchunks;
  if (P.dim == 3 && !P.all_direct) {
    if (D.form_hermite_n > 0) {
      long long hoff = 0;
      for (int t = 0; t < D.form_hermite_n; t++) {
        const FormTask& f = form[t];
        long long p3 = (long long)(f.p + 1) * (f.p + 1) * (f.p + 1);
        for (int c = 0; c < f.n; c += D.form_chunk) {
          fchunks.push_back({t, f.s0 + c, std::min(D.form_chunk, f.n - c), hoff});
          hoff += p3;
        }
      }
      D.nfchunks = (int)fchunks.size();
      // chunk ranges of equal order (the tasks are sorted by order)
      long long best = -1;
      for (size_t t = 0; t < fchunks.size();) {
        size_t u = t;
        const int pt = form[fchunks[t].task].p;
        long long n = 0;
        while (u < fchunks.size() && form[fchunks[u].task].p == pt) n += fchunks[u++].n;
        const double Pn = pt + 1;
        D.group_flops.push_back(2.0 * (double)n * Pn * Pn * Pn * P.nd);
        D.group_alg_flops.push_back(4.0 * (double)n * P.npw * P.npw * P.npw * P.nd);
        if (n > best) { best = n; D.dom_fchunk_group = (int)D.fchunk_groups.size(); }
        D.fchunk_groups.push_back({pt, (int)t, (int)u});
        t = u;
      }
    }
  }
  // flops of the routes taken.  Plane-wave sums: in 3D two real products of half
  // the nodes per coefficient, in 2D (the NUFFT scheme) a complex one
  {
    const double cols = P.ifdipole ? P.dim : 1, pw = (P.dim == 3 ? 4.0 : 8.0) * P.nexp;
    double f = 0.0, e = eval_flops;
    for (double g : D.group_flops) f += cols * g;  // the Hermite blocks, every density
    for (int t = D.form_hermite_n; t < (int)form.size(); t++) f += cols * pw * form[t].n * P.nd;
    for (int t = D.eval_taylor_n; t < D.neval; t++) e += pw * pgh * ev[t].n;
    if (sep) {
      f += P.nd * sep_flops(P.dim, true, up, P.npw);
      e += sep_flops(P.dim, false, dn, P.npw);
    }
    D.form_route_flops = f;
    D.eval_route_flops = P.nd * e;
  }
  size_t ns = P.ns, nt = P.nt, nd = P.nd, dim = P.dim;
  // FP32 coordinates of the mixed near field (charges only)
  const bool fmix = D.ndir > 0 && !P.ifdipole;
  // mp -> loc rows (formed on the device)
  const size_t n_wsh = P.all_direct ? 0 : (size_t)(P.dim == 2 ? 9 : 27) * P.nexp;
  size_t total = bytes_of(H.box_centers) + bytes_of(H.h2x) + bytes_of(H.x2l) + bytes_of(H.hx) + al(n_wsh * 16) + al(H.w1.size() * 8) + 2 * al((size_t)P.ns * 4) + 2 * al((size_t)P.nt * 4) +
                 al((size_t)(std::max(P.ntermmax, 1) + 2) * 8) +
                 bytes_of(form) +
                 bytes_of(H.m2l) + bytes_of(H.m2l_nbr) + bytes_of(ev) + bytes_of(H.dir) +
                 al((size_t)H.dnear.ndir * sizeof(DirTask)) + al((size_t)H.dnear.nsrc * sizeof(SrcRange)) +
                 bytes_of(H.dir_src) + al((size_t)H.nmp * nd * P.nexp * 16) +
                 al((size_t)H.nloc * nd * P.nexp * 16) + al(ns * dim * 8) + al(ns * nd * 8) +
                 al(nt * dim * 8) + al(ns * nd * out_comps(dim, P.ifpgh) * 8) +
                 (fmix ? al(ns * dim * 8) + al((P.ifpghtarg > 0 ? nt : 0) * dim * 8) : 0) +
                 al(P.ifdipole ? ns * dim * 8 : 0) + al(P.ifdipole ? ns * nd * 8 : 0) +
                 al(nt * nd * out_comps(dim, P.ifpghtarg) * 8) +
                 bytes_of(fchunks) +
                 bytes_of(up.leaves) + bytes_of(up.cols) + bytes_of(up.slabs) + bytes_of(up.boxes) +
                 bytes_of(up.box_kids) + bytes_of(dn.cols) + bytes_of(dn.leaves) + bytes_of(dn.slabs) +
                 bytes_of(dn.boxes) + bytes_of(dn.box_kids) + bytes_of(dn.col_slot) + bytes_of(dn.leaf_col) + bytes_of(sums) + bytes_of(ctask) + bytes_of(pwf) + bytes_of(pwf_src) + bytes_of(sep_ph) +
                 al(std::max(up.t1, dn.t1) * nd * 8) + al(std::max(up.t2, dn.t2) * nd * 8) +
                 al(hbuf_doubles * 8) + bytes_of(form_hoff) + bytes_of(horner) +
                 al(lo_doubles * 8) + 4096;
  D.bytes = total;
  if (size_only) {
    *size_only = total;
    return cudaSuccess;
  }
  const double tm0 = tnow();
  D.stream = pst;
  CK(device_pool_setup());
  CK(cudaMallocAsync(reinterpret_cast<void**>(&D.base), total, pst));
  const double tm1 = tnow();
  char* cur = D.base;
  cudaStream_t s = pst;
  // Everything that goes up from the host, laid out in the arena as it
  // comes, goes in one copy from a pinned mirror of that range (filled by the
  // host threads); no pageable copy (each would wait for the stream) and no
  // synchronisation here: the kernels below follow the copy on the stream.
  std::vector<double2> w1(H.w1.size() / 2);
  memcpy(w1.data(), H.w1.data(), H.w1.size() * 8);
  std::vector<double> isq(std::max(P.ntermmax, 1) + 2, 0.0);
  for (size_t j = 1; j < isq.size(); j++) isq[j] = 1.0 / std::sqrt((double)j);
  double2* d_w1 = nullptr;
  {
    char* const b0 = cur;
    Staged st;
    st.add(cur, D.centers, H.box_centers);
    st.add(cur, D.h2x, H.h2x);
    st.add(cur, D.x2l, H.x2l);
    st.add(cur, D.hx, H.hx);
    st.add(cur, d_w1, w1);
    st.add(cur, D.isq, isq);
    st.add(cur, D.form, form);
    st.add(cur, D.m2l, H.m2l);
    st.add(cur, D.m2l_nbr, H.m2l_nbr);
    st.add(cur, D.eval, ev);
    if (!H.dnear.mem) {  // else built on the device: copied after this block
      st.add(cur, D.dir, H.dir);
      st.add(cur, D.dir_src, H.dir_src);
    }
    st.add(cur, D.fchunks, fchunks);
    st.add(cur, D.up.leaves, up.leaves);
    st.add(cur, D.up.cols, up.cols);
    st.add(cur, D.up.slabs, up.slabs);
    st.add(cur, D.up.boxes, up.boxes);
    st.add(cur, D.up.box_kids, up.box_kids);
    st.add(cur, D.dn.leaves, dn.leaves);
    st.add(cur, D.dn.cols, dn.cols);
    st.add(cur, D.dn.slabs, dn.slabs);
    st.add(cur, D.dn.boxes, dn.boxes);
    st.add(cur, D.dn.box_kids, dn.box_kids);
    st.add(cur, D.dn.col_slot, dn.col_slot);
    st.add(cur, D.dn.leaf_col, dn.leaf_col);
    st.add(cur, D.form_sums, sums);
    D.form_nsums = (int)sums.size();
    st.add(cur, D.ctask, ctask);
    st.add(cur, D.pwf, pwf);
    st.add(cur, D.pwf_src, pwf_src);
    double* ph = nullptr;
    st.add(cur, ph, sep_ph);
    D.up.ph = reinterpret_cast<double2*>(ph);
    D.up.nboxes = (int)up.boxes.size();
    D.up.groups = up.groups;
    D.dn.ph = D.up.ph;
    D.up.hx = P.dim == 3 ? D.h2x : D.hx;
    D.up.sms = D.dn.sms = D.sm_count;
    D.dn.nboxes = (int)dn.boxes.size();
    D.dn.groups = dn.groups;
    D.npwf = (int)pwf.size();
    st.add(cur, D.form_hoff, form_hoff);
    st.add(cur, D.horner, horner);
    CK(st.upload(b0, s));
  }
  // mp -> loc rows formed on the device from their 1D factors
  D.wsh = reinterpret_cast<double2*>(cur); cur += al(n_wsh * 16);
  if (n_wsh > 0) {
    const int blocks = (int)std::min<size_t>((n_wsh + 255) / 256, (size_t)D.sm_count * 16);
    k_shift_tables<<<blocks, 256, 0, s>>>(P.dim, P.npw, P.nexp, d_w1, D.wsh);
    CK(cudaGetLastError());
  }
  std::vector<int> inv[2];  // until the copies below have ended
  if (d_isrc) {
    // permutations built on the device (fgt_devtree.cu): copy, invert there;
    // targets that are the sources share the sources' arrays
    auto carve = [&](int*& dst, size_t n) {
      dst = reinterpret_cast<int*>(cur);
      cur += al(n * 4);
    };
    const bool same = H.same_points && P.nt == P.ns;
    carve(D.isrc, P.ns);
    carve(D.isrc_inv, P.ns);
    if (same) {
      D.itarg = D.isrc;
      D.itarg_inv = D.isrc_inv;
    } else {
      carve(D.itarg, P.nt);
      carve(D.itarg_inv, P.nt);
    }
    if (P.ns > 0) {
      CK(cudaMemcpyAsync(D.isrc, d_isrc, (size_t)P.ns * 4, cudaMemcpyDeviceToDevice, pst));
      k_invperm<<<(P.ns + 255) / 256, 256, 0, pst>>>(D.isrc, P.ns, D.isrc_inv);
    }
    if (P.nt > 0 && !same) {
      CK(cudaMemcpyAsync(D.itarg, d_itarg, (size_t)P.nt * 4, cudaMemcpyDeviceToDevice, pst));
      k_invperm<<<(P.nt + 255) / 256, 256, 0, pst>>>(D.itarg, P.nt, D.itarg_inv);
    }
  } else {
    CK(put(cur, D.isrc, H.tree.isrc, s));
    CK(put(cur, D.itarg, H.tree.itarg, s));
    const std::vector<int>* perm[2] = {&H.tree.isrc, &H.tree.itarg};
    for (int k = 0; k < 2; k++) {
      inv[k].resize(perm[k]->size());
      for (size_t i = 0; i < inv[k].size(); i++) inv[k][(*perm[k])[i]] = (int)i;
      CK(put(cur, k ? D.itarg_inv : D.isrc_inv, inv[k], s));
    }
  }
  if (H.dnear.mem) {
    D.dir = reinterpret_cast<DirTask*>(cur);
    cur += al((size_t)H.dnear.ndir * sizeof(DirTask));
    D.dir_src = reinterpret_cast<SrcRange*>(cur);
    cur += al((size_t)H.dnear.nsrc * sizeof(SrcRange));
    if (H.dnear.ndir)
      CK(cudaMemcpyAsync(D.dir, H.dnear.dir, (size_t)H.dnear.ndir * sizeof(DirTask), cudaMemcpyDeviceToDevice, s));
    if (H.dnear.nsrc)
      CK(cudaMemcpyAsync(D.dir_src, H.dnear.src, (size_t)H.dnear.nsrc * sizeof(SrcRange), cudaMemcpyDeviceToDevice,
                         s));
  }
  D.lo = reinterpret_cast<double*>(cur); cur += al(lo_doubles * 8);
  D.hbuf = reinterpret_cast<double*>(cur); cur += al(hbuf_doubles * 8);
  // the intermediates of the two directions, one after the other
  D.up.t1 = D.dn.t1 = reinterpret_cast<double*>(cur); cur += al(std::max(up.t1, dn.t1) * nd * 8);
  D.up.t2 = D.dn.t2 = reinterpret_cast<double*>(cur); cur += al(std::max(up.t2, dn.t2) * nd * 8);
  D.mp = reinterpret_cast<double2*>(cur); cur += al((size_t)H.nmp * nd * P.nexp * 16);
  D.loc = reinterpret_cast<double2*>(cur); cur += al((size_t)H.nloc * nd * P.nexp * 16);
  D.ssort = reinterpret_cast<double*>(cur); cur += al(ns * dim * 8);
  D.csort = reinterpret_cast<double*>(cur); cur += al(ns * nd * 8);
  D.nsort = reinterpret_cast<double*>(cur); cur += al(P.ifdipole ? ns * dim * 8 : 0);
  D.dsort = reinterpret_cast<double*>(cur); cur += al(P.ifdipole ? ns * nd * 8 : 0);
  D.tsort = reinterpret_cast<double*>(cur); cur += al(nt * dim * 8);
  if (fmix) {
    D.fsrc = reinterpret_cast<float*>(cur); cur += al(ns * dim * 8);
    D.ftrg = reinterpret_cast<float*>(cur); cur += al((P.ifpghtarg > 0 ? nt : 0) * dim * 8);
  }
  D.psort = reinterpret_cast<double*>(cur); cur += al(ns * nd * out_comps(dim, P.ifpgh) * 8);
  D.ptsort = reinterpret_cast<double*>(cur); cur += al(nt * nd * out_comps(dim, P.ifpghtarg) * 8);
  CK(cudaStreamSynchronize(s));
  if (getenv("FGT_TREE_TIMING"))
    fprintf(stderr, "device plan prep parts: route sort %.4f up lists %.4f down lists and tasks %.4f rest %.4f\n",
            tq[1] - tin, tp[0] - tq[1], tp[1] - tp[0], tm0 - tp[1]);
  if (getenv("FGT_TREE_TIMING"))
    fprintf(stderr, "device plan: prep %.4f malloc %.4f upload %.4f (%zu bytes); eval tasks: taylor %d "
            "(max order %d) pw %d; form tasks: hermite %d (max order %d) pw %d\n",
            tm0 - tin, tm1 - tm0, tnow() - tm1, total, D.eval_taylor_n,
            D.eval_pmax + 1, D.eval_pw_n, D.form_hermite_n,
            D.form_pmax + 1, D.form_pw_n);
  return cudaSuccess;
}

void device_plan_destroy(DevicePlan& D) {
  if (D.base) cudaFreeAsync(D.base, D.stream);
  D.base = nullptr;
}

void device_plan_set_grids(DevicePlan& D, int sms, bool yield) {
  // no grid of theirs reaches 12 CTAs per SM of 2^24
  D.up.sms = D.dn.sms = yield ? 1 << 24 : sms > 0 ? std::min(sms, D.sm_count) : D.sm_count;
}

static KP make_kp(const DevicePlan& D) {
  KP k;
  const Params& P = D.P;
  k.dim = P.dim; k.nd = P.nd; k.npw = P.npw; k.n2 = P.npw / 2; k.nexp = P.nexp;
  k.dsq = P.dsq; k.delta = P.delta; k.dmax = P.dmax;
  k.t1 = P.npw > 0 ? 0.5 * P.pmax / (P.npw / 2) : 0.0;
  k.centers = D.centers; k.h2x = D.h2x; k.x2l = D.x2l; k.ws = nullptr;
  k.wsh = D.wsh; k.mp = D.mp; k.loc = D.loc;
  k.src = D.ssort; k.chg = D.csort; k.trg = D.tsort; k.pot = D.psort; k.pottarg = D.ptsort;
  k.nc_s = out_comps(P.dim, P.ifpgh);
  k.nc_t = out_comps(P.dim, P.ifpghtarg);
  k.ifcharge = P.ifcharge;
  k.ifdipole = P.ifdipole;
  k.dnrm = D.nsort;
  k.dstr = D.dsort;
  k.fsrc = D.fsrc;
  k.ftrg = D.ftrg;
  return k;
}

// node weights for the direct 3D form kernel live in the x2l/h2x neighbourhood:
// ws(k) = h2x[0 * npw + k] (j = 0 row of h2x is ws_k).
cudaError_t device_check_finite(const double* x, size_t n, int* d_flag, cudaStream_t st) {
  if (n == 0) return cudaSuccess;
  int dev = 0, sms = 148;
  CK(cudaGetDevice(&dev));
  CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  const size_t blocks = std::min<size_t>((n + 255) / 256, (size_t)sms * 8);
  k_all_finite<<<(unsigned)blocks, 256, 0, st>>>(x, n, d_flag);
  return cudaGetLastError();
}

cudaError_t device_plan_set_points(DevicePlan& D, const double* src, const double* trg,
                                   cudaStream_t st) {
  const Params& P = D.P;
  const int gb = std::max(1, std::min(8 * D.sm_count, (std::max(P.ns, P.nt) + 255) / 256));
  if (P.ns > 0) {
    const int vec = (reinterpret_cast<uintptr_t>(src) & 15) == 0;
    k_gather_pts<<<gb, 256, 0, st>>>(src, nullptr, D.ssort, nullptr, D.isrc, P.ns, P.dim, P.nd, vec);
  }
  if (P.nt > 0 && P.ifpghtarg > 0) {
    const int vec = (reinterpret_cast<uintptr_t>(trg) & 15) == 0;
    k_gather_pts<<<gb, 256, 0, st>>>(trg, nullptr, D.tsort, nullptr, D.itarg, P.nt, P.dim, P.nd, vec);
  }
  if (D.fsrc) {
    const double cs = std::sqrt(1.4426950408889634 / P.delta);
    if (P.ns > 0)
      k_mixed_coords<<<gb, 256, 0, st>>>(D.ssort, P.ns, P.dim, P.cen0[0], P.cen0[1], P.cen0[2], cs, D.fsrc);
    if (P.nt > 0 && P.ifpghtarg > 0)
      k_mixed_coords<<<gb, 256, 0, st>>>(D.tsort, P.nt, P.dim, P.cen0[0], P.cen0[1], P.cen0[2], cs, D.ftrg);
  }
  return cudaGetLastError();
}

// Runs launch(std::integral_constant<int, G>) with G = pgh in {1, 2, 3}.
template <class F>
cudaError_t with_pgh(int pgh, F&& launch) {
  switch (pgh) {
    case 1: return launch(std::integral_constant<int, 1>());
    case 2: return launch(std::integral_constant<int, 2>());
    case 3: return launch(std::integral_constant<int, 3>());
    default: return cudaErrorNotSupported;
  }
}

cudaError_t device_plan_execute(DevicePlan& D, const Inputs& in, const Outputs& outs,
                                int precision, cudaStream_t st, StageTimes* times, int phase) {
  const Params& P = D.P;
  // phase 1: gather, form, merge (the cut level's mp expansions);
  // phase 2: mp -> loc, split, eval, near field, scatter; 0: both
  const bool ph1 = phase != 2, ph2 = phase != 1;
  KP k = make_kp(D);
  // the derivative order the kernels compute: the larger of the two sets'
  const int pgh = std::max(1, std::max(P.ifpgh, P.ifpghtarg));
  // mixed form of stages (a) and (c): FP32 arithmetic with FP64 accumulation
  // in the 2D Hermite block and Taylor evaluation (charges, potentials)
  const bool mixed_ac = precision == PREC_MIXED && !P.ifdipole;
  k.ws = D.h2x;  // row j = 0 of h2x holds the weights
  const int nd = P.nd;
  cudaEvent_t ev[9], dev0 = nullptr, dev1 = nullptr;
  if (times) {
    for (int i = 0; i < 9; i++) CK(cudaEventCreate(&ev[i]));
    CK(cudaEventCreate(&dev0));
    CK(cudaEventCreate(&dev1));
    times->dom_ms = 0;
    times->dom_flops = 0;
    times->dom_alg_flops = 0;
    times->dom_name[0] = 0;
  }
  auto mark = [&](int i) { if (times) cudaEventRecord(ev[i], st); };
  long long launches = 0;
  mark(0);
  // charges into tree order (coordinates were sorted once, at plan set-up)
  const int gb = std::max(1, std::min(8 * D.sm_count, (std::max(P.ns, P.nt) + 255) / 256));
  if (ph1 && P.ns > 0 && P.ifcharge) {
    if (nd == 1) k_gather1<<<gb, 256, 0, st>>>(in.charge, D.isrc, P.ns, D.csort);
    else k_gather_pts<<<gb, 256, 0, st>>>(nullptr, in.charge, nullptr, D.csort, D.isrc, P.ns, P.dim, nd, 0);
    launches++;
  }
  if (ph1 && P.ns > 0 && P.ifdipole) {  // directions and strengths of the dipoles
    k_gather_pts<<<gb, 256, 0, st>>>(in.rnormal, in.dipstr, D.nsort, D.dsort, D.isrc, P.ns, P.dim, nd, 0);
    launches++;
  }
  if (ph1 && P.ifpgh > 0 && P.ns > 0) CK(cudaMemsetAsync(D.psort, 0, (size_t)P.ns * nd * k.nc_s * 8, st));
  if (ph1 && P.ifpghtarg > 0 && P.nt > 0) CK(cudaMemsetAsync(D.ptsort, 0, (size_t)P.nt * nd * k.nc_t * 8, st));
  mark(1);
  const int n2 = P.npw / 2;
  const int echunks = (int)std::min<long long>(65535, ((long long)nd * P.nexp + 255) / 256);
  if (!P.all_direct) {
   if (ph1) {
    // (a) form
    if (P.dim == 2 && D.form_hermite_n > 0) {
      for (size_t gi = 0; gi < D.form_groups.size(); gi++) {
        const OrderGroup& G = D.form_groups[gi];
        const int Pn = G.p + 1;
        const FormTask* tk = D.form + G.beg;
        const int ntk = G.end - G.beg;
        const bool dom = times && (int)gi == D.dom_form_group;
        if (dom) cudaEventRecord(dev0, st);
        // one block of P <= 32 rows and columns, of 24 beyond (order 41: four
        // blocks of 24 hold 48, of 32 would hold 64)
#define FORM_MMA(NT)                                                                                         \
  do {                                                                                                       \
    const size_t sh = (size_t)4 * 2 * (8 * NT) * 36 * 8;                                                     \
    const int nb = (Pn + 8 * NT - 1) / (8 * NT);                                                             \
    const dim3 g(G.warp ? (ntk + 3) / 4 : ntk, nd, nb * nb);                                                 \
    auto run = [&](auto kernel) -> cudaError_t {                                                             \
      CK(smem_limit(kernel));                                                                                \
      kernel<<<g, 128, sh, st>>>(k, tk, ntk, D.form_hoff + G.beg, D.hbuf);                                   \
      return cudaSuccess;                                                                                    \
    };                                                                                                       \
    if (P.ifdipole) CK(G.warp ? run(k_form2d_mma<NT, true, true>) : run(k_form2d_mma<NT, true, false>));     \
    else CK(G.warp ? run(k_form2d_mma<NT, false, true>) : run(k_form2d_mma<NT, false, false>));              \
  } while (0)
        if (mixed_ac && Pn <= 16) CK(launch_form2d_f32(k, tk, G.end - G.beg, nd, D.form_hoff + G.beg, D.hbuf, Pn, st));
        else if (Pn <= 8) FORM_MMA(1);
        else if (Pn <= 16) FORM_MMA(2);
        else if (Pn <= 24 || Pn > 32) FORM_MMA(3);
        else FORM_MMA(4);
#undef FORM_MMA
        if (dom) {
          cudaEventRecord(dev1, st);
          if (mixed_ac && Pn <= 16) snprintf(times->dom_name, sizeof(times->dom_name), "k_form2d_f32");
          else snprintf(times->dom_name, sizeof(times->dom_name), "k_form2d_mma<%d>", Pn > 32 ? 3 : (Pn + 7) / 8);
          times->dom_flops = D.group_flops[gi];
          times->dom_alg_flops = D.group_alg_flops[gi];
        }
        launches++;
      }
    }
    if (P.dim == 3 && D.form_hermite_n > 0) {
      for (size_t gi = 0; gi < D.fchunk_groups.size(); gi++) {
        const OrderGroup& G = D.fchunk_groups[gi];
        const int Pn = G.p + 1, mt = (Pn + 7) / 8;
        const bool dom = times && (int)gi == D.dom_fchunk_group;
        if (dom) cudaEventRecord(dev0, st);
        const size_t sh = form3_smem(Pn);
        const dim3 fg(G.end - G.beg, nd);
        const FormChunk* ch = D.fchunks + G.beg;
        // The tcgen05 Hermite blocks (BF16 x 3) only on request: building
        // their Pn^2 split operand rows per source costs more than the FP64
        // DMMA kernel's whole block (3D blobs, Pn = 14: form 4.2 vs 3.45 ms),
        // so the mixed form keeps the FP64 blocks by default.
        const bool tc_form = getenv("FGT_FORM3D_TC") != nullptr;
        if (mixed_ac && tc_form && form3d_tc_supported(Pn)) {
          // mixed form: the Hermite blocks as BF16 x 3 tensor-core products
          CK(launch_form3d_tc(k, D.form, ch, G.end - G.beg, nd, Pn, D.hbuf, D.isq, st));
          if (dom) {
            cudaEventRecord(dev1, st);
            snprintf(times->dom_name, sizeof(times->dom_name), "k_form3d_tc<%d>", Pn);
            times->dom_flops = D.group_flops[gi];
            times->dom_alg_flops = D.group_alg_flops[gi];
          }
          launches++;
          continue;
        }
#define FORM3_CASE(PMAX)                                                                          \
  else if (Pn <= PMAX) {                                                                          \
    constexpr int MT = (PMAX + 7) / 8, KQ = form3_kq(PMAX), NL = form3_nlp(PMAX);                 \
    if (P.ifdipole) {                                                                             \
      CK(smem_limit(k_form3d_mma<MT, KQ, NL, true>));                                             \
      k_form3d_mma<MT, KQ, NL, true><<<fg, 128, sh, st>>>(k, D.form, ch, D.hbuf, D.isq);          \
    } else {                                                                                      \
      CK(smem_limit(k_form3d_mma<MT, KQ, NL, false>));                                            \
      k_form3d_mma<MT, KQ, NL, false><<<fg, 128, sh, st>>>(k, D.form, ch, D.hbuf, D.isq);         \
    }                                                                                             \
  }
        if (Pn > 32) return cudaErrorNotSupported;
        FORM3_CASE(8) FORM3_CASE(12) FORM3_CASE(16) FORM3_CASE(24) FORM3_CASE(32)
#undef FORM3_CASE
        if (dom) {
          cudaEventRecord(dev1, st);
          snprintf(times->dom_name, sizeof(times->dom_name), "k_form3d_mma<%d>", mt);
          times->dom_flops = D.group_flops[gi];
          times->dom_alg_flops = D.group_alg_flops[gi];
        }
        launches++;
      }
    }
    if (D.form_nsums > 0) {
      k_sum_blocks<<<dim3(D.form_nsums, 32), 256, 0, st>>>(D.form_sums, nd, D.hbuf);
      launches++;
    }
    if (P.dim == 2 && D.form_pw_n > 0) {  // the NUFFT scheme's direct form
      const size_t sh = (size_t)FORM_CH * (P.npw + n2) * 16;
      if (sh > 227 * 1024) return cudaErrorNotSupported;
      CK(smem_limit(k_form2d_pw));
      k_form2d_pw<<<dim3(D.form_pw_n, nd), 256, sh, st>>>(k, D.form + D.form_hermite_n);
      launches++;
    }
    mark(2);
    // (b) the leaves' blocks to the cut level's expansions
    if (D.up.nboxes > 0) {
      CK(sep_up(k, D.up, D.hbuf, st, launches));
    }
    if (D.npwf > 0) CK(launch_form3d_pw(k, D.pwf, D.npwf, D.pwf_src, st, launches));
   }  // phase 1
    mark(3);
   if (ph2) {
    if (D.nm2l > 0) {
      k_m2l<<<dim3(D.nm2l, echunks), 256, 0, st>>>(k, D.m2l, D.m2l_nbr);
      launches++;
    }
    mark(4);
    mark(5);
    // (c) eval
    // the blocks that the mixed 2D evaluation reads are written as FP32 pairs
    // (the condition of its launch below)
    if (D.dn.nboxes > 0) CK(sep_down(k, D.dn, D.lo, mixed_ac && pgh == 1 ? 32 : 0, st, launches));
    if (P.dim == 2 && D.neval > 0) {
      for (const OrderGroup& G : D.horner_groups) {
        const int Pn = G.p + 1, np2 = (Pn + 1) / 2;
        const dim3 g(G.end - G.beg, nd);
        const HornerTask* tk = D.horner + G.beg;
        const size_t sh = (size_t)Pn * np2 * 16;
        if (sh > 227 * 1024) return cudaErrorNotSupported;
        if (mixed_ac && pgh == 1 && np2 <= 16) {
          CK(launch_eval2d_horner_f32(k, tk, G.end - G.beg, nd, Pn, D.lo, st));
          launches++;
          continue;
        }
        if (G.per > 0) {
          const dim3 gw((unsigned)(((long long)(G.end - G.beg) * G.per + 3) / 4), nd);
          const cudaError_t e2 = with_pgh(pgh, [&](auto PG) -> cudaError_t {
            switch ((Pn + 3) / 4) {
#define EVAL2_CASE(N) \
  case N: k_eval2d_mma<N, decltype(PG)::value><<<gw, 128, 0, st>>>(k, tk, G.end - G.beg, G.per, D.lo); break;
              EVAL2_CASE(7) EVAL2_CASE(8) EVAL2_CASE(9) EVAL2_CASE(10)
#undef EVAL2_CASE
              default: return cudaErrorNotSupported;
            }
            return cudaSuccess;
          });
          CK(e2);
          launches++;
          continue;
        }
        {
          const cudaError_t e_pgh = with_pgh(pgh, [&](auto G) -> cudaError_t {
          constexpr int PG = decltype(G)::value;
          switch (np2) {
#define HORNER_CASE(N)                                                                            \
  case N:                                                                                         \
    CK(smem_limit(k_eval2d_horner<N, PG>)); \
    k_eval2d_horner<N, PG><<<g, 128, sh, st>>>(k, tk, D.lo);                                      \
    break;
            HORNER_CASE(1) HORNER_CASE(2) HORNER_CASE(3) HORNER_CASE(4) HORNER_CASE(5) HORNER_CASE(6)
            HORNER_CASE(7) HORNER_CASE(8) HORNER_CASE(9) HORNER_CASE(10) HORNER_CASE(11) HORNER_CASE(12)
            HORNER_CASE(13) HORNER_CASE(14) HORNER_CASE(15) HORNER_CASE(16) HORNER_CASE(17) HORNER_CASE(18)
            HORNER_CASE(19) HORNER_CASE(20) HORNER_CASE(21) HORNER_CASE(22) HORNER_CASE(23) HORNER_CASE(24)
            HORNER_CASE(25) HORNER_CASE(26) HORNER_CASE(27) HORNER_CASE(28) HORNER_CASE(29) HORNER_CASE(30)
            HORNER_CASE(31) HORNER_CASE(32)
#undef HORNER_CASE
            default:
              CK(smem_limit(k_eval2d_horner_any<PG>));
              k_eval2d_horner_any<PG><<<g, 128, sh, st>>>(k, tk, D.lo);
          }
          return cudaSuccess;
        });
          CK(e_pgh);
        }
        launches++;
      }
      if (D.eval_pw_n > 0) {
        {
          const cudaError_t e_pgh = with_pgh(pgh, [&](auto G) -> cudaError_t {
          k_eval2d<decltype(G)::value><<<dim3(D.eval_pw_n, nd), 256, 0, st>>>(k, D.eval + D.eval_taylor_n);
          return cudaSuccess;
        });
          CK(e_pgh);
        }
        launches++;
      }
    }
    if (P.dim == 3 && D.dn.nboxes > 0) {
      for (const OrderGroup& G : D.ctask_groups) {
        CK(sep_eval_cols(k, D.dn, D.ctask + G.beg, G.end - G.beg, G.p + 1, pgh, st));
        launches++;
      }
      for (const OrderGroup& G : D.horner_groups) {
        const int Pn = G.p + 1, np2 = (Pn + 1) / 2;
        const dim3 g(G.end - G.beg, nd);
        const HornerTask* tk = D.horner + G.beg;
        const size_t sh = (size_t)Pn * Pn * np2 * 16;
        if (sh > 227 * 1024) return cudaErrorNotSupported;
        if (mixed_ac && pgh == 1 && eval3d_tc_supported(Pn)) {
          // mixed form: the Taylor evaluation as BF16 x 3 tensor-core products
          CK(launch_eval3d_tc(k, tk, G.end - G.beg, nd, Pn, D.lo, st));
          launches++;
          continue;
        }
        {
          const cudaError_t e_pgh = with_pgh(pgh, [&](auto G) -> cudaError_t {
          constexpr int PG = decltype(G)::value;
          switch (np2) {
#define HORNER3_CASE(N)                                                                           \
  case N:                                                                                         \
    CK(smem_limit(k_eval3d_horner<N, PG>)); \
    k_eval3d_horner<N, PG><<<g, 128, sh, st>>>(k, tk, D.lo);                                      \
    break;
            HORNER3_CASE(1) HORNER3_CASE(2) HORNER3_CASE(3) HORNER3_CASE(4) HORNER3_CASE(5)
            HORNER3_CASE(6) HORNER3_CASE(7) HORNER3_CASE(8) HORNER3_CASE(9) HORNER3_CASE(10)
            HORNER3_CASE(11) HORNER3_CASE(12) HORNER3_CASE(13) HORNER3_CASE(14) HORNER3_CASE(15)
#undef HORNER3_CASE
            default: return cudaErrorNotSupported;
          }
          return cudaSuccess;
        });
          CK(e_pgh);
        }
        launches++;
      }
    }
    if (P.dim == 3 && D.eval_pw_n > 0) {  // the plane-wave route
      CK(launch_eval3d_pw(k, D.eval + D.eval_taylor_n, D.eval_pw_n, D.eval_pw_max, pgh, st));
      launches++;
    }
   }  // phase 2
  } else {
    mark(2); mark(3); mark(4); mark(5);
  }
  mark(6);
  // (d) near field
  if (ph2 && D.ndir > 0) {
    dim3 g((D.ndir + 3) / 4, nd);
    // dipoles take the FP64 near field (the mixed form is charges only)
    const bool mixed = precision == PREC_MIXED && !P.ifdipole;
    const double l2e = 1.4426950408889634;
    const double cs = std::sqrt(l2e / P.delta);
    const float amax = (float)(P.dmax * l2e / P.delta);
    if (mixed && pgh == 1) {
      // potentials only: the packed-FP32 kernel
      CK(launch_direct_mixed_x2(k, D.dir, D.ndir, nd, D.dir_src, amax, st));
    } else {
          const cudaError_t e_pgh = with_pgh(pgh, [&](auto G) -> cudaError_t {
      constexpr int PG = decltype(G)::value;
      if (P.dim == 2) {
        if (mixed) k_direct_mixed<2, PG><<<g, 128, 0, st>>>(k, D.dir, D.ndir, D.dir_src, cs, amax);
        else if (P.ifdipole) k_direct<2, PG, true><<<g, 128, 0, st>>>(k, D.dir, D.ndir, D.dir_src);
        else k_direct<2, PG, false><<<g, 128, 0, st>>>(k, D.dir, D.ndir, D.dir_src);
      } else {
        if (mixed) k_direct_mixed<3, PG><<<g, 128, 0, st>>>(k, D.dir, D.ndir, D.dir_src, cs, amax);
        else if (P.ifdipole) k_direct<3, PG, true><<<g, 128, 0, st>>>(k, D.dir, D.ndir, D.dir_src);
        else k_direct<3, PG, false><<<g, 128, 0, st>>>(k, D.dir, D.ndir, D.dir_src);
      }
      return cudaSuccess;
    });
          CK(e_pgh);
        }
    launches++;
  }
  mark(7);
  // sorted rows [nc][nd] -> pot (nd, n), grad (nd, dim, n), hess (nd, H, n)
  const int nh = P.dim == 2 ? 3 : 6;
  auto unsort = [&](const double* in, const int* inv, int n, int nc, double* pot, double* grad,
                    double* hess) {
    // one density, one component per point: the random gather of the charges
    if (!pot && (nc == 1 || (!grad && !hess))) return;
    if (nd == 1 && nc == 1) k_gather1<<<gb, 256, 0, st>>>(in, inv, n, pot);
    else {
      const int w1 = nc > 1 ? P.dim * nd : 0, w2 = nc > 1 + P.dim ? nh * nd : 0;
      const long long ctas = ((long long)n * (nd + w1 + w2) + 255) / 256;
      k_unsort<<<(int)std::min<long long>(8 * D.sm_count, ctas), 256, 0, st>>>(in, inv, n, nd, w1, w2, pot, grad, hess);
    }
    launches++;
  };
  if (ph2 && P.ifpgh > 0 && P.ns > 0) unsort(D.psort, D.isrc_inv, P.ns, k.nc_s, outs.pot, outs.grad, outs.hess);
  if (ph2 && P.ifpghtarg > 0 && P.nt > 0)
    unsort(D.ptsort, D.itarg_inv, P.nt, k.nc_t, outs.pottarg, outs.gradtarg, outs.hesstarg);
  mark(8);
  D.launches = launches;
  CK(cudaGetLastError());
  if (times) {
    CK(cudaEventSynchronize(ev[8]));
    // stage i spans marks i..i+1; the shift stages merge/m2l/split are 2..5
    float t[8];
    for (int i = 0; i < 8; i++) cudaEventElapsedTime(&t[i], ev[i], ev[i + 1]);
    for (int i = 0; i < 8; i++) times->ms[i] = t[i];
    if (times->dom_name[0]) cudaEventElapsedTime(&times->dom_ms, dev0, dev1);
    for (int i = 0; i < 9; i++) cudaEventDestroy(ev[i]);
    cudaEventDestroy(dev0);
    cudaEventDestroy(dev1);
  }
  return cudaSuccess;
}

cudaError_t device_plan_box_expansion(const HostPlan& H, DevicePlan& D, int box, double* out, cudaStream_t st) {
  const Tree& t = H.tree;
  const Params& P = H.P;
  const int lb = t.level[box];
  auto inside = [&](int b) {
    while (t.level[b] > lb) b = t.parent[b];
    return b == box;
  };
  std::vector<int> boxes, at(t.nboxes, -1);
  for (size_t i = 0; i < D.up_box.size(); i++)
    if (inside(D.up_box[i])) {
      boxes.push_back(D.up_box[i]);
      at[D.up_box[i]] = (int)i;
    }
  PwFormTask pw{box, 0, 0, 0, 1};
  std::vector<SrcRange> pw_src;
  for (const FormTask& f : H.form)
    if (f.route == ROUTE_PW && inside(f.box)) {
      pw_src.push_back({f.s0, f.n});
      pw.cnt++;
    }
  std::vector<int> order;
  for (int l = lb; l <= P.nlevels; l++) order.push_back(H.nlocal[l]);
  uvector<SepItem> items;
  SepRows rows;
  sep_order(t, lb, boxes, sep_rank(order), items, rows);
  std::vector<SepLeaf> leaf;
  for (const SepItem& s : items) leaf.push_back(D.up_leaf[at[s.box]]);
  std::vector<int> slot(t.llast[lb] - t.lfirst[lb] + 1, -1);
  slot[box - t.lfirst[lb]] = 0;
  SepLists L;
  sep_lists(P.dim, items, rows, leaf, order, slot.data(), box - t.lfirst[lb], P.npw, L);
  std::vector<double> ph;
  sep_phases(H, rows, t.boxsize[lb], ph);
  const std::vector<PwFormTask> pwt(1, pw);
  const size_t nd = P.nd, per = nd * P.nexp * 16;
  char* mem = nullptr;
  CK(cudaMallocAsync(reinterpret_cast<void**>(&mem),
                     bytes_of(L.leaves) + bytes_of(L.cols) + bytes_of(L.slabs) + bytes_of(L.boxes) +
                         bytes_of(L.box_kids) + bytes_of(ph) + bytes_of(pwt) + bytes_of(pw_src) + al(L.t1 * nd * 8) +
                         al(L.t2 * nd * 8) + al(per) + 4096,
                     st));
  auto run = [&]() -> cudaError_t {
    char* cur = mem;
    SepDev S;
    PwFormTask* dpw = nullptr;
    SrcRange* dsrc = nullptr;
    double* dph = nullptr;
    CK(put(cur, S.leaves, L.leaves, st));
    CK(put(cur, S.cols, L.cols, st));
    CK(put(cur, S.slabs, L.slabs, st));
    CK(put(cur, S.boxes, L.boxes, st));
    CK(put(cur, S.box_kids, L.box_kids, st));
    CK(put(cur, dph, ph, st));
    CK(put(cur, dpw, pwt, st));
    CK(put(cur, dsrc, pw_src, st));
    S.ph = reinterpret_cast<double2*>(dph);
    S.nboxes = 1;
    S.groups = L.groups;
    S.sms = D.sm_count;
    S.hx = D.up.hx;
    S.t1 = reinterpret_cast<double*>(cur); cur += al(L.t1 * nd * 8);
    S.t2 = reinterpret_cast<double*>(cur); cur += al(L.t2 * nd * 8);
    KP k = make_kp(D);
    k.ws = D.h2x;  // row j = 0
    k.mp = reinterpret_cast<double2*>(cur);
    long long launches = 0;
    CK(sep_up(k, S, D.hbuf, st, launches));
    CK(launch_form3d_pw(k, dpw, pw.cnt > 0 ? 1 : 0, dsrc, st, launches));
    CK(cudaMemcpyAsync(out, k.mp, per, cudaMemcpyDeviceToHost, st));
    return cudaStreamSynchronize(st);
  };
  const cudaError_t e = run();
  cudaFreeAsync(mem, st);
  return e;
}

cudaError_t probe_fp64_mma(double* tflops) {
  int dev = 0, sms = 148;
  CK(cudaGetDevice(&dev));
  CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  cudaEvent_t e0, e1;
  CK(cudaEventCreate(&e0));
  CK(cudaEventCreate(&e1));
  const int iters = 4096, blocks = sms * 16;
  k_probe_dmma<<<blocks, 128>>>(nullptr, 64);  // warm-up
  CK(cudaEventRecord(e0));
  k_probe_dmma<<<blocks, 128>>>(nullptr, iters);
  CK(cudaEventRecord(e1));
  CK(cudaEventSynchronize(e1));
  float ms = 0;
  cudaEventElapsedTime(&ms, e0, e1);
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  const double fma = (double)blocks * 4 * 8 * 256 * iters;
  *tflops = 2.0 * fma / (ms * 1e-3) / 1e12;
  return cudaGetLastError();
}

size_t large_delta_work_doubles(const Params& P, bool deterministic) {
  const size_t Pn = P.nlocal0 + 1;
  const size_t nent = P.dim == 2 ? Pn * Pn : Pn * Pn * Pn;
  return (size_t)P.nd * nent * (deterministic ? 1 + LD_PARTS : 1);
}

cudaError_t large_delta_execute(const Params& P, const double* src, const Inputs& in,
                                const double* trg, const Outputs& outs, double* work,
                                cudaStream_t st, bool deterministic) {
  KP k;
  memset(&k, 0, sizeof(k));
  k.dim = P.dim; k.nd = P.nd; k.dsq = P.dsq; k.delta = P.delta;
  k.src = src; k.chg = in.charge;
  k.ifcharge = P.ifcharge; k.ifdipole = P.ifdipole;
  k.dnrm = in.rnormal; k.dstr = in.dipstr;  // caller order: this path sorts nothing
  int p = P.nlocal0;
  int Pn = p + 1;
  size_t nent = P.dim == 2 ? (size_t)Pn * Pn : (size_t)Pn * Pn * Pn;
  // the centre travels by value in the kernel arguments (no host->device copy)
  const double3 cen = make_double3(P.cen0[0], P.cen0[1], P.dim == 3 ? P.cen0[2] : 0.0);
  double* local = work;
  CK(cudaMemsetAsync(local, 0, nent * P.nd * sizeof(double), st));
  size_t sh = 3 * FORM_CH * Pn * 8;
  if (sh > 227 * 1024) return cudaErrorNotSupported;
  if (sh > 48 * 1024) {
    CK(smem_limit(k_ld_form<2>));
    CK(smem_limit(k_ld_form<3>));
  }
  // deterministic: per-CTA partial blocks after the local block, summed in
  // CTA order; otherwise atomic accumulation (last-bit order dependence)
  double* partial = deterministic ? local + nent * P.nd : nullptr;
  int blocks = std::max(1, std::min(deterministic ? LD_PARTS : 1024, (P.ns + 255) / 256));
  if (P.ns > 0) {
    if (P.dim == 2) k_ld_form<2><<<dim3(blocks, P.nd), 256, sh, st>>>(k, P.ns, p, cen, local, partial);
    else k_ld_form<3><<<dim3(blocks, P.nd), 256, sh, st>>>(k, P.ns, p, cen, local, partial);
    if (deterministic) {
      const int sb = std::max(1, std::min(1024, (int)((nent + 255) / 256)));
      k_ld_sum<<<dim3(sb, P.nd), 256, 0, st>>>((int)nent, blocks, partial, local);
    }
  }
  auto ev = [&](const double* pts, int n, int pgh, double* pot, double* grad, double* hess) -> cudaError_t {
    if (n <= 0 || pgh <= 0) return cudaSuccess;
    int b = std::max(1, std::min(4096, (n + 255) / 256));
    return with_pgh(pgh, [&](auto G) -> cudaError_t {
      constexpr int PG = decltype(G)::value;
      if (P.dim == 2) k_ld_eval<2, PG><<<dim3(b, P.nd), 256, 0, st>>>(k, n, pts, pot, grad, hess, p, cen, local);
      else k_ld_eval<3, PG><<<dim3(b, P.nd), 256, 0, st>>>(k, n, pts, pot, grad, hess, p, cen, local);
      return cudaSuccess;
    });
  };
  CK(ev(trg, P.nt, P.ifpghtarg, outs.pottarg, outs.gradtarg, outs.hesstarg));
  CK(ev(src, P.ns, P.ifpgh, outs.pot, outs.grad, outs.hess));
  return cudaGetLastError();
}


// ------------------------------------------------------------ allocation-free large-delta call
// Some callers cannot let this library allocate device memory: codes that
// hand over device arrays from their own pool and run under a fixed memory
// budget, and latency-critical loops that must not pay for cudaMalloc, which
// can synchronise the whole device.  For them the large-delta transform (one
// Taylor local about a given centre, the reference's fgt2d_large_delta /
// fgt3d_large_delta) runs with its only scratch -- the local expansion -- in
// this fixed device array.  Every device that loads the
// library holds it (512 KB) until the process exits; every call shares it, so
// calls that overlap on the GPU race; each call clears what it accumulates.
namespace {
constexpr size_t kNoAllocScratchDoubles = 65536;
__device__ __align__(256) double g_noalloc_scratch[kNoAllocScratchDoubles + 8];
std::mutex g_noalloc_mu;
double* g_noalloc_ptr[64] = {nullptr};
}  // namespace

size_t large_delta_noalloc_capacity() { return kNoAllocScratchDoubles; }

cudaError_t large_delta_noalloc(const Params& P, const double* src, const double* chg,
                                const double* trg, double* pot, double* pottarg, cudaStream_t st) {
  const size_t Pn = (size_t)P.nlocal0 + 1;
  const size_t nent = P.dim == 2 ? Pn * Pn : Pn * Pn * Pn;
  if (P.nlocal0 < 0 || nent * P.nd > kNoAllocScratchDoubles) return cudaErrorInvalidValue;
  int dev = 0;
  CK(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  double* work = nullptr;
  {
    // the host name of the array is not a device address: its address on
    // this device is looked up once, with this device current
    std::lock_guard<std::mutex> lk(g_noalloc_mu);
    if (!g_noalloc_ptr[dev]) {
      void* ptr = nullptr;
      CK(cudaGetSymbolAddress(&ptr, g_noalloc_scratch));
      g_noalloc_ptr[dev] = static_cast<double*>(ptr);
    }
    work = g_noalloc_ptr[dev];
  }
  // the source staging of the local-expansion kernel grows with the order
  const int sh = (int)(3 * FORM_CH * Pn * 8);
  if (sh > 48 * 1024) {
    CK(smem_limit(k_ld_form<2>));
    CK(smem_limit(k_ld_form<3>));
  }
  // large_delta_execute clears the local expansion (work[0..nd*nent)) on the
  // stream before accumulating into it; the centre goes by value in the
  // kernel arguments, so the call makes no host->device copy
  Outputs o;
  o.pot = pot;
  o.pottarg = pottarg;
  Inputs in;
  in.charge = chg;
  return large_delta_execute(P, src, in, trg, o, work, st, false);
}

}  // namespace fgtb
