// Separable 3D transforms over the subtree of each cut-level box.
//
// The plane-wave expansions below the cut level serve one purpose on the way
// up: their shifted sum is the cut-level box's expansion (merge).  Shift and
// Hermite -> plane-wave transform are both tensor products, so the sum is
// taken one dimension at a time, where the leaves share it:
//
//   PW_A(kx, ky, kz) = sum_ix px(ix, kx) sum_jx i^jx hx[jx][kx]
//                      sum_iy py(iy, ky) sum_jy i^jy hx[jy][ky]
//                      sum_iz pz(iz, kz) sum_jz i^jz hx[jz][kz] H_b[jx][jy][jz]
//
// over the leaves b = (ix, iy, iz) of A, p(i, k) = exp(-i t_k sh_i) with sh_i
// the offset of box i from A's centre.  The z transform runs once per leaf,
// the y transform once per column of leaves and the x transform, the largest,
// once per slab of columns; no expansion below the cut level is formed.  This
// replaces a whole transform of every leaf (g3dh2pw_real_vec,
// g3drouts.f:1565-1685) and the merge over the levels (g3dshiftpw_vec):
// the same sums in another order.
//
// What bounds the kernels: the latency of their operand loads at the few warps
// that their registers allow (18 to 28% of the SM's; FP64 tensor pipe 20 to
// 33%, DRAM 25 to 43% in ncu); every operand is read once from global memory
// straight into the fragment that needs it, so there is no shared memory and
// the warps are independent.  Measured against
// a whole transform per leaf and level-by-level merges (B200, transforms and
// merges of one execute): 4e6 blob sources, eps 1e-6, 2.75 -> 0.85 ms; 3e5
// uniform points, eps 1e-9, delta 1e-3, 4.95 -> 1.38 ms; eps 1e-12, delta
// 1e-2, 24.2 -> 0.42 ms (orders whose whole transform did not fit in shared
// memory ran on the scalar pipes).
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <type_traits>

#include "fgt_kcommon.cuh"
#include "fgt_sep.hpp"

namespace fgtb {

namespace {

// ------------------------------------------------------------ upward
// z pass: T1[m][kz] = sum over the column's leaves of pz(kz) (E + i O),
// E/O = sum over even / odd l of H[l][m] hs[l][kz] with the signed table
// hs[l] = (-1)^(l/2) h2x[l], m = jx + P jy, kz over the tiles t0 .. t0 + MT - 1
// of the stored node half.  One CTA of four independent warps per column (and
// share of its row tiles); a warp owns eight rows m, keeps the MT node tiles
// of the table in registers and the sum over the leaves in its accumulators.
// A fragment reads eight consecutive doubles of four rows l; the next leaf's
// are loaded before this leaf's products.
template <int KS, int MT>
__global__ void __launch_bounds__(128) k_up_z(KP k, const SepNode* __restrict__ cols,
                                              const SepLeaf* __restrict__ leaves, int Pn, int t0,
                                              const double* __restrict__ hbuf, double* __restrict__ T1,
                                              const double2* __restrict__ ph) {
  const SepNode C = cols[blockIdx.x];
  const int ind = blockIdx.z, npw = k.npw, n2 = k.n2, P2 = Pn * Pn, P3 = P2 * Pn;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, r = lane >> 2, c = lane & 3;
  double hz[MT][2][KS];
#pragma unroll
  for (int t = 0; t < MT; t++)
#pragma unroll
    for (int par = 0; par < 2; par++)
#pragma unroll
      for (int s = 0; s < KS; s++) {
        const int j = 8 * s + 2 * c + par, kz = 8 * (t0 + t) + r;
        const bool ok = j < Pn && kz < n2;
        hz[t][par][s] = ok ? ((j & 2) ? -k.h2x[j * npw + kz] : k.h2x[j * npw + kz]) : 0.0;
      }
  double* out = T1 + (size_t)C.off * k.nd + (size_t)ind * P2 * n2 * 2;
  const int mtiles = (P2 + 7) / 8;
  for (int mt = blockIdx.y * 4 + warp; mt < mtiles; mt += gridDim.y * 4) {
    const int m = 8 * mt + r, mm = min(m, P2 - 1);
    auto load = [&](int q, double (&a)[2][KS], int& row) {
      const SepLeaf L = leaves[q];
      row = L.row * npw;
      const double* H = hbuf + (size_t)L.off * k.nd + (size_t)ind * P3 + mm;
#pragma unroll
      for (int s = 0; s < KS; s++)
#pragma unroll
        for (int par = 0; par < 2; par++) {
          const int j = 8 * s + 2 * c + par;
          a[par][s] = j < Pn ? H[j * P2] : 0.0;
        }
      for (int ch = 1; ch < L.n; ch++) {  // the few further partial blocks, in chunk order
        const double* Hc = H + (size_t)ch * P3 * k.nd;
#pragma unroll
        for (int s = 0; s < KS; s++)
#pragma unroll
          for (int par = 0; par < 2; par++) {
            const int j = 8 * s + 2 * c + par;
            a[par][s] += j < Pn ? Hc[j * P2] : 0.0;
          }
      }
    };
    double acc[MT][4];
#pragma unroll
    for (int t = 0; t < MT; t++) acc[t][0] = acc[t][1] = acc[t][2] = acc[t][3] = 0.0;
    double an[2][KS];
    int rown;
    load(C.beg, an, rown);
    for (int q = C.beg; q < C.beg + C.cnt; q++) {
      double a[2][KS];
      const int row = rown;
#pragma unroll
      for (int s = 0; s < KS; s++) {
        a[0][s] = an[0][s];
        a[1][s] = an[1][s];
      }
      if (q + 1 < C.beg + C.cnt) load(q + 1, an, rown);
#pragma unroll
      for (int t = 0; t < MT; t++) {
        double e0 = 0.0, e1 = 0.0, o0 = 0.0, o1 = 0.0;
#pragma unroll
        for (int s = 0; s < KS; s++) {
          dmma_884(e0, e1, a[0][s], hz[t][0][s]);
          dmma_884(o0, o1, a[1][s], hz[t][1][s]);
        }
        const int kz = min(8 * (t0 + t) + 2 * c, n2 - 1), kz1 = min(kz + 1, n2 - 1);
        const double2 p0 = __ldg(ph + row + kz), p1 = __ldg(ph + row + kz1);
        // (E + i O) conj(p)
        acc[t][0] += e0 * p0.x + o0 * p0.y;
        acc[t][1] += o0 * p0.x - e0 * p0.y;
        acc[t][2] += e1 * p1.x + o1 * p1.y;
        acc[t][3] += o1 * p1.x - e1 * p1.y;
      }
    }
    if (m < P2) {
      double2* o = reinterpret_cast<double2*>(out) + (size_t)m * n2;
#pragma unroll
      for (int t = 0; t < MT; t++) {
        const int kz = 8 * (t0 + t) + 2 * c;
        if (kz < n2) o[kz] = make_double2(acc[t][0], acc[t][1]);
        if (kz + 1 < n2) o[kz + 1] = make_double2(acc[t][2], acc[t][3]);
      }
    }
  }
}

// y pass (Y: the columns of a slab) and x pass (the slabs of a box): a child
// holds T[j][col], j < its order, complex columns contiguous; its sums over
// even and odd j against the positive node half, E and O, are turned by the
// child's phase and added, and the node and its mirror get E + i O and
// E - i O:
//   Y: col = (jx, kz) -> T2[jx][(kz, ky)],   X: col = (kz, ky) -> the box's
//   expansion [(kz, ky)][kx].
// CTAs of four independent warps; a warp owns four complex columns and the
// node tiles t0 .. t0 + MT - 1; Pm is the largest order + 1 of the children.
template <int KS, int MT, bool Y>
__global__ void __launch_bounds__(128) k_up_xy(KP k, const SepNode* __restrict__ nodes,
                                               const SepNode* __restrict__ kids, const int* __restrict__ idx,
                                               int Pm, int t0, const double* __restrict__ Tin,
                                               double* __restrict__ Tout, const double2* __restrict__ ph) {
  const SepNode N = nodes[blockIdx.x];
  const int ind = blockIdx.z, npw = k.npw, n2 = k.n2;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, r = lane >> 2, c = lane & 3;
  const int ncol = Y ? N.p * n2 : n2 * npw;
  double hn[MT][2][KS];
#pragma unroll
  for (int t = 0; t < MT; t++)
#pragma unroll
    for (int par = 0; par < 2; par++)
#pragma unroll
      for (int s = 0; s < KS; s++) {
        const int j = 8 * s + 2 * c + par, m = 8 * (t0 + t) + r;
        const bool ok = j < Pm && m < n2;
        hn[t][par][s] = ok ? ((j & 2) ? -k.h2x[j * npw + n2 + m] : k.h2x[j * npw + n2 + m]) : 0.0;
      }
  double2* out = Y ? reinterpret_cast<double2*>(Tout + (size_t)N.off * k.nd) + (size_t)ind * N.p * n2 * npw
                   : k.mp + ((size_t)N.off * k.nd + ind) * k.nexp;
  const int ntiles = (ncol + 3) / 4;
  for (int nt = blockIdx.y * 4 + warp; nt < ntiles; nt += gridDim.y * 4) {
    const int col = min(8 * nt + r, 2 * ncol - 1);
    auto load = [&](int q, double (&b)[2][KS], int& row) {
      const SepNode K = kids[idx ? idx[q] : q];
      row = K.row * npw;
      const double* T = Tin + (size_t)K.off * k.nd + (size_t)ind * 2 * K.p * ncol + col;
#pragma unroll
      for (int s = 0; s < KS; s++)
#pragma unroll
        for (int par = 0; par < 2; par++) {
          const int j = 8 * s + 2 * c + par;
          b[par][s] = j < K.p ? T[(size_t)j * 2 * ncol] : 0.0;
        }
    };
    double acc[MT][4];
#pragma unroll
    for (int t = 0; t < MT; t++) acc[t][0] = acc[t][1] = acc[t][2] = acc[t][3] = 0.0;
    double bn[2][KS];
    int rown = 0;
    if (N.cnt > 0) load(N.beg, bn, rown);
    for (int q = N.beg; q < N.beg + N.cnt; q++) {
      double b[2][KS];
      const int row = rown;
#pragma unroll
      for (int s = 0; s < KS; s++) {
        b[0][s] = bn[0][s];
        b[1][s] = bn[1][s];
      }
      if (q + 1 < N.beg + N.cnt) load(q + 1, bn, rown);
#pragma unroll
      for (int t = 0; t < MT; t++) {
        double e0 = 0.0, e1 = 0.0, o0 = 0.0, o1 = 0.0;
#pragma unroll
        for (int s = 0; s < KS; s++) {
          dmma_884(e0, e1, hn[t][0][s], b[0][s]);
          dmma_884(o0, o1, hn[t][1][s], b[1][s]);
        }
        // the node's phase is conj(p), its mirror's p: E' = cr E + ci O and
        // O' = cr O - ci E give E' + i O' and E' - i O'
        const double2 p = __ldg(ph + row + n2 + min(8 * (t0 + t) + r, n2 - 1));
        acc[t][0] += p.x * e0 + p.y * o0;
        acc[t][1] += p.x * e1 + p.y * o1;
        acc[t][2] += p.x * o0 - p.y * e0;
        acc[t][3] += p.x * o1 - p.y * e1;
      }
    }
    const int q = 4 * nt + c;  // the lane's complex column
    if (q < ncol) {
#pragma unroll
      for (int t = 0; t < MT; t++) {
        const int m = 8 * (t0 + t) + r;
        if (m < n2) {
          const double2 vp = make_double2(acc[t][0] - acc[t][3], acc[t][1] + acc[t][2]);
          const double2 vm = make_double2(acc[t][0] + acc[t][3], acc[t][1] - acc[t][2]);
          double2* o = Y ? out + (size_t)(q / n2) * n2 * npw + (q % n2) * npw : out + (size_t)q * npw;
          o[n2 + m] = vp;
          o[n2 - 1 - m] = vm;
        }
      }
    }
  }
}

// ------------------------------------------------------------ downward
// The mirror image: the cut level's local expansions to the leaves' Taylor
// blocks (g3dpw2local_real_vec, g3drouts.f:1690-1880, after the split),
//   U1[a][kz][ky]  = i^a sum_kx x2l[a][kx] px(kx) L[kz][ky][kx]    per slab
//   U2[b][a][kz]   = i^b sum_ky x2l[b][ky] py(ky) U1[a][kz][ky]    per column
//   lo[c][b][a]    = 2 Re i^c sum_kz x2l[c][kz] pz(kz) U2[b][a][kz] per leaf
// with p(i, k) = exp(+i t_k sh_i).  The mirror nodes make every sum two real
// products of depth n2: with S = L[m] p + L[mb] p* and D = L[m] p - L[mb] p*,
// even orders take tx . S, odd ones i tx . D, tx[a] = (-1)^(a/2) x2l[a].
// Measured against a whole conversion per leaf (B200, one execute): 4e6 blob
// targets, eps 1e-6, 3.33 -> 0.69 ms; 3e5 uniform points, eps 1e-9, delta
// 1e-3, 7.4 -> 0.78 ms (no blocks: evaluated from the columns below).

// x pass (boxes -> slabs) and, with Y, y pass (slabs -> columns).  A warp owns
// four complex columns of the parent, held in registers with their mirror
// sums, and serves the children in turn: four multiply-adds per element turn
// it to the child's phase, 2 U products of KS steps give the child's 16 U
// orders from 16 u0 on.  X: columns (kz, ky) -> U1[(kz, ky)][a]; Y: columns
// (kz, a) -> U2[kz][b][a].  GEN: node halves beyond 4 KS in blocks, with the
// parent read again for every child.
template <int KS, int U, bool Y, bool GEN>
__global__ void __launch_bounds__(128) k_down_xy(KP k, const SepNode* __restrict__ nodes,
                                                 const SepNode* __restrict__ kids, const int* __restrict__ idx,
                                                 int Pm, int u0, const double* __restrict__ Tin,
                                                 double* __restrict__ Tout, const double2* __restrict__ ph) {
  const SepNode N = nodes[blockIdx.x];
  const int ind = blockIdx.z, npw = k.npw, n2 = k.n2, nkb = GEN ? (n2 + 4 * KS - 1) / (4 * KS) : 1;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, r = lane >> 2, c = lane & 3;
  const int ncol = Y ? n2 * N.p : n2 * npw, kst = Y ? N.p : 1;
  const double sg = (r & 1) ? 1.0 : -1.0;
  const double2* src = Y ? reinterpret_cast<const double2*>(Tin + (size_t)N.off * k.nd) + (size_t)ind * N.p * n2 * npw
                         : k.loc + ((size_t)N.off * k.nd + ind) * k.nexp;
  double tx[U][2][KS];
  auto table = [&](int kb) {
#pragma unroll
    for (int u = 0; u < U; u++)
#pragma unroll
      for (int par = 0; par < 2; par++)
#pragma unroll
        for (int s = 0; s < KS; s++) {
          const int a = 2 * (8 * (u0 + u) + r) + par, m = 4 * (KS * kb + s) + c;
          tx[u][par][s] = (a < Pm && m < n2) ? ((a & 2) ? -k.x2l[a * npw + m] : k.x2l[a * npw + m]) : 0.0;
        }
  };
  double os[KS], od[KS], ts[KS], td[KS];
  auto load = [&](const double2* L, int kb) {
#pragma unroll
    for (int s = 0; s < KS; s++) {
      const int m = min(4 * (KS * kb + s) + c, n2 - 1);
      const double2 a = L[(size_t)m * kst], b = L[(size_t)(npw - 1 - m) * kst];
      const double o1 = (r & 1) ? a.y : a.x, o2 = (r & 1) ? b.y : b.x;
      const double t1 = sg * ((r & 1) ? a.x : a.y), t2 = sg * ((r & 1) ? b.x : b.y);
      os[s] = o1 + o2;
      od[s] = o1 - o2;
      ts[s] = t1 + t2;
      td[s] = t1 - t2;
    }
  };
  if (!GEN) table(0);
  const int ntiles = (ncol + 3) / 4;
  for (int nt = blockIdx.y * 4 + warp; nt < ntiles; nt += gridDim.y * 4) {
    const int qb = min(4 * nt + (r >> 1), ncol - 1);  // the column of the lane's operand
    const double2* L = src + (Y ? (size_t)(qb / N.p) * npw * N.p + qb % N.p : (size_t)qb * npw);
    if (!GEN) load(L, 0);
    for (int i = N.beg; i < N.beg + N.cnt; i++) {
      const SepNode K = kids[idx ? idx[i] : i];
      if (!Y && K.p <= 16 * u0) continue;
      double acc[U][4];
#pragma unroll
      for (int u = 0; u < U; u++) acc[u][0] = acc[u][1] = acc[u][2] = acc[u][3] = 0.0;
      for (int kb = 0; kb < nkb; kb++) {
        if (GEN) {
          table(kb);
          load(L, kb);
        }
#pragma unroll
        for (int s = 0; s < KS; s++) {
          const double2 p = __ldg(ph + K.row * npw + min(4 * (KS * kb + s) + c, n2 - 1));
          const double S = fma(p.y, td[s], p.x * os[s]), D = fma(p.y, ts[s], p.x * od[s]);
#pragma unroll
          for (int u = 0; u < U; u++)
            if (u == 0 || 16 * (u0 + u) < K.p) {
              dmma_884(acc[u][0], acc[u][1], tx[u][0][s], S);
              dmma_884(acc[u][2], acc[u][3], tx[u][1][s], D);
            }
        }
      }
      const int q = 4 * nt + c;  // the lane's complex column
      if (q < ncol) {
        double2* o;
        int st;
        if (Y) {
          const int P = N.p, kz = q / P;
          st = P;
          o = reinterpret_cast<double2*>(Tout + (size_t)K.off * k.nd) + ((size_t)ind * n2 + kz) * P * P + (q - kz * P);
        } else {
          st = 1;
          o = reinterpret_cast<double2*>(Tout + (size_t)K.off * k.nd) + ((size_t)ind * n2 * npw + q) * K.p;
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
          const int a = 2 * (8 * (u0 + u) + r);
          if (a < K.p) o[(size_t)a * st] = make_double2(acc[u][0], acc[u][1]);
          if (a + 1 < K.p) o[(size_t)(a + 1) * st] = make_double2(-acc[u][3], acc[u][2]);
        }
      }
    }
  }
}

// z pass: a column's U2 to its leaves' Taylor blocks, rows of E = P rounded up
// to even doubles (the padding zero), orders P <= 32 (16 U).  A warp owns
// eight (b, a) and keeps their n2 values in registers for all the leaves.
template <int KS, int U, bool GEN>
__global__ void __launch_bounds__(128) k_down_z(KP k, const SepNode* __restrict__ cols,
                                                const SepLeaf* __restrict__ leaves, int Pn,
                                                const double* __restrict__ Tin, double* __restrict__ lo_all,
                                                const double2* __restrict__ ph) {
  const SepNode C = cols[blockIdx.x];
  const int ind = blockIdx.z, npw = k.npw, n2 = k.n2, P2 = Pn * Pn, E = (Pn + 1) & ~1;
  const int nkb = GEN ? (n2 + 4 * KS - 1) / (4 * KS) : 1;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, r = lane >> 2, c = lane & 3;
  const double2* src = reinterpret_cast<const double2*>(Tin + (size_t)C.off * k.nd) + (size_t)ind * P2 * n2;
  double tx[U][2][KS];
  auto table = [&](int kb) {
#pragma unroll
    for (int u = 0; u < U; u++)
#pragma unroll
      for (int par = 0; par < 2; par++)
#pragma unroll
        for (int s = 0; s < KS; s++) {
          const int a = 2 * (8 * u + r) + par, m = 4 * (KS * kb + s) + c;
          tx[u][par][s] = (a < Pn && m < n2) ? ((a & 2) ? -k.x2l[a * npw + m] : k.x2l[a * npw + m]) : 0.0;
        }
  };
  double2 z[KS];
  auto load = [&](const double2* L, int kb) {
#pragma unroll
    for (int s = 0; s < KS; s++) z[s] = L[(size_t)min(4 * (KS * kb + s) + c, n2 - 1) * P2];
  };
  if (!GEN) table(0);
  const int ntiles = (P2 + 7) / 8;
  for (int nt = blockIdx.y * 4 + warp; nt < ntiles; nt += gridDim.y * 4) {
    const double2* L = src + min(8 * nt + r, P2 - 1);
    if (!GEN) load(L, 0);
    for (int i = C.beg; i < C.beg + C.cnt; i++) {
      const SepLeaf F = leaves[i];
      double acc[U][4];
#pragma unroll
      for (int u = 0; u < U; u++) acc[u][0] = acc[u][1] = acc[u][2] = acc[u][3] = 0.0;
      for (int kb = 0; kb < nkb; kb++) {
        if (GEN) {
          table(kb);
          load(L, kb);
        }
#pragma unroll
        for (int s = 0; s < KS; s++) {
          const double2 p = __ldg(ph + F.row * npw + min(4 * (KS * kb + s) + c, n2 - 1));
          const double re = fma(-z[s].y, p.y, z[s].x * p.x), im = fma(z[s].y, p.x, z[s].x * p.y);
#pragma unroll
          for (int u = 0; u < U; u++) {
            dmma_884(acc[u][0], acc[u][1], tx[u][0][s], re);
            dmma_884(acc[u][2], acc[u][3], tx[u][1][s], im);
          }
        }
      }
      double* out = lo_all + F.off + (size_t)ind * P2 * E;
#pragma unroll
      for (int ii = 0; ii < 2; ii++) {
        const int q = 8 * nt + 2 * c + ii;
        if (q < P2) {
          const int b = q / Pn, a = q - b * Pn;
          const bool pad = a == Pn - 1 && E > Pn;
#pragma unroll
          for (int u = 0; u < U; u++) {
            const int ce = 2 * (8 * u + r);
            double* o = out + ((size_t)ce * Pn + b) * E + a;
            if (ce < Pn) {
              o[0] = 2.0 * acc[u][ii];
              if (pad) o[1] = 0.0;
            }
            if (ce + 1 < Pn) {
              o[Pn * E] = -2.0 * acc[u][2 + ii];
              if (pad) o[Pn * E + 1] = 0.0;
            }
          }
        }
      }
    }
  }
}

// ------------------------------------------------------------ evaluation from a column
// The Taylor block of a leaf costs P^3 n2 multiply-adds and two passes over
// memory, whatever its number of points; a leaf of few points is evaluated
// from its column's U2 instead:
//   pot(x, y, z) = sum_b,a y^b x^a sum_kz Re(Z(kz) U2[kz][b][a]),
//   Z(kz) = 2 pz(kz) sum_{c<P} x2l[c][kz] (i z)^c,
// the same truncated sum with the z contraction taken at the points.  One CTA
// of four warps per chunk of at most 8 MT points: the rows (Re Z, -Im Z) of
// the points (and of their z derivatives: PGH products) in shared memory,
// U2[kz][q = (b, a)] read from global memory straight into the B fragments
// (each element once per chunk), the warps taking the tiles of q in turn, two
// at a time; the lane's sums of W[point][q] x^a y^b (and with the derivative
// powers) are added over the lanes and warps at the end in a fixed order.
// Bound by the tensor pipe (38 to 47%, each product waiting for the last) and
// the operand loads.  Measured: 1e5 uniform
// points, eps 1e-6 (24 points a leaf, order 21), 1.02 ms with blocks and
// Horner -> 0.18 ms; 3e5 points, eps 1e-9, 3.2 -> 1.0 ms (orders 20 and 31);
// gradients of 1e5 points at eps 1e-9, 37.5 -> 0.94 ms.
template <int PGH>
__host__ __device__ constexpr int colev_tiles() { return PGH == 1 ? 4 : PGH == 2 ? 3 : 2; }

struct ColevDims {
  int K, lda, ldx;
  size_t total;  // doubles
  __host__ __device__ ColevDims(int Pn, int n2, int MT, int pgh) {
    K = (2 * n2 + 3) & ~3;
    lda = (K & 15) <= 4 ? (K & ~15) + 4 : (K & ~15) + 20;  // 4 (mod 16): conflict-free A fragments
    ldx = Pn | 1;
    const int rows = 8 * MT, nc = pgh == 1 ? 1 : pgh == 2 ? 4 : 10;
    total = (size_t)pgh * rows * lda + (size_t)2 * pgh * rows * ldx + (size_t)4 * rows * nc + rows;
  }
};

template <int MT, int PGH>
__device__ __forceinline__ void colev_body(const double2* __restrict__ U2, const double* Zs, const double* Xs,
                                           const double* Ys, const ColevDims& Z, int rows, int Pn, int n2,
                                           double (*sum)[ncomp<3, PGH>()]) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, r = lane >> 2, c = lane & 3;
  const int P2 = Pn * Pn, ks = Z.K >> 2, ntp = (P2 + 15) / 16;
  const double* Ud = reinterpret_cast<const double*>(U2) + (c & 1);
#pragma unroll
  for (int i = 0; i < MT; i++)
#pragma unroll
    for (int v = 0; v < ncomp<3, PGH>(); v++) sum[i][v] = 0.0;
  for (int np = warp; np < ntp; np += 4) {
    double acc[2][MT][PGH][2];
#pragma unroll
    for (int h = 0; h < 2; h++)
#pragma unroll
      for (int i = 0; i < MT; i++)
#pragma unroll
        for (int g = 0; g < PGH; g++) acc[h][i][g][0] = acc[h][i][g][1] = 0.0;
    const double* B0 = Ud + (size_t)2 * min(16 * np + r, P2 - 1);
    const double* B1 = Ud + (size_t)2 * min(16 * np + 8 + r, P2 - 1);
    auto fetch = [&](int s, double (&b)[4][2]) {
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const size_t o = (size_t)2 * min(2 * (s + j) + (c >> 1), n2 - 1) * P2;
        b[j][0] = B0[o];
        b[j][1] = B1[o];
      }
    };
    double bn[4][2];
    fetch(0, bn);
    for (int s = 0; s < ks; s += 4) {
      double b[4][2];
#pragma unroll
      for (int j = 0; j < 4; j++) {
        b[j][0] = bn[j][0];
        b[j][1] = bn[j][1];
      }
      if (s + 4 < ks) fetch(s + 4, bn);
#pragma unroll
      for (int j = 0; j < 4; j++)
        if (s + j < ks) {
#pragma unroll
          for (int i = 0; i < MT; i++)
#pragma unroll
            for (int g = 0; g < PGH; g++) {
              const double a = Zs[((size_t)g * rows + 8 * i + r) * Z.lda + 4 * (s + j) + c];
              dmma_884(acc[0][i][g][0], acc[0][i][g][1], a, b[j][0]);
              dmma_884(acc[1][i][g][0], acc[1][i][g][1], a, b[j][1]);
            }
        }
    }
#pragma unroll
    for (int h = 0; h < 2; h++)
#pragma unroll
      for (int e = 0; e < 2; e++) {
        const int q = 16 * np + 8 * h + 2 * c + e;
        if (q < P2) {
          const int bq = q / Pn, aq = q - bq * Pn;
#pragma unroll
          for (int i = 0; i < MT; i++) {
            const int xo = (8 * i + r) * Z.ldx + aq, yo = (8 * i + r) * Z.ldx + bq, sz = rows * Z.ldx;
            const double x0 = Xs[xo], y0 = Ys[yo], xy = x0 * y0;
            const double w0 = acc[h][i][0][e];
            sum[i][0] = fma(w0, xy, sum[i][0]);
            if constexpr (PGH >= 2) {
              const double x1 = Xs[sz + xo], y1 = Ys[sz + yo], w1 = acc[h][i][1][e];
              sum[i][1] = fma(w0, x1 * y0, sum[i][1]);
              sum[i][2] = fma(w0, x0 * y1, sum[i][2]);
              sum[i][3] = fma(w1, xy, sum[i][3]);
              if constexpr (PGH >= 3) {
                const double x2 = Xs[2 * sz + xo], y2 = Ys[2 * sz + yo], w2 = acc[h][i][2][e];
                sum[i][4] = fma(w0, x2 * y0, sum[i][4]);
                sum[i][5] = fma(w0, x0 * y2, sum[i][5]);
                sum[i][6] = fma(w2, xy, sum[i][6]);
                sum[i][7] = fma(w0, x1 * y1, sum[i][7]);
                sum[i][8] = fma(w1, x1 * y0, sum[i][8]);
                sum[i][9] = fma(w1, x0 * y1, sum[i][9]);
              }
            }
          }
        }
      }
  }
}

template <int PGH>
__global__ void __launch_bounds__(128) k_eval3d_col(KP k, const ColTask* __restrict__ tasks,
                                                    const double* __restrict__ Tin,
                                                    const double2* __restrict__ ph) {
  constexpr int MT = colev_tiles<PGH>(), ROWS = 8 * MT, NC = ncomp<3, PGH>();
  const ColTask T = tasks[blockIdx.x];
  const int ind = blockIdx.y, Pn = T.p, P2 = Pn * Pn, npw = k.npw, n2 = k.n2, tid = threadIdx.x;
  const ColevDims Z(Pn, n2, MT, PGH);
  extern __shared__ double sm[];
  double* Zs = sm;                                  // [PGH][ROWS][lda]
  double* Xs = Zs + (size_t)PGH * ROWS * Z.lda;     // [PGH][ROWS][ldx]: x^a and its derivatives
  double* Ys = Xs + (size_t)PGH * ROWS * Z.ldx;
  double* red = Ys + (size_t)PGH * ROWS * Z.ldx;    // [4][ROWS][NC]
  double* zc = red + (size_t)4 * ROWS * NC;         // [ROWS]
  const double* pts = T.set ? k.trg : k.src;
  if (tid < ROWS) {
    const int i = T.i0 + min(tid, T.n - 1);
    double v[3];
#pragma unroll
    for (int d = 0; d < 3; d++) v[d] = (pts[(size_t)3 * i + d] - k.centers[3 * T.box + d]) * k.dsq;
    zc[tid] = v[2];
#pragma unroll
    for (int d = 0; d < 2; d++) {
      double* X = (d ? Ys : Xs) + tid * Z.ldx;
      double p0 = 1.0, p1 = 0.0, p2 = 0.0;  // x^a, a x^(a-1), a (a-1) x^(a-2)
      for (int a = 0; a < Pn; a++) {
        X[a] = p0;
        if (PGH >= 2) X[ROWS * Z.ldx + a] = p1;
        if (PGH >= 3) X[2 * ROWS * Z.ldx + a] = p2;
        if (PGH >= 3) p2 = fma(p2, v[d], 2.0 * p1);
        if (PGH >= 2) p1 = fma(p1, v[d], p0);
        p0 *= v[d];
      }
    }
  }
  __syncthreads();
  // Z rows: Horner in i z with the derivative chains s' <- s' (i z) + i s
  for (int e = tid; e < ROWS * (Z.K >> 1); e += 128) {
    const int pt = e / (Z.K >> 1), kz = e - pt * (Z.K >> 1);
    double2 f[3];
    f[0] = f[1] = f[2] = make_double2(0.0, 0.0);
    if (kz < n2 && pt < T.n) {
      const double u = zc[pt];
      double2 s0 = make_double2(0.0, 0.0), s1 = s0, s2 = s0;
      for (int j = Pn - 1; j >= 0; j--) {
        if (PGH >= 3) s2 = make_double2(fma(-s2.y, u, -2.0 * s1.y), fma(s2.x, u, 2.0 * s1.x));
        if (PGH >= 2) s1 = make_double2(fma(-s1.y, u, -s0.y), fma(s1.x, u, s0.x));
        s0 = make_double2(fma(-s0.y, u, __ldg(k.x2l + j * npw + kz)), s0.x * u);
      }
      const double2 p = __ldg(ph + T.row * npw + kz), p2 = make_double2(2.0 * p.x, 2.0 * p.y);
      f[0] = cmul(s0, p2);
      if (PGH >= 2) f[1] = cmul(s1, p2);
      if (PGH >= 3) f[2] = cmul(s2, p2);
    }
#pragma unroll
    for (int g = 0; g < PGH; g++) {
      double* a = Zs + ((size_t)g * ROWS + pt) * Z.lda + 2 * kz;
      a[0] = f[g].x;
      a[1] = -f[g].y;
    }
  }
  __syncthreads();
  const double2* U2 = reinterpret_cast<const double2*>(Tin + (size_t)T.off * k.nd) + (size_t)ind * P2 * n2;
  double sum[MT][NC];
  const int nmt = (T.n + 7) / 8;
#pragma unroll
  for (int i = 0; i < MT; i++)
#pragma unroll
    for (int v = 0; v < NC; v++) sum[i][v] = 0.0;
  if (nmt == 1) colev_body<1, PGH>(U2, Zs, Xs, Ys, Z, ROWS, Pn, n2, sum);
  else if (nmt == 2) colev_body<2, PGH>(U2, Zs, Xs, Ys, Z, ROWS, Pn, n2, sum);
  else if constexpr (MT >= 3) {
    if (MT == 3 || nmt == 3) colev_body<3, PGH>(U2, Zs, Xs, Ys, Z, ROWS, Pn, n2, sum);
    else colev_body<MT, PGH>(U2, Zs, Xs, Ys, Z, ROWS, Pn, n2, sum);
  }
  const int lane = tid & 31, warp = tid >> 5, r = lane >> 2, c = lane & 3;
#pragma unroll
  for (int i = 0; i < MT; i++)
#pragma unroll
    for (int v = 0; v < NC; v++) {
      double a = sum[i][v];
      a += __shfl_xor_sync(FULL_MASK, a, 1);
      a += __shfl_xor_sync(FULL_MASK, a, 2);
      if (c == 0) red[((size_t)warp * ROWS + 8 * i + r) * NC + v] = a;
    }
  __syncthreads();
  double* out = T.set ? k.pottarg : k.pot;
  const int nc = T.set ? k.nc_t : k.nc_s;
  for (int e = tid; e < T.n * NC; e += 128) {
    const int pt = e / NC, v = e - pt * NC;
    if (v >= nc) continue;
    double a = 0.0;
#pragma unroll
    for (int w = 0; w < 4; w++) a += red[((size_t)w * ROWS + pt) * NC + v];
    const double sc = v == 0 ? 1.0 : v < 4 ? k.dsq : k.dsq * k.dsq;
    out[((size_t)(T.i0 + pt) * nc + v) * k.nd + ind] += a * sc;
  }
}

// CTAs per node so that the launch fills the SMs several times over
int split_for(int nodes, int nd, int tiles, int sms) {
  const long long have = (long long)nodes * nd, want = (long long)sms * 12;
  const int most = (tiles + 3) / 4;
  return (int)std::max<long long>(1, std::min<long long>(most, (want + have - 1) / std::max(1LL, have)));
}

}  // namespace

#define CK(x)                               \
  do {                                      \
    cudaError_t e_ = (x);                   \
    if (e_ != cudaSuccess) return e_;       \
  } while (0)

cudaError_t sep_up_3d(const KP& k, const SepDev& S, const double* hbuf, cudaStream_t st, long long& launches) {
  const int n2 = k.n2, tiles = (n2 + 7) / 8;
  int pmax = 1;
  for (const SepGroup& G : S.groups) {
    const int Pn = G.p + 1, ks = (Pn + 7) / 8;
    if (ks > 4) return cudaErrorNotSupported;
    pmax = std::max(pmax, Pn);
    const int ncol = G.cend - G.cbeg, nslab = G.send - G.sbeg;
    const dim3 gz(ncol, split_for(ncol, k.nd, (Pn * Pn + 7) / 8, S.sms), k.nd);
    const dim3 gy(nslab, split_for(nslab, k.nd, (Pn * n2 + 3) / 4, S.sms), k.nd);
    for (int t0 = 0; t0 < tiles; t0 += 4) {
      switch (4 * (ks - 1) + std::min(4, tiles - t0) - 1) {
#define UP_CASE(KS_, MT_)                                                                                       \
  case 4 * (KS_ - 1) + MT_ - 1:                                                                                 \
    k_up_z<KS_, MT_><<<gz, 128, 0, st>>>(k, S.cols + G.cbeg, S.leaves, Pn, t0, hbuf, S.t1, S.ph);               \
    break;
#define UP_CASES                                                                                                \
  UP_CASE(1, 1) UP_CASE(1, 2) UP_CASE(1, 3) UP_CASE(1, 4) UP_CASE(2, 1) UP_CASE(2, 2) UP_CASE(2, 3) UP_CASE(2, 4) \
  UP_CASE(3, 1) UP_CASE(3, 2) UP_CASE(3, 3) UP_CASE(3, 4) UP_CASE(4, 1) UP_CASE(4, 2) UP_CASE(4, 3) UP_CASE(4, 4)
        UP_CASES
#undef UP_CASE
      }
      launches++;
    }
    for (int t0 = 0; t0 < tiles; t0 += 4) {
      switch (4 * (ks - 1) + std::min(4, tiles - t0) - 1) {
#define UP_CASE(KS_, MT_)                                                                                       \
  case 4 * (KS_ - 1) + MT_ - 1:                                                                                 \
    k_up_xy<KS_, MT_, true><<<gy, 128, 0, st>>>(k, S.slabs + G.sbeg, S.cols, nullptr, Pn, t0, S.t1, S.t2, S.ph); \
    break;
        UP_CASES
#undef UP_CASE
      }
      launches++;
    }
  }
  if (S.nboxes > 0) {
    const dim3 gx(S.nboxes, split_for(S.nboxes, k.nd, (n2 * k.npw + 3) / 4, S.sms), k.nd);
    for (int t0 = 0; t0 < tiles; t0 += 4) {
      switch (4 * ((pmax + 7) / 8 - 1) + std::min(4, tiles - t0) - 1) {
#define UP_CASE(KS_, MT_)                                                                                       \
  case 4 * (KS_ - 1) + MT_ - 1:                                                                                 \
    k_up_xy<KS_, MT_, false><<<gx, 128, 0, st>>>(k, S.boxes, S.slabs, S.box_kids, pmax, t0, S.t2, nullptr, S.ph); \
    break;
        UP_CASES
#undef UP_CASE
      }
      launches++;
    }
  }
  return cudaGetLastError();
}

cudaError_t sep_down_3d(const KP& k, const SepDev& S, double* lo, cudaStream_t st, long long& launches) {
  const int n2 = k.n2, ksm = (n2 + 3) / 4;
  int pmax = 0;
  for (const SepGroup& G : S.groups) pmax = std::max(pmax, G.p + 1);
  if (S.nboxes <= 0 || pmax == 0) return cudaSuccess;
  auto cases = [&](int U, auto launch) {
    const int v = ksm > 8 ? 0 : ksm;
    switch (2 * v + U - 1) {
#define DOWN_CASE(N)                                                                            \
  case 2 * N: launch(std::integral_constant<int, N>(), std::integral_constant<int, 1>(), std::false_type()); break; \
  case 2 * N + 1: launch(std::integral_constant<int, N>(), std::integral_constant<int, 2>(), std::false_type()); break;
      DOWN_CASE(1) DOWN_CASE(2) DOWN_CASE(3) DOWN_CASE(4) DOWN_CASE(5) DOWN_CASE(6) DOWN_CASE(7) DOWN_CASE(8)
#undef DOWN_CASE
      default: launch(std::integral_constant<int, 8>(), std::integral_constant<int, 2>(), std::true_type()); break;
    }
    launches++;
  };
  const dim3 gx(S.nboxes, split_for(S.nboxes, k.nd, (n2 * k.npw + 3) / 4, S.sms), k.nd);
  for (int u0 = 0; 16 * u0 < pmax; u0 += 2)
    cases(pmax - 16 * u0 <= 16 ? 1 : 2, [&](auto N, auto U, auto G) {
      k_down_xy<decltype(N)::value, decltype(U)::value, false, decltype(G)::value>
          <<<gx, 128, 0, st>>>(k, S.boxes, S.slabs, S.box_kids, pmax, u0, nullptr, S.t2, S.ph);
    });
  for (const SepGroup& G : S.groups) {
    const int Pn = G.p + 1, nslab = G.send - G.sbeg, ncol = G.cend - G.cbeg;
    const dim3 gy(nslab, split_for(nslab, k.nd, (n2 * Pn + 3) / 4, S.sms), k.nd);
    for (int u0 = 0; 16 * u0 < Pn; u0 += 2)
      cases(Pn - 16 * u0 <= 16 ? 1 : 2, [&](auto N, auto U, auto F) {
        k_down_xy<decltype(N)::value, decltype(U)::value, true, decltype(F)::value>
            <<<gy, 128, 0, st>>>(k, S.slabs + G.sbeg, S.cols, nullptr, Pn, u0, S.t2, S.t1, S.ph);
      });
    if (!G.blocks) continue;  // evaluated from the columns
    if (Pn > 32) return cudaErrorNotSupported;
    const dim3 gz(ncol, split_for(ncol, k.nd, (Pn * Pn + 7) / 8, S.sms), k.nd);
    cases(Pn <= 16 ? 1 : 2, [&](auto N, auto U, auto F) {
      k_down_z<decltype(N)::value, decltype(U)::value, decltype(F)::value>
          <<<gz, 128, 0, st>>>(k, S.cols + G.cbeg, S.leaves, Pn, S.t1, lo, S.ph);
    });
  }
  return cudaGetLastError();
}

int sep_col_points(int pgh) { return 8 * (pgh <= 1 ? colev_tiles<1>() : pgh == 2 ? colev_tiles<2>() : colev_tiles<3>()); }

cudaError_t sep_eval_cols(const KP& k, const SepDev& S, const ColTask* tasks, int ntask, int Pn, int pgh,
                          cudaStream_t st) {
  if (ntask <= 0) return cudaSuccess;
  const dim3 g(ntask, k.nd);
  const size_t sh = ColevDims(Pn, k.n2, sep_col_points(pgh) / 8, pgh).total * 8;
  if (sh > 227 * 1024) return cudaErrorNotSupported;
#define COLEV_CASE(PG)                                            \
  {                                                               \
    CK(smem_limit(k_eval3d_col<PG>));                             \
    k_eval3d_col<PG><<<g, 128, sh, st>>>(k, tasks, S.t1, S.ph);   \
  }
  if (pgh <= 1) COLEV_CASE(1)
  else if (pgh == 2) COLEV_CASE(2)
  else COLEV_CASE(3)
#undef COLEV_CASE
  return cudaGetLastError();
}

}  // namespace fgtb
