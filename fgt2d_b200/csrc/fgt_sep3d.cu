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
// What bounds the kernels: the FP64 tensor pipe (mma.m8n8k4, 16 cycles per
// SM sub-partition) in the z pass, memory in the others; every operand is
// read once from global memory straight into the fragment that needs it, so
// there is no shared memory and the warps are independent.  Measured against
// a whole transform per leaf and level-by-level merges (B200, transforms and
// merges of one execute): 4e6 blob sources, eps 1e-6, 2.75 -> 0.85 ms; 3e5
// uniform points, eps 1e-9, delta 1e-3, 4.95 -> 1.38 ms; eps 1e-12, delta
// 1e-2, 24.2 -> 0.42 ms (orders whose whole transform did not fit in shared
// memory ran on the scalar pipes).
#include <algorithm>
#include <cmath>
#include <cstdint>

#include "fgt_kcommon.cuh"
#include "fgt_sep3d.hpp"

namespace fgtb {

// ------------------------------------------------------------ lists
void sep_sort(const Tree& t, const std::vector<int>& root_box, std::vector<SepItem>& items) {
  const int n = (int)items.size();
#pragma omp parallel for schedule(static) if (n > 4096)
  for (int i = 0; i < n; i++) {
    SepItem& s = items[i];
    const int a = root_box[s.root], l = t.level[s.box];
    s.d = l - t.level[a];
    for (int q = 0; q < 3; q++)
      s.x[q] = (int)std::lround((t.c(s.box, q) - t.c(a, q)) / t.boxsize[l] + 0.5 * ((1 << s.d) - 1));
  }
  int dmax = 0, pmax = 0;
  for (const SepItem& s : items) {
    dmax = std::max(dmax, s.d);
    pmax = std::max(pmax, s.p);
  }
  // one key per item, (p, d, root, x, y, z) from the top, sorted by digits of
  // 11 bits; the items move once
  auto width = [](unsigned long long v) {
    int w = 0;
    while (v >> w) w++;
    return w;
  };
  const int wr = width(root_box.size()), wd = width(dmax), wp = width(pmax), bits = 3 * dmax + wr + wd + wp;
  if (bits > 64) {  // a tree deeper than the keys hold
    std::stable_sort(items.begin(), items.end(), [](const SepItem& a, const SepItem& b) {
      if (a.p != b.p) return a.p < b.p;
      if (a.d != b.d) return a.d < b.d;
      if (a.root != b.root) return a.root < b.root;
      return std::lexicographical_compare(a.x, a.x + 3, b.x, b.x + 3);
    });
    return;
  }
  struct Key {
    uint64_t k;
    int i;
  };
  std::vector<Key> key(n), tmp(n);
  for (int i = 0; i < n; i++) {
    const SepItem& s = items[i];
    uint64_t k = ((uint64_t)s.p << wd | (uint64_t)s.d) << wr | (uint64_t)s.root;
    for (int q = 0; q < 3; q++) k = k << dmax | (uint64_t)s.x[q];
    key[i] = {k, i};
  }
  for (int b = 0; b < bits; b += 11) {
    int cnt[2049] = {0};
    for (const Key& e : key) cnt[((e.k >> b) & 2047) + 1]++;
    for (int i = 0; i < 2048; i++) cnt[i + 1] += cnt[i];
    for (const Key& e : key) tmp[cnt[(e.k >> b) & 2047]++] = e;
    key.swap(tmp);
  }
  std::vector<SepItem> out(n);
  for (int i = 0; i < n; i++) out[i] = items[key[i].i];
  items.swap(out);
}

void sep_lists(const std::vector<SepItem>& items, const std::vector<int>& slot, int npw, SepLists& S) {
  const int n = (int)items.size(), n2 = npw / 2, nroot = (int)slot.size();
  S = SepLists();
  S.leaves.reserve(n);
  auto row = [](const SepItem& s, int q) { return (1 << s.d) - 1 + s.x[q]; };
  std::vector<int> slab_root;
  for (int i = 0; i < n; i++) {
    const SepItem& s = items[i];
    const long long Pn = s.p + 1;
    const SepItem* o = i ? &items[i - 1] : nullptr;
    const bool group = !o || o->p != s.p;
    const bool slab = group || o->d != s.d || o->root != s.root || o->x[0] != s.x[0];
    if (group) S.groups.push_back({s.p, (int)S.cols.size(), 0, (int)S.slabs.size(), 0});
    if (slab) {
      S.slabs.push_back({(long long)S.t2, (int)S.cols.size(), 0, row(s, 0), (int)Pn});
      S.t2 += (size_t)(Pn * n2 * npw * 2);
      slab_root.push_back(s.root);
    }
    if (slab || o->x[1] != s.x[1]) {
      S.cols.push_back({(long long)S.t1, i, 0, row(s, 1), (int)Pn});
      S.t1 += (size_t)(Pn * Pn * n2 * 2);
      S.slabs.back().cnt++;
    }
    S.cols.back().cnt++;
    S.leaves.push_back({s.off, row(s, 2), s.n});
    S.groups.back().cend = (int)S.cols.size();
    S.groups.back().send = (int)S.slabs.size();
  }
  std::vector<int> cnt(nroot + 1, 0);
  for (int r : slab_root) cnt[r + 1]++;
  for (int r = 0; r < nroot; r++) {
    S.boxes.push_back({(long long)slot[r], cnt[r], cnt[r + 1], 0, 0});
    cnt[r + 1] += cnt[r];
  }
  S.box_slabs.resize(slab_root.size());
  for (size_t i = 0; i < slab_root.size(); i++) S.box_slabs[cnt[slab_root[i]]++] = (int)i;
}

void sep_phases(const HostPlan& H, int dmax, double bs0, std::vector<double>& ph) {
  const int npw = H.P.npw;
  ph.resize((size_t)2 * npw * ((size_t(2) << dmax) - 1));
  for (int d = 0; d <= dmax; d++)
    for (int i = 0; i < (1 << d); i++) {
      const double sh = (i + 0.5 - 0.5 * (1 << d)) * std::ldexp(bs0, -d) * H.P.dsq;
      double* r = ph.data() + (size_t)2 * npw * ((1 << d) - 1 + i);
      for (int m = 0; m < npw; m++) {
        r[2 * m] = std::cos(H.ts[m] * sh);
        r[2 * m + 1] = std::sin(H.ts[m] * sh);
      }
    }
}

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
      for (int ch = 1; ch < L.n; ch++) {  // further partial blocks, in chunk order
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

// A leaf's expansion times the phases from its centre to the box's, summed
// over the leaves of a box; one coefficient per thread (memory-bound).
__global__ void __launch_bounds__(256) k_up_add(KP k, const double2* __restrict__ src,
                                                const double2* __restrict__ ph,
                                                const MergeGroup* __restrict__ groups,
                                                const SepShift* __restrict__ shifts) {
  const MergeGroup G = groups[blockIdx.x];
  const int ind = blockIdx.z, npw = k.npw, e = blockIdx.y * blockDim.x + threadIdx.x;
  if (e >= k.nexp) return;
  const int kx = e % npw, ky = (e / npw) % npw, kz = e / (npw * npw);
  double2* dst = k.mp + ((size_t)G.dst * k.nd + ind) * k.nexp + e;
  double2 a = *dst;
  for (int t = G.beg; t < G.beg + G.cnt; t++) {
    const SepShift S = shifts[t];
    const double2 f = cmul(ph[S.row[0] * npw + kx], cmul(ph[S.row[1] * npw + ky], ph[S.row[2] * npw + kz]));
    a = cfmac(src[((size_t)S.src * k.nd + ind) * k.nexp + e], f, a);
  }
  *dst = a;
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

cudaError_t sep_add(const KP& k, const double2* src, const double2* ph, const MergeGroup* groups, int ngroups,
                    const SepShift* shifts, cudaStream_t st) {
  if (ngroups <= 0) return cudaSuccess;
  k_up_add<<<dim3(ngroups, (k.nexp + 255) / 256, k.nd), 256, 0, st>>>(k, src, ph, groups, shifts);
  return cudaGetLastError();
}

cudaError_t sep_up(const KP& k, const SepDev& S, const double* hbuf, cudaStream_t st, long long& launches) {
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
    k_up_xy<KS_, MT_, false><<<gx, 128, 0, st>>>(k, S.boxes, S.slabs, S.box_slabs, pmax, t0, S.t2, nullptr, S.ph); \
    break;
        UP_CASES
#undef UP_CASE
      }
      launches++;
    }
  }
  return cudaGetLastError();
}

}  // namespace fgtb
