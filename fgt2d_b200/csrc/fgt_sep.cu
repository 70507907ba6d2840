// Separable transforms between the leaves and the cut-level boxes: the lists of
// both dimensions and the 2D kernels (3D: fgt_sep3d.cu, which explains the
// sums).  2D has one level less: on the way up the x transform runs once per
// leaf and the y transform once per row of leaves of equal y (and depth),
//   PW_A(ky, kx) = sum_iy py(iy, ky) sum_jy i^jy hx[jy][ky]
//                  sum_ix px(ix, kx) sum_jx i^jx hx[jx][kx] H_b[jx][jy],
// on the way down the other way round, and no expansion below the cut level is
// formed.  The nodes come in mirror pairs, so every complex sum is two real
// products over half the nodes on the FP64 tensor cores (mma.m8n8k4); the
// operands are read once from global memory straight into the fragments, the
// warps are independent and take (node, tile) pairs of a launch in turn: rows
// have one to four tiles, so a CTA per row left most warps idle.
// Bound by latency and the intermediate's two passes over memory (it stays in
// L2).  Measured against a transform per leaf, merges level by level and the
// split fused into a conversion per leaf (B200, one execute, up and down): 3e5
// sources and 1e5 targets with Hessians, eps 1e-9, 221 -> 113 us; dipoles of two
// densities, 2e5 sources, 423 -> 209; 1e5 + 1e5 points, 73 -> 61.
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <type_traits>

#include "fgt_kcommon.cuh"
#include "fgt_sep.hpp"

namespace fgtb {

// ------------------------------------------------------------ lists
std::vector<int> sep_rank(const std::vector<int>& order) {
  std::vector<int> by(order.size()), rank(order.size());
  for (size_t d = 0; d < by.size(); d++) by[d] = (int)d;
  std::stable_sort(by.begin(), by.end(), [&](int a, int b) { return order[a] < order[b]; });
  for (size_t i = 0; i < by.size(); i++) rank[by[i]] = (int)i;
  return rank;
}

void sep_order(const Tree& t, int lroot, const std::vector<int>& boxes, const std::vector<int>& rank,
               uvector<SepItem>& items, SepRows& rows) {
  const int n = (int)boxes.size(), a0 = t.lfirst[lroot], dmax = (int)rank.size() - 1, dim = t.dim;
  const bool dense = dmax <= SEP_DENSE;
  auto root_of = [&](int b) {
    while (t.level[b] > lroot) b = t.parent[b];
    return b;
  };
  const double bs0 = t.boxsize[lroot];
  auto offset = [&](int b, int a, int d) { return (t.c(b, d) - t.c(a, d)) / bs0; };
  rows.base.assign(dmax + 1, 0);
  rows.at.clear();
  if (dense) {
    for (int d = 0; d <= dmax; d++) {
      rows.base[d] = (1 << d) - 1;
      for (int i = 0; i < (1 << d); i++) rows.at.push_back((i + 0.5) / (1 << d) - 0.5);
    }
  } else {
    std::vector<std::vector<double>> at(dmax + 1);
    for (int b : boxes) {
      const int a = root_of(b);
      for (int d = 0; d < dim; d++) at[t.level[b] - lroot].push_back(offset(b, a, d));
    }
    for (int d = 0; d <= dmax; d++) {
      std::sort(at[d].begin(), at[d].end());
      at[d].erase(std::unique(at[d].begin(), at[d].end()), at[d].end());
      rows.base[d] = (int)rows.at.size();
      rows.at.insert(rows.at.end(), at[d].begin(), at[d].end());
    }
  }
  // the place of a box: its row less the first of its depth
  auto place = [&](int b, int a, int dep, int d) {
    const double v = offset(b, a, d);
    if (dense) return std::max(0, std::min((1 << dep) - 1, (int)std::lround((v + 0.5) * (1 << dep) - 0.5)));
    const auto first = rows.at.begin() + rows.base[dep];
    return (int)(std::lower_bound(first, dep < dmax ? rows.at.begin() + rows.base[dep + 1] : rows.at.end(), v) - first);
  };
  auto width = [](unsigned long long v) {
    int w = 0;
    while (v >> w) w++;
    return w;
  };
  // one key per item, (rank, root, x, y, z, number), sorted by digits of at
  // most 12 bits; the items are written once, in order
  const int wn = width(n), wr = width(t.llast[lroot] - a0), wd = width(dmax);
  const int wx = dense ? dmax : width(rows.at.size());
  const bool packed = dim * wx + wr + wd + wn <= 64;
  uvector<SepItem> raw(n);
  uvector<uint64_t> key(packed ? n : 0), tmp(packed ? n : 0);
#pragma omp parallel for schedule(static) if (n > 2048)
  for (int i = 0; i < n; i++) {
    SepItem& s = raw[i];
    s.box = boxes[i];
    s.num = i;
    const int a = root_of(s.box);
    s.root = a - a0;
    s.d = t.level[s.box] - lroot;
    s.x[2] = 0;
    for (int q = 0; q < dim; q++) {
      const int e = dim == 2 ? 1 - q : q;  // 2D: y, x
      s.x[q] = place(s.box, a, s.d, e);
    }
    if (packed) {
      uint64_t k = (uint64_t)rank[s.d] << wr | (uint64_t)s.root;
      for (int q = 0; q < dim; q++) k = k << wx | (uint64_t)s.x[q];
      key[i] = k << wn | (uint64_t)i;
    }
  }
  if (!packed) {  // more roots and places than the keys hold
    std::stable_sort(raw.begin(), raw.end(), [&](const SepItem& a, const SepItem& b) {
      if (a.d != b.d) return rank[a.d] < rank[b.d];
      if (a.root != b.root) return a.root < b.root;
      return std::lexicographical_compare(a.x, a.x + 3, b.x, b.x + 3);
    });
    items.swap(raw);
    return;
  }
  const int bits = dim * wx + wr + wd, digit = (bits + (bits + 11) / 12 - 1) / std::max(1, (bits + 11) / 12);
  for (int b = wn; b < wn + bits; b += digit) {
    int cnt[4097] = {0};
    const uint64_t dm = (uint64_t(1) << digit) - 1;
    for (uint64_t k : key) cnt[((k >> b) & dm) + 1]++;
    for (int i = 0; i < (int)dm; i++) cnt[i + 1] += cnt[i];
    for (uint64_t k : key) tmp[cnt[(k >> b) & dm]++] = k;
    key.swap(tmp);
  }
  items.resize(n);
  const uint64_t mask = (uint64_t(1) << wn) - 1;
#pragma omp parallel for schedule(static) if (n > 2048)
  for (int i = 0; i < n; i++) items[i] = raw[key[i] & mask];
}

void sep_lists(int dim, const uvector<SepItem>& items, const SepRows& rows, std::vector<SepLeaf>& leaf,
               const std::vector<int>& order, const int* slot, int also, int npw, SepLists& out) {
  const int n = (int)items.size(), n2 = npw / 2;
  SepLists S;  // this thread's until it is whole
  S.leaves.swap(leaf);
  S.cols.resize(n);
  if (dim == 3) {
    S.slabs.resize(n);
  } else {
    S.col_slot.resize(n);
    S.leaf_col.resize(n);
  }
  // the slabs (2D: columns) by root: ascending within a depth, then merged
  typedef std::pair<int, int> RootKid;
  std::vector<RootKid> kids(n);
  std::vector<size_t> runs;
  int nc = 0, nk = 0, ns = 0;
  size_t t1 = 0, t2 = 0;
  for (int i = 0; i < n;) {
    // the items of one depth
    const int d = items[i].d, p = order[d], row0 = rows.base[d];
    const long long Pn = p + 1;
    if (S.groups.empty() || S.groups.back().p != p) S.groups.push_back({p, nc, nc, ns, ns, i, i});
    runs.push_back(nk);
    const SepItem* o = nullptr;
    for (; i < n && items[i].d == d; o = &items[i++]) {
      const SepItem& s = items[i];
      const bool slab = !o || o->root != s.root || o->x[0] != s.x[0];
      if (slab) {
        kids[nk] = {s.root, nk};
        nk++;
      }
      if (dim == 3) {
        if (slab) {
          S.slabs[ns++] = {(long long)t2, nc, 0, row0 + s.x[0], (int)Pn};
          t2 += (size_t)(Pn * n2 * npw * 2);
        }
        if (slab || o->x[1] != s.x[1]) {
          S.cols[nc++] = {(long long)t1, i, 0, row0 + s.x[1], (int)Pn};
          t1 += (size_t)(Pn * Pn * n2 * 2);
          S.slabs[ns - 1].cnt++;
        }
        S.leaves[i].row = row0 + s.x[2];
      } else {
        if (slab) {
          S.col_slot[nc] = slot[s.root];
          S.cols[nc++] = {(long long)t1, i, 0, row0 + s.x[0], (int)Pn};
          t1 += (size_t)(Pn * n2 * 2);
        }
        S.leaf_col[i] = nc - 1;
        S.leaves[i].row = row0 + s.x[1];
      }
      S.cols[nc - 1].cnt++;
    }
    SepGroup& G = S.groups.back();
    G.lend = i;
    G.cend = nc;
    G.send = ns;
  }
  S.cols.resize(nc);
  if (dim == 2) S.col_slot.resize(nc);
  if (dim == 3) S.slabs.resize(ns);
  S.t1 = t1;
  S.t2 = t2;
  kids.resize(nk);
  for (size_t r = 1; r < runs.size(); r++)
    std::inplace_merge(kids.begin(), kids.begin() + runs[r],
                       r + 1 < runs.size() ? kids.begin() + runs[r + 1] : kids.end());
  S.box_kids.resize(kids.size());
  for (size_t i = 0; i < kids.size(); i++) {
    if (i == 0 || kids[i].first != kids[i - 1].first) S.boxes.push_back({(long long)slot[kids[i].first], (int)i, 0, 0, 0});
    S.boxes.back().cnt++;
    S.box_kids[i] = kids[i].second;
  }
  if (also >= 0 && kids.empty()) S.boxes.push_back({(long long)slot[also], 0, 0, 0, 0});
  out = std::move(S);
}

double sep_flops(int dim, bool up, const SepLists& S, int npw) {
  const double n2 = npw / 2, w = npw, turn = up ? 8.0 : 16.0;
  double f = 0.0;
  for (const SepGroup& G : S.groups) {
    const double P = G.p + 1, leaves = G.lend - G.lbeg, cols = G.cend - G.cbeg, slabs = G.send - G.sbeg;
    if (dim == 2) {
      f += leaves * (2 * P * P * n2 + 8 * P * n2) + cols * (4 * P * n2 * n2 + turn * n2 * n2);
    } else {
      if (G.blocks) f += leaves * (2 * P * P * P * n2 + 8 * P * P * n2);
      f += cols * (4 * P * P * n2 * n2 + turn * P * n2 * n2) + slabs * (4 * P * n2 * n2 * w + turn * n2 * n2 * w);
    }
  }
  return f;
}

void sep_phases(const HostPlan& H, const SepRows& rows, double bs0, std::vector<double>& ph) {
  const int npw = H.P.npw;
  ph.resize((size_t)2 * npw * rows.at.size());
  for (size_t i = 0; i < rows.at.size(); i++) {
    const double sh = rows.at[i] * bs0 * H.P.dsq;
    double* r = ph.data() + (size_t)2 * npw * i;
    for (int m = 0; m < npw; m++) {
      r[2 * m] = std::cos(H.ts[m] * sh);
      r[2 * m + 1] = std::sin(H.ts[m] * sh);
    }
  }
}

namespace {

// The (node, tile) pairs of a launch over its warps.
struct Tiles {
  long long at, end, step;
  __device__ __forceinline__ Tiles(int nnode, int tiles) {
    at = (long long)blockIdx.x * 4 + (threadIdx.x >> 5);
    end = (long long)nnode * tiles;
    step = (long long)gridDim.x * 4;
  }
};
dim3 tiles_grid(int nnode, int tiles, int nd, int sms) {
  const long long items = (long long)nnode * tiles, most = std::max<long long>(1, (long long)sms * 16 / nd);
  return dim3((unsigned)std::max<long long>(1, std::min((items + 3) / 4, most)), 1, nd);
}

// ------------------------------------------------------------ upward
// x pass: T1[jy][kx] = sum over the row's leaves of conj(p(kx)) (E + i O), E/O
// = sum over even / odd jx of H[jx][jy] hs[jx][kx] with the signed table
// hs[j] = (-1)^(j/2) hx[j], kx in the positive node half.  A warp owns eight
// powers jy of a row and eight nodes, keeps its part of the table in registers
// and the sum over the leaves in its accumulators.  GEN: orders beyond 8 KS,
// in blocks of powers with the table read again.
template <int KS, bool GEN>
__global__ void __launch_bounds__(128) k_up2d_x(KP k, const SepNode* __restrict__ rows, int nrow,
                                                const SepLeaf* __restrict__ leaves, int Pn,
                                                const double* __restrict__ hx, const double* __restrict__ hbuf,
                                                double* __restrict__ T1, const double2* __restrict__ ph) {
  const int ind = blockIdx.z, npw = k.npw, n2 = k.n2, PP = Pn * Pn;
  const int nkb = GEN ? (Pn + 8 * KS - 1) / (8 * KS) : 1;
  const int lane = threadIdx.x & 31, r = lane >> 2, c = lane & 3;
  const int ntk = (n2 + 7) / 8, tiles = (Pn + 7) / 8 * ntk;
  double hz[2][KS];
  const Tiles work(nrow, tiles);
  for (long long w = work.at; w < work.end; w += work.step) {
    const int row = (int)(w / tiles), tile = (int)(w - (long long)row * tiles), mt = tile / ntk, t0 = tile - mt * ntk;
    auto table = [&](int kb) {
#pragma unroll
      for (int par = 0; par < 2; par++)
#pragma unroll
        for (int s = 0; s < KS; s++) {
          const int j = 8 * (KS * kb + s) + 2 * c + par, kx = 8 * t0 + r;
          const bool ok = j < Pn && kx < n2;
          hz[par][s] = ok ? ((j & 2) ? -hx[j * npw + kx] : hx[j * npw + kx]) : 0.0;
        }
    };
    if (!GEN) table(0);
    const SepNode C = rows[row];
    const int m = 8 * mt + r, mm = min(m, Pn - 1);
    double acc[4] = {0.0, 0.0, 0.0, 0.0};
    SepLeaf Ln = leaves[C.beg];
#pragma unroll 1
    for (int q = C.beg; q < C.beg + C.cnt; q++) {
      const SepLeaf L = Ln;
      if (q + 1 < C.beg + C.cnt) Ln = leaves[q + 1];
      double v[4] = {0.0, 0.0, 0.0, 0.0};
      for (int kb = 0; kb < nkb; kb++) {
        if (GEN) table(kb);
        double a[2][KS];
        const double* H = hbuf + (size_t)L.off * k.nd + (size_t)ind * PP + mm;
#pragma unroll
        for (int s = 0; s < KS; s++)
#pragma unroll
          for (int par = 0; par < 2; par++) {
            const int j = 8 * (KS * kb + s) + 2 * c + par;
            a[par][s] = j < Pn ? H[(size_t)j * Pn] : 0.0;
          }
#pragma unroll
        for (int s = 0; s < KS; s++) {
          dmma_884(v[0], v[1], a[0][s], hz[0][s]);
          dmma_884(v[2], v[3], a[1][s], hz[1][s]);
        }
      }
      const int kx = min(8 * t0 + 2 * c, n2 - 1), kx1 = min(kx + 1, n2 - 1);
      const double2 p0 = __ldg(ph + L.row * npw + kx), p1 = __ldg(ph + L.row * npw + kx1);
      // (E + i O) conj(p)
      acc[0] += v[0] * p0.x + v[2] * p0.y;
      acc[1] += v[2] * p0.x - v[0] * p0.y;
      acc[2] += v[1] * p1.x + v[3] * p1.y;
      acc[3] += v[3] * p1.x - v[1] * p1.y;
    }
    if (m < Pn) {
      double2* o = reinterpret_cast<double2*>(T1 + (size_t)C.off * k.nd) + ((size_t)ind * Pn + m) * n2;
      const int kx = 8 * t0 + 2 * c;
      if (kx < n2) o[kx] = make_double2(acc[0], acc[1]);
      if (kx + 1 < n2) o[kx + 1] = make_double2(acc[2], acc[3]);
    }
  }
}

// y pass: a box's rows (of every order) to its expansion [ky][kx].  The rows'
// sums over even and odd jy against the positive half of ky, E and O, are
// turned by the row's phase and added; node and mirror get E + i O and E - i O.
// A warp owns four complex columns kx and eight nodes ky; Pm is the largest
// order + 1 of the rows.
template <int KS, bool GEN>
__global__ void __launch_bounds__(128) k_up2d_y(KP k, const SepNode* __restrict__ boxes, int nbox,
                                                const SepNode* __restrict__ rows, const int* __restrict__ idx, int Pm,
                                                const double* __restrict__ hx, const double* __restrict__ T1,
                                                const double2* __restrict__ ph) {
  const int ind = blockIdx.z, npw = k.npw, n2 = k.n2, nkb = GEN ? (Pm + 8 * KS - 1) / (8 * KS) : 1;
  const int lane = threadIdx.x & 31, r = lane >> 2, c = lane & 3;
  const int ntk = (n2 + 7) / 8, tiles = (n2 + 3) / 4 * ntk;
  double hn[2][KS];
  const Tiles work(nbox, tiles);
  for (long long w = work.at; w < work.end; w += work.step) {
    const int box = (int)(w / tiles), tile = (int)(w - (long long)box * tiles), nt = tile / ntk, t0 = tile - nt * ntk;
    const int m = 8 * t0 + r;
    auto table = [&](int kb) {
#pragma unroll
      for (int par = 0; par < 2; par++)
#pragma unroll
        for (int s = 0; s < KS; s++) {
          const int j = 8 * (KS * kb + s) + 2 * c + par;
          const double v = j < Pm && m < n2 ? hx[j * npw + m] : 0.0;
          hn[par][s] = (j & 2) ? -v : v;
        }
    };
    if (!GEN) table(0);
    const SepNode N = boxes[box];
    const int col = min(8 * nt + r, 2 * n2 - 1);
    auto load = [&](const SepNode& K, int kb, double (&b)[2][KS]) {
      const double* T = T1 + (size_t)K.off * k.nd + (size_t)ind * 2 * K.p * n2 + col;
#pragma unroll
      for (int s = 0; s < KS; s++)
#pragma unroll
        for (int par = 0; par < 2; par++) {
          const int j = 8 * (KS * kb + s) + 2 * c + par;
          b[par][s] = j < K.p ? T[(size_t)j * 2 * n2] : 0.0;
        }
    };
    double acc[4] = {0.0, 0.0, 0.0, 0.0}, bn[2][KS];
    SepNode Kn = {};
    if (N.cnt > 0) {
      Kn = rows[idx[N.beg]];
      if (!GEN) load(Kn, 0, bn);
    }
#pragma unroll 1
    for (int q = N.beg; q < N.beg + N.cnt; q++) {
      const SepNode K = Kn;
      double b[2][KS];
      if (q + 1 < N.beg + N.cnt) Kn = rows[idx[q + 1]];
      if (!GEN) {
#pragma unroll
        for (int s = 0; s < KS; s++) {
          b[0][s] = bn[0][s];
          b[1][s] = bn[1][s];
        }
        if (q + 1 < N.beg + N.cnt) load(Kn, 0, bn);
      }
      double v[4] = {0.0, 0.0, 0.0, 0.0};
      for (int kb = 0; kb < nkb; kb++) {
        if (GEN) {
          table(kb);
          load(K, kb, b);
        }
#pragma unroll
        for (int s = 0; s < KS; s++) {
          dmma_884(v[0], v[1], hn[0][s], b[0][s]);
          dmma_884(v[2], v[3], hn[1][s], b[1][s]);
        }
      }
      // the node's phase is conj(p), its mirror's p: E' = cr E + ci O and
      // O' = cr O - ci E give E' + i O' and E' - i O'
      const double2 p = __ldg(ph + K.row * npw + min(m, n2 - 1));
      acc[0] += p.x * v[0] + p.y * v[2];
      acc[1] += p.x * v[1] + p.y * v[3];
      acc[2] += p.x * v[2] - p.y * v[0];
      acc[3] += p.x * v[3] - p.y * v[1];
    }
    const int q = 4 * nt + c;  // the lane's complex column
    if (q < n2 && m < n2) {
      double2* o = k.mp + ((size_t)N.off * k.nd + ind) * k.nexp + q;
      o[(size_t)m * n2] = make_double2(acc[0] - acc[3], acc[1] + acc[2]);
      o[(size_t)(n2 + m) * n2] = make_double2(acc[0] + acc[3], acc[1] - acc[2]);
    }
  }
}

// ------------------------------------------------------------ downward
// The mirror image: the cut level's local expansions to the leaves' Taylor
// blocks (g2dpw2local_real_vec after the split),
//   U[b][kx]  = i^b sum_ky x2l[b][ky] py(ky) L[ky][kx]       per row
//   lo[b][a]  = 2 Re i^a sum_kx x2l[a][kx] px(kx) U[b][kx]   per leaf
// with p(i, k) = exp(+i t_k sh_i).  The mirror nodes make every sum two real
// products of depth n2: with S = L[m] p + L[mb] p* and D = L[m] p - L[mb] p*,
// even orders take tx . S, odd ones i tx . D, tx[a] = (-1)^(a/2) x2l[a].

// y pass: four complex columns kx of a box per warp, turned to the row's phase
// with four multiply-adds per element; 2 U products of KS steps give 16 U
// orders b from 32 blockIdx.y on: U[kx][b].  The rows of every order in one
// launch (Pm: the largest order + 1), each with the tiles that it has; small
// plans are bound by their launches.  GEN: node halves beyond 4 KS in blocks.
template <int KS, int U, bool GEN>
__global__ void __launch_bounds__(128) k_down2d_y(KP k, const SepNode* __restrict__ rows, int nrow,
                                                  const int* __restrict__ slots, int Pm,
                                                  double* __restrict__ T1, const double2* __restrict__ ph) {
  const int ind = blockIdx.z, npw = k.npw, n2 = k.n2, nkb = GEN ? (n2 + 4 * KS - 1) / (4 * KS) : 1;
  const int lane = threadIdx.x & 31, r = lane >> 2, c = lane & 3, ctile = (n2 + 3) / 4;
  const int u0 = 2 * blockIdx.y;
  const double sg = (r & 1) ? 1.0 : -1.0;
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
  if (!GEN) table(0);
  const Tiles work(nrow, ctile);
  for (long long w = work.at; w < work.end; w += work.step) {
    const int row = (int)(w / ctile), nt = (int)(w - (long long)row * ctile);
    const SepNode K = rows[row];
    if (K.p <= 16 * u0) continue;
    const double2* L = k.loc + ((size_t)slots[row] * k.nd + ind) * k.nexp + min(4 * nt + (r >> 1), n2 - 1);
    double acc[U][4];
#pragma unroll
    for (int u = 0; u < U; u++) acc[u][0] = acc[u][1] = acc[u][2] = acc[u][3] = 0.0;
    for (int kb = 0; kb < nkb; kb++) {
      if (GEN) table(kb);
#pragma unroll
      for (int s = 0; s < KS; s++) {
        const int m = min(4 * (KS * kb + s) + c, n2 - 1);
        const double2 a = L[(size_t)m * n2], b = L[(size_t)(n2 + m) * n2];
        const double o1 = (r & 1) ? a.y : a.x, o2 = (r & 1) ? b.y : b.x;
        const double t1 = sg * ((r & 1) ? a.x : a.y), t2 = sg * ((r & 1) ? b.x : b.y);
        const double2 p = __ldg(ph + K.row * npw + m);
        const double S = fma(p.y, t1 - t2, p.x * (o1 + o2)), D = fma(p.y, t1 + t2, p.x * (o1 - o2));
#pragma unroll
        for (int u = 0; u < U; u++)
          if (u == 0 || 16 * (u0 + u) < K.p) {
            dmma_884(acc[u][0], acc[u][1], tx[u][0][s], S);
            dmma_884(acc[u][2], acc[u][3], tx[u][1][s], D);
          }
      }
    }
    const int q = 4 * nt + c;  // the lane's complex column
    if (q < n2) {
      double2* o = reinterpret_cast<double2*>(T1 + (size_t)K.off * k.nd) + ((size_t)ind * n2 + q) * K.p;
#pragma unroll
      for (int u = 0; u < U; u++) {
        const int a = 2 * (8 * (u0 + u) + r);
        if (a < K.p) o[a] = make_double2(acc[u][0], acc[u][1]);
        if (a + 1 < K.p) o[a + 1] = make_double2(-acc[u][3], acc[u][2]);
      }
    }
  }
}

// x pass: eight rows b of a leaf's block per warp, 16 U orders a from
// 32 blockIdx.y on;
// rows of E = P rounded up to even (the padding zero).  f32: each coefficient
// as the FP32 pair (v, v) that the mixed evaluation reads.
template <int KS, int U, bool GEN>
__global__ void __launch_bounds__(128) k_down2d_x(KP k, const SepNode* __restrict__ rows,
                                                  const SepLeaf* __restrict__ leaves,
                                                  const int* __restrict__ leaf_row, int nleaf, int Pn, int f32,
                                                  const double* __restrict__ T1, double* __restrict__ lo_all,
                                                  const double2* __restrict__ ph) {
  const int ind = blockIdx.z, npw = k.npw, n2 = k.n2, E = (Pn + 1) & ~1;
  const int nkb = GEN ? (n2 + 4 * KS - 1) / (4 * KS) : 1;
  const int lane = threadIdx.x & 31, r = lane >> 2, c = lane & 3, mtiles = (Pn + 7) / 8, u0 = 2 * blockIdx.y;
  double tx[U][2][KS];
  auto table = [&](int kb) {
#pragma unroll
    for (int u = 0; u < U; u++)
#pragma unroll
      for (int par = 0; par < 2; par++)
#pragma unroll
        for (int s = 0; s < KS; s++) {
          const int a = 2 * (8 * (u0 + u) + r) + par, m = 4 * (KS * kb + s) + c;
          tx[u][par][s] = (a < Pn && m < n2) ? ((a & 2) ? -k.x2l[a * npw + m] : k.x2l[a * npw + m]) : 0.0;
        }
  };
  if (!GEN) table(0);
  const Tiles work(nleaf, mtiles);
  for (long long w = work.at; w < work.end; w += work.step) {
    const int leaf = (int)(w / mtiles), nt = (int)(w - (long long)leaf * mtiles);
    const SepLeaf F = leaves[leaf];
    const double2* L = reinterpret_cast<const double2*>(T1 + (size_t)rows[leaf_row[leaf]].off * k.nd) +
                       (size_t)ind * Pn * n2 + min(8 * nt + r, Pn - 1);
    double acc[U][4];
#pragma unroll
    for (int u = 0; u < U; u++) acc[u][0] = acc[u][1] = acc[u][2] = acc[u][3] = 0.0;
    for (int kb = 0; kb < nkb; kb++) {
      if (GEN) table(kb);
#pragma unroll
      for (int s = 0; s < KS; s++) {
        const int m = min(4 * (KS * kb + s) + c, n2 - 1);
        const double2 z = L[(size_t)m * Pn], p = __ldg(ph + F.row * npw + m);
        const double re = fma(-z.y, p.y, z.x * p.x), im = fma(z.y, p.x, z.x * p.y);
#pragma unroll
        for (int u = 0; u < U; u++)
          if (u == 0 || 16 * (u0 + u) < Pn) {
            dmma_884(acc[u][0], acc[u][1], tx[u][0][s], re);
            dmma_884(acc[u][2], acc[u][3], tx[u][1][s], im);
          }
      }
    }
    double* out = lo_all + F.off + (size_t)ind * Pn * E;
#pragma unroll
    for (int i = 0; i < 2; i++) {
      const int q = 8 * nt + 2 * c + i;
      if (q >= Pn) continue;
#pragma unroll
      for (int u = 0; u < U; u++) {
        const int a = 2 * (8 * (u0 + u) + r);
        if (a >= Pn) continue;
        const double ve = 2.0 * acc[u][i], vo = a + 1 < Pn ? -2.0 * acc[u][2 + i] : 0.0;
        if (f32) {
          const float e = (float)ve, o = (float)vo;
          reinterpret_cast<float4*>(out)[(q * E + a) >> 1] = make_float4(e, e, o, o);
        } else {
          *reinterpret_cast<double2*>(out + q * E + a) = make_double2(ve, vo);
        }
      }
    }
  }
}

template <int N>
using int_c = std::integral_constant<int, N>;

cudaError_t sep_up_2d(const KP& k, const SepDev& S, const double* hbuf, cudaStream_t st, long long& launches) {
  const int n2 = k.n2, ntk = (n2 + 7) / 8;
  auto cases = [&](int Pn, auto launch) {
    switch (Pn > 32 ? 5 : (Pn + 7) / 8) {
      case 1: launch(int_c<1>(), std::false_type()); break;
      case 2: launch(int_c<2>(), std::false_type()); break;
      case 3: launch(int_c<3>(), std::false_type()); break;
      case 4: launch(int_c<4>(), std::false_type()); break;
      default: launch(int_c<4>(), std::true_type()); break;
    }
    launches++;
  };
  int pmax = 1;
  for (const SepGroup& G : S.groups) {
    const int Pn = G.p + 1, nrow = G.cend - G.cbeg;
    pmax = std::max(pmax, Pn);
    const dim3 g = tiles_grid(nrow, (Pn + 7) / 8 * ntk, k.nd, S.sms);
    cases(Pn, [&](auto KS, auto GEN) {
      k_up2d_x<decltype(KS)::value, decltype(GEN)::value>
          <<<g, 128, 0, st>>>(k, S.cols + G.cbeg, nrow, S.leaves, Pn, S.hx, hbuf, S.t1, S.ph);
    });
  }
  if (S.nboxes > 0) {
    const dim3 g = tiles_grid(S.nboxes, (n2 + 3) / 4 * ntk, k.nd, S.sms);
    cases(pmax, [&](auto KS, auto GEN) {
      k_up2d_y<decltype(KS)::value, decltype(GEN)::value>
          <<<g, 128, 0, st>>>(k, S.boxes, S.nboxes, S.cols, S.box_kids, pmax, S.hx, S.t1, S.ph);
    });
  }
  return cudaGetLastError();
}

cudaError_t sep_down_2d(const KP& k, const SepDev& S, double* lo, int f32, cudaStream_t st, long long& launches) {
  const int n2 = k.n2, ksm = (n2 + 3) / 4;
  // launch(KS, U, GEN) for orders up to Pn, blockIdx.y the blocks of 32 orders
  auto cases = [&](int Pn, auto launch) {
    switch (2 * (ksm > 8 ? 0 : ksm) + (Pn <= 16 ? 0 : 1)) {
#define DOWN_CASE(N)                                                        \
  case 2 * N: launch(int_c<N>(), int_c<1>(), std::false_type()); break;     \
  case 2 * N + 1: launch(int_c<N>(), int_c<2>(), std::false_type()); break;
      DOWN_CASE(1) DOWN_CASE(2) DOWN_CASE(3) DOWN_CASE(4) DOWN_CASE(5) DOWN_CASE(6) DOWN_CASE(7) DOWN_CASE(8)
#undef DOWN_CASE
      default: launch(int_c<8>(), int_c<2>(), std::true_type()); break;
    }
    launches++;
  };
  int pmax = 0, nrow = 0;
  for (const SepGroup& G : S.groups) {
    pmax = std::max(pmax, G.p + 1);
    nrow = std::max(nrow, G.cend);
  }
  if (nrow == 0) return cudaSuccess;
  dim3 gy = tiles_grid(nrow, ksm, k.nd, S.sms);
  gy.y = (pmax + 31) / 32;
  cases(pmax, [&](auto N, auto U, auto F) {
    k_down2d_y<decltype(N)::value, decltype(U)::value, decltype(F)::value>
        <<<gy, 128, 0, st>>>(k, S.cols, nrow, S.col_slot, pmax, S.t1, S.ph);
  });
  for (const SepGroup& G : S.groups) {
    const int Pn = G.p + 1, nleaf = G.lend - G.lbeg;
    dim3 gx = tiles_grid(nleaf, (Pn + 7) / 8, k.nd, S.sms);
    gx.y = (Pn + 31) / 32;
    cases(Pn, [&](auto N, auto U, auto F) {
      k_down2d_x<decltype(N)::value, decltype(U)::value, decltype(F)::value><<<gx, 128, 0, st>>>(
          k, S.cols, S.leaves + G.lbeg, S.leaf_col + G.lbeg, nleaf, Pn, Pn <= f32, S.t1, lo, S.ph);
    });
  }
  return cudaGetLastError();
}
}  // namespace

cudaError_t sep_up(const KP& k, const SepDev& S, const double* hbuf, cudaStream_t st, long long& launches) {
  return k.dim == 3 ? sep_up_3d(k, S, hbuf, st, launches) : sep_up_2d(k, S, hbuf, st, launches);
}
cudaError_t sep_down(const KP& k, const SepDev& S, double* lo, int f32, cudaStream_t st, long long& launches) {
  return k.dim == 3 ? sep_down_3d(k, S, lo, st, launches) : sep_down_2d(k, S, lo, f32, st, launches);
}

}  // namespace fgtb
