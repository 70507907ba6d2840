// 3D plane-wave route on the FP64 tensor cores: the exact exponential sums
// between a box's expansion and its points (g3dpwevalp/g/h_vec,
// g3drouts.f:2268-2660), in the plane-wave scheme for the leaves whose order
// is too high for a block, in the NUFFT scheme for every box.
#include <algorithm>

#include "fgt_kcommon.cuh"

namespace fgtb {

namespace {

// ------------------------------------------------------------ evaluation
//   pot = 2 Re sum_q W(q) sum_kx e^{i t_kx x} L[q][kx],  q = (kz, ky) over the
// stored half in z, W(q) = e^{i t_kz z} e^{i t_ky y}.  The x sum is the large
// one (npw^2 n2 terms a point); with the mirror node mb of m it is two real
// products of depth n2,
//   sum_{m < n2} cos(t_m x) (L[m] + L[mb]) + i sin(t_m x) (L[m] - L[mb]),
// with the points as rows (eight per tile) and the complex columns q; its x
// derivatives are the same products with the rows -t sin, t cos and -t^2 cos,
// -t^2 sin (PGH pairs of products).  One CTA of four warps per chunk of at
// most 8 MT points: rows and the phases of y and z in shared memory, the
// expansion read from global memory (L2) straight into the fragments, once
// per chunk; the warps take pairs of column tiles in turn, and the lane's
// sums over its columns are added in a fixed order at the end.  Bound by the
// tensor pipe.  Measured (B200, eps 1e-6, npw 26; before: a thread per point and
// node on the scalar pipe): forces of 3e5 blob points 1375 -> 157 us, potentials
// of 1e5 uniform points 171 -> 67 us.
template <int PGH>
__host__ __device__ constexpr int pwev_tiles() { return PGH == 1 ? 4 : PGH == 2 ? 2 : 1; }

struct PwevDims {
  int K, lda, ldy;
  size_t total;  // doubles
  __host__ __device__ PwevDims(int npw, int MT, int pgh) {
    const int n2 = npw / 2, rows = 8 * MT, nc = pgh == 1 ? 1 : pgh == 2 ? 4 : 10;
    K = (n2 + 3) & ~3;
    lda = (K & 15) <= 4 ? (K & ~15) + 4 : (K & ~15) + 20;  // 4 (mod 16): conflict-free A fragments
    ldy = ((npw + 3) & ~7) + 4;                             // 4 (mod 8) complex
    total = (size_t)2 * pgh * rows * lda + (size_t)2 * rows * (ldy + n2) + (size_t)4 * rows * nc + 3 * rows;
  }
};

template <int MT, int PGH>
__device__ __forceinline__ void pwev_body(const KP& k, const double* __restrict__ L, const double* A,
                                          const double2* Y, const double2* Zp, const PwevDims& Z, int rows,
                                          double (*sum)[ncomp<3, PGH>()]) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, r = lane >> 2, c = lane & 3;
  const int npw = k.npw, n2 = k.n2, ncol = n2 * npw, ks = Z.K >> 2, ntp = (ncol + 7) / 8, ra = rows * Z.lda;
#pragma unroll
  for (int i = 0; i < MT; i++)
#pragma unroll
    for (int v = 0; v < ncomp<3, PGH>(); v++) sum[i][v] = 0.0;
  for (int np = warp; np < ntp; np += 4) {
    double acc[2][MT][PGH][4];
#pragma unroll
    for (int h = 0; h < 2; h++)
#pragma unroll
      for (int i = 0; i < MT; i++)
#pragma unroll
        for (int g = 0; g < PGH; g++) acc[h][i][g][0] = acc[h][i][g][1] = acc[h][i][g][2] = acc[h][i][g][3] = 0.0;
    const double* B[2];
#pragma unroll
    for (int h = 0; h < 2; h++) B[h] = L + (size_t)min(8 * np + 4 * h + (r >> 1), ncol - 1) * 2 * npw + (r & 1);
    auto fetch = [&](int s, double (&a)[2][2], double (&b)[2][2]) {
#pragma unroll
      for (int j = 0; j < 2; j++) {
        const int m = min(4 * (s + j) + c, n2 - 1);
#pragma unroll
        for (int h = 0; h < 2; h++) {
          a[j][h] = B[h][2 * m];
          b[j][h] = B[h][2 * (npw - 1 - m)];
        }
      }
    };
    double an[2][2], bn[2][2];
    fetch(0, an, bn);
    for (int s = 0; s < ks; s += 2) {
      double S[2][2], D[2][2];
#pragma unroll
      for (int j = 0; j < 2; j++)
#pragma unroll
        for (int h = 0; h < 2; h++) {
          S[j][h] = an[j][h] + bn[j][h];
          D[j][h] = an[j][h] - bn[j][h];
        }
      if (s + 2 < ks) fetch(s + 2, an, bn);
#pragma unroll
      for (int j = 0; j < 2; j++)
        if (s + j < ks) {
#pragma unroll
          for (int i = 0; i < MT; i++)
#pragma unroll
            for (int g = 0; g < PGH; g++) {
              const double* ap = A + (size_t)2 * g * ra + (8 * i + r) * Z.lda + 4 * (s + j) + c;
              const double as = ap[0], ad = ap[ra];
#pragma unroll
              for (int h = 0; h < 2; h++) {
                dmma_884(acc[h][i][g][0], acc[h][i][g][1], as, S[j][h]);
                dmma_884(acc[h][i][g][2], acc[h][i][g][3], ad, D[j][h]);
              }
            }
        }
    }
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const int q = 8 * np + 4 * h + c;  // the lane's column
      if (q < ncol) {
        const int kz = q / npw, ky = q - kz * npw;
        const double ty = (2 * (ky - n2) + 1) * k.t1, tz = (2 * (kz - n2) + 1) * k.t1;
#pragma unroll
        for (int i = 0; i < MT; i++) {
          const double2 w = cmul(Y[(8 * i + r) * Z.ldy + ky], Zp[(8 * i + r) * n2 + kz]);
          double2 f[PGH];  // (sums of x derivative order g) W
#pragma unroll
          for (int g = 0; g < PGH; g++)
            f[g] = cmul(make_double2(acc[h][i][g][0] - acc[h][i][g][3], acc[h][i][g][1] + acc[h][i][g][2]), w);
          sum[i][0] += f[0].x;
          if constexpr (PGH >= 2) {
            sum[i][1] += f[1].x;
            sum[i][2] = fma(-ty, f[0].y, sum[i][2]);
            sum[i][3] = fma(-tz, f[0].y, sum[i][3]);
          }
          if constexpr (PGH >= 3) {
            sum[i][4] += f[2].x;
            sum[i][5] = fma(-ty * ty, f[0].x, sum[i][5]);
            sum[i][6] = fma(-tz * tz, f[0].x, sum[i][6]);
            sum[i][7] = fma(-ty, f[1].y, sum[i][7]);
            sum[i][8] = fma(-tz, f[1].y, sum[i][8]);
            sum[i][9] = fma(-ty * tz, f[0].x, sum[i][9]);
          }
        }
      }
    }
  }
}

template <int PGH>
__global__ void __launch_bounds__(128) k_eval3d_pw(KP k, const EvalTask* __restrict__ tasks) {
  constexpr int MT = pwev_tiles<PGH>(), ROWS = 8 * MT, NC = ncomp<3, PGH>();
  const EvalTask T = tasks[blockIdx.x];
  const int ind = blockIdx.y, npw = k.npw, n2 = k.n2, tid = threadIdx.x;
  const PwevDims Z(npw, MT, PGH);
  extern __shared__ double sm[];
  double* A = sm;                                                       // [PGH][2][ROWS][lda]
  double2* Y = reinterpret_cast<double2*>(A + (size_t)2 * PGH * ROWS * Z.lda);  // [ROWS][ldy]
  double2* Zp = Y + (size_t)ROWS * Z.ldy;                               // [ROWS][n2]
  double* red = reinterpret_cast<double*>(Zp + (size_t)ROWS * n2);      // [4][ROWS][NC]
  double* xyz = red + (size_t)4 * ROWS * NC;                            // [3][ROWS]
  const double* L = reinterpret_cast<const double*>(k.loc + ((size_t)T.slot * k.nd + ind) * k.nexp);
  const double* pts = T.set ? k.trg : k.src;
  double* out = T.set ? k.pottarg : k.pot;
  const int nc = T.set ? k.nc_t : k.nc_s;
  for (int p0 = blockIdx.z * ROWS; p0 < T.n; p0 += gridDim.z * ROWS) {
    const int np = min(ROWS, T.n - p0);
    __syncthreads();
    for (int e = tid; e < 3 * ROWS; e += 128) {
      const int d = e / ROWS, pt = e - d * ROWS;
      xyz[e] = (pts[(size_t)3 * (T.i0 + p0 + min(pt, np - 1)) + d] - k.centers[3 * T.box + d]) * k.dsq;
    }
    __syncthreads();
    for (int e = tid; e < ROWS * (Z.K + npw + n2); e += 128) {
      const int pt = e % ROWS, m = e / ROWS;
      if (m < Z.K) {
        double sn = 0.0, cs = 0.0, t = 0.0;
        if (m < n2 && pt < np) {
          t = (2 * (m - n2) + 1) * k.t1;
          sincos(t * xyz[pt], &sn, &cs);
        }
        double* a = A + pt * Z.lda + m;
        const int ra = ROWS * Z.lda;
        a[0] = cs;
        a[ra] = sn;
        if (PGH >= 2) {
          a[2 * ra] = -t * sn;
          a[3 * ra] = t * cs;
        }
        if (PGH >= 3) {
          a[4 * ra] = -t * t * cs;
          a[5 * ra] = -t * t * sn;
        }
      } else if (m < Z.K + npw) {
        const int ky = m - Z.K;
        Y[pt * Z.ldy + ky] = cexpi((2 * (ky - n2) + 1) * k.t1 * xyz[ROWS + pt]);
      } else {
        const int kz = m - Z.K - npw;
        Zp[pt * n2 + kz] = cexpi((2 * (kz - n2) + 1) * k.t1 * xyz[2 * ROWS + pt]);
      }
    }
    __syncthreads();
    double sum[MT][NC];
#pragma unroll
    for (int i = 0; i < MT; i++)
#pragma unroll
      for (int v = 0; v < NC; v++) sum[i][v] = 0.0;
    const int nmt = (np + 7) / 8;
    if (nmt == 1) {
      pwev_body<1, PGH>(k, L, A, Y, Zp, Z, ROWS, sum);
    } else if constexpr (MT >= 2) {
      if (MT == 2 || nmt == 2) pwev_body<2, PGH>(k, L, A, Y, Zp, Z, ROWS, sum);
      else if constexpr (MT >= 4) {
        if (nmt == 3) pwev_body<3, PGH>(k, L, A, Y, Zp, Z, ROWS, sum);
        else pwev_body<4, PGH>(k, L, A, Y, Zp, Z, ROWS, sum);
      }
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
    for (int e = tid; e < np * NC; e += 128) {
      const int pt = e / NC, v = e - pt * NC;
      if (v >= nc) continue;
      double a = 0.0;
#pragma unroll
      for (int w = 0; w < 4; w++) a += red[((size_t)w * ROWS + pt) * NC + v];
      out[((size_t)(T.i0 + p0 + pt) * nc + v) * k.nd + ind] += 2.0 * a * (v == 0 ? 1.0 : v < 4 ? k.dsq : k.dsq * k.dsq);
    }
  }
}

// ------------------------------------------------------------ formation
//   mp[q][kx] (+)= sum_s X_s(kx) b_s(q),  b_s = q_s Y_s(ky) Z_s(kz), q = (kz, ky)
// with X_s(kx) = w_kx e^{-i t_kx x_s} (and Y, Z likewise), conjugate at the
// mirror node: E = sum Re X b and O = sum Im X b over the positive nodes m are
// two real products with the sources as depth, and node m gets E + i O, its
// mirror E - i O.  A task is a box with the source ranges whose expansion it
// takes about the box's centre.  A warp keeps NP column pairs (eight complex
// columns each) of the box in registers for all its sources; those come 32 at
// a time, their factors formed once per CTA (a thread per source and
// dimension, by recurrence) into shared memory, where a B fragment is one
// complex product of two of them.  With dipoles a source stages three columns
// (dip3_coef, the factor of one dimension times v_d (-i t dsq)), ten sources
// at a time.  Bound by the tensor pipe (45%) and by the barriers around the
// factors' staging.  Measured (B200, eps 1e-9, npw 38;
// before: a thread per coefficient on the scalar pipe, an expansion per leaf,
// then the merges): 3e5 uniform points 1.2 -> 0.53 ms; 1e5 for gradients, where
// every leaf takes this route, 2.3 -> 0.92 ms.
template <int MT>
__host__ __device__ constexpr int pwform_pairs() { return MT == 1 ? 4 : MT == 2 ? 3 : MT == 3 ? 2 : 1; }
constexpr int PWF_SC = 32;  // source columns per batch

struct PwformDims {
  int lda, ldy;
  size_t total;
  __host__ __device__ PwformDims(int npw, int MT) {
    lda = PWF_SC + 4;
    ldy = ((npw + 3) & ~7) + 4;
    total = (size_t)2 * 8 * MT * lda + (size_t)2 * PWF_SC * (ldy + npw / 2);
  }
};

template <int MT>
__global__ void __launch_bounds__(128) k_form3d_pw(KP k, const PwFormTask* __restrict__ tasks,
                                                   const SrcRange* __restrict__ ranges, int t0) {
  constexpr int NP = pwform_pairs<MT>();
  const PwFormTask T = tasks[blockIdx.x];
  const int ind = blockIdx.z, npw = k.npw, n2 = k.n2, ncol = n2 * npw, tid = threadIdx.x;
  const int lane = tid & 31, warp = tid >> 5, r = lane >> 2, c = lane & 3;
  const PwformDims Z(npw, MT);
  extern __shared__ double sm[];
  double* A = sm;                                                        // [2][8 MT][lda]: Re, Im X[m][s]
  double2* Y = reinterpret_cast<double2*>(A + (size_t)2 * 8 * MT * Z.lda);  // [s][ldy]
  double2* Zf = Y + (size_t)PWF_SC * Z.ldy;                              // [s][n2]
  const int vc = k.ifdipole ? 3 : 1, chs = PWF_SC / vc;
  const int pair0 = (blockIdx.y * 4 + warp) * NP;
  double acc[NP][2][MT][4];
  int yo[NP][2], zo[NP][2];
#pragma unroll
  for (int p = 0; p < NP; p++)
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const int q = min(8 * (pair0 + p) + 4 * h + (r >> 1), ncol - 1);
      zo[p][h] = q / npw;
      yo[p][h] = q - zo[p][h] * npw;
#pragma unroll
      for (int t = 0; t < MT; t++) acc[p][h][t][0] = acc[p][h][t][1] = acc[p][h][t][2] = acc[p][h][t][3] = 0.0;
    }
  for (int e = T.beg; e < T.beg + T.cnt; e++) {
    const SrcRange R = ranges[e];
    for (int c0 = 0; c0 < R.n; c0 += chs) {
      const int m = vc * min(chs, R.n - c0), mp = (m + 3) & ~3;
      __syncthreads();
      if (tid < 3 * PWF_SC) {
        const int d = tid / PWF_SC, s = tid - d * PWF_SC;
        if (s < mp) {
          double u = 0.0, q = 0.0, dv[3] = {0.0, 0.0, 0.0}, ca = 0.0, cb = 0.0;
          if (s < m) {
            const int i = R.s0 + c0 + s / vc;
            u = (k.src[(size_t)3 * i + d] - k.centers[3 * T.box + d]) * k.dsq;
            q = src_charge(k, i, ind);
            if (k.ifdipole) src_dipole<3>(k, i, ind, dv);
            dip3_coef(s % vc, d, q, dv, ca, cb);
          }
          double2 f = cexpi(-k.t1 * u);
          const double2 ff = cmul(f, f);
          for (int j = 0; j < n2; j++) {  // positive node j: t = (2j+1) t1 at n2 + j, its mirror at n2 - 1 - j
            const double w = k.ws[n2 + j], td = (2 * j + 1) * k.t1 * k.dsq * cb;
            // (ca - i t dsq cb) w e^{-i t u}
            const double2 g = make_double2(w * fma(ca, f.x, td * f.y), w * fma(ca, f.y, -td * f.x));
            if (d == 0) {
              const int mr = j - 8 * t0;
              if (mr >= 0 && mr < 8 * MT) {
                A[mr * Z.lda + s] = g.x;
                A[(8 * MT + mr) * Z.lda + s] = g.y;
              }
            } else if (d == 1) {
              Y[s * Z.ldy + n2 + j] = g;
              Y[s * Z.ldy + n2 - 1 - j] = make_double2(g.x, -g.y);
            } else {
              Zf[s * n2 + n2 - 1 - j] = make_double2(g.x, -g.y);
            }
            f = cmul(f, ff);
          }
          if (d == 0)
            for (int mr = max(0, n2 - 8 * t0); mr < 8 * MT; mr++) A[mr * Z.lda + s] = A[(8 * MT + mr) * Z.lda + s] = 0.0;
        }
      }
      __syncthreads();
      for (int st = 0; st < mp; st += 4) {
        double a[MT][2];
#pragma unroll
        for (int t = 0; t < MT; t++) {
          a[t][0] = A[(8 * t + r) * Z.lda + st + c];
          a[t][1] = A[(8 * MT + 8 * t + r) * Z.lda + st + c];
        }
        const double2* Ys = Y + (st + c) * Z.ldy;
        const double2* Zs = Zf + (st + c) * n2;
#pragma unroll
        for (int p = 0; p < NP; p++)
#pragma unroll
          for (int h = 0; h < 2; h++) {
            const double2 y = Ys[yo[p][h]], z = Zs[zo[p][h]];
            const double b = (r & 1) ? fma(y.x, z.y, y.y * z.x) : fma(y.x, z.x, -y.y * z.y);
#pragma unroll
            for (int t = 0; t < MT; t++) {
              dmma_884(acc[p][h][t][0], acc[p][h][t][1], a[t][0], b);
              dmma_884(acc[p][h][t][2], acc[p][h][t][3], a[t][1], b);
            }
          }
      }
    }
  }
  double2* out = k.mp + ((size_t)T.slot * k.nd + ind) * k.nexp;
#pragma unroll
  for (int p = 0; p < NP; p++)
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const int q = 8 * (pair0 + p) + 4 * h + c;  // the lane's column
      if (q < ncol) {
#pragma unroll
        for (int t = 0; t < MT; t++) {
          const int m = 8 * (t0 + t) + r;
          if (m < n2) {
            const double* v = acc[p][h][t];
            double2* op = out + (size_t)q * npw + n2 + m;
            double2* om = out + (size_t)q * npw + n2 - 1 - m;
            double2 vp = make_double2(v[0] - v[3], v[1] + v[2]), vm = make_double2(v[0] + v[3], v[1] - v[2]);
            if (T.add) {
              const double2 a = *op, b = *om;
              vp = make_double2(vp.x + a.x, vp.y + a.y);
              vm = make_double2(vm.x + b.x, vm.y + b.y);
            }
            *op = vp;
            *om = vm;
          }
        }
      }
    }
}

}  // namespace

#define CK(x)                               \
  do {                                      \
    cudaError_t e_ = (x);                   \
    if (e_ != cudaSuccess) return e_;       \
  } while (0)

cudaError_t launch_eval3d_pw(const KP& k, const EvalTask* tasks, int ntask, int nmax, int pgh, cudaStream_t st) {
  if (ntask <= 0) return cudaSuccess;
#define PWEV_CASE(PG)                                                                             \
  {                                                                                               \
    constexpr int MT = pwev_tiles<PG>();                                                          \
    const size_t sh = PwevDims(k.npw, MT, PG).total * 8;                                          \
    if (sh > 227 * 1024) return cudaErrorNotSupported;                                            \
    CK(smem_limit(k_eval3d_pw<PG>));                                                              \
    const dim3 g(ntask, k.nd, std::max(1, std::min(256, (nmax + 8 * MT - 1) / (8 * MT))));         \
    k_eval3d_pw<PG><<<g, 128, sh, st>>>(k, tasks);                                                \
  }
  if (pgh <= 1) PWEV_CASE(1)
  else if (pgh == 2) PWEV_CASE(2)
  else PWEV_CASE(3)
#undef PWEV_CASE
  return cudaGetLastError();
}

cudaError_t launch_form3d_pw(const KP& k, const PwFormTask* tasks, int ntask, const SrcRange* ranges,
                             cudaStream_t st, long long& launches) {
  if (ntask <= 0) return cudaSuccess;
  const int tiles = (k.n2 + 7) / 8, pairs = (k.n2 * k.npw + 7) / 8;
  for (int t0 = 0; t0 < tiles; t0 += 4) {
    switch (std::min(4, tiles - t0)) {
#define PWF_CASE(MT)                                                                                    \
  case MT: {                                                                                            \
    const size_t sh = PwformDims(k.npw, MT).total * 8;                                                  \
    if (sh > 227 * 1024) return cudaErrorNotSupported;                                                  \
    CK(smem_limit(k_form3d_pw<MT>));                                                                    \
    const dim3 g(ntask, (pairs + 4 * pwform_pairs<MT>() - 1) / (4 * pwform_pairs<MT>()), k.nd);         \
    k_form3d_pw<MT><<<g, 128, sh, st>>>(k, tasks, ranges, t0);                                          \
    break;                                                                                              \
  }
      PWF_CASE(1) PWF_CASE(2) PWF_CASE(3) PWF_CASE(4)
#undef PWF_CASE
    }
    launches++;
  }
  return cudaGetLastError();
}

}  // namespace fgtb
