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
// tensor pipe.
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

}  // namespace fgtb
