// Y L^{-dagger} or Y L for the Cholesky factor L of a small Gram matrix M = L L^dagger, by one CTA in shared memory:
// the body of chol_apply.cu (rows of Y spread over the SMs) and recover_small.cu (all rows in one CTA).
//
// Y's rows stand below M's and are eliminated along with them: what the elimination leaves of a row y is y L^{-dagger},
// so neither the inverse factor nor a product with it are needed.  Bound: the serial chain.  A panel of NB
// columns (8 real, 4 complex) costs every thread the factorisation of the panel's diagonal block, done redundantly
// in registers without a barrier, then one row of the panel, then a rank-NB update of the trailing part with two rows a
// thread: 2 barriers per NB columns.
//
// Where M is near the identity (the second CholeskyQR pass; the weights of an idempotent density) the symmetric
// factors M^{-1/2} and M^{1/2} take the place of the triangular ones: with E = M - 1 the series
// 1 - E/2 + 3/8 E^2 and 1 + E/2 - E^2/8, whose next terms 5/16 E^3 and 1/16 E^3 are below 2e-17 for
// ||E||_inf <= kNearNorm.  Two products of the rows with E replace the chain.
#pragma once

#include "rr_common.cuh"

namespace rr {
namespace cholr {

constexpr int THREADS = 256;
constexpr double kNearNorm = 4e-6;

template <int PL>
struct Panel {
  static constexpr int NB = PL == 1 ? 8 : 4;
};

// acc -= a conj(b)
template <int PL>
__device__ __forceinline__ void sub_conj(double (&acc)[PL], const double (&a)[PL], const double (&b)[PL]) {
  if constexpr (PL == 1) {
    acc[0] = fma(-a[0], b[0], acc[0]);
  } else {
    acc[0] = fma(-a[0], b[0], fma(-a[1], b[1], acc[0]));
    acc[1] = fma(-a[1], b[0], fma(a[0], b[1], acc[1]));
  }
}

template <int PL>
__device__ __forceinline__ void ld(double (&v)[PL], const double* p) {
  if constexpr (PL == 1) {
    v[0] = *p;
  } else {
    const double2 d = *reinterpret_cast<const double2*>(p);
    v[0] = d.x;
    v[1] = d.y;
  }
}
template <int PL>
__device__ __forceinline__ void st(double* p, const double (&v)[PL]) {
  if constexpr (PL == 1) *p = v[0];
  else *reinterpret_cast<double2*>(p) = make_double2(v[0], v[1]);
}

// out[row][c] = sum_{k >= k0(c)} rows[row][k] F[k][c] over the CTA's rows, k0 = LOWER ? c : 0; out has the rows' pitch.
template <int PL, bool LOWER>
__device__ __forceinline__ void rows_times(const double* rows, const double* F, int r, int ldm, int nrows, double* out) {
  for (int e = threadIdx.x; e < nrows * r; e += THREADS) {
    const int row = e / r, c = e - row * r;
    double acc[PL] = {};
#pragma unroll 4
    for (int k = LOWER ? c : 0; k < r; ++k) {
      double y[PL], f[PL];
      ld<PL>(y, rows + (row * ldm + k) * PL);
      ld<PL>(f, F + (k * ldm + c) * PL);
      if constexpr (PL == 1) {
        acc[0] = fma(y[0], f[0], acc[0]);
      } else {
        acc[0] = fma(y[0], f[0], fma(-y[1], f[1], acc[0]));
        acc[1] = fma(y[0], f[1], fma(y[1], f[0], acc[1]));
      }
    }
    st<PL>(out + (row * ldm + c) * PL, acc);
  }
}

// A: M (r x r, pitch ldm elements) with the nrows rows of Y below it; buf0, buf1: as many rows each.  far: this thread saw an
// element of M - 1 beyond kNearNorm / r.  The rows become Y L^{-dagger}, or Y L with times_l; status (may be null)
// |= 1 on a non-positive pivot.  Ends with a barrier.
template <int PL>
__device__ __forceinline__ void chol_rows(double* A, int r, int ldm, int nrows, double* buf0, double* buf1, bool times_l, bool far,
                                          int* status) {
  constexpr int NB = Panel<PL>::NB;
  const int tid = threadIdx.x;
  double* Yc = A + r * ldm * PL;
  if (!__syncthreads_or(far)) {
    for (int i = tid; i < r; i += THREADS) A[(i * ldm + i) * PL] -= 1.0;
    __syncthreads();
    rows_times<PL, false>(Yc, A, r, ldm, nrows, buf0);
    __syncthreads();
    rows_times<PL, false>(buf0, A, r, ldm, nrows, buf1);
    __syncthreads();
    const double c1 = times_l ? 0.5 : -0.5, c2 = times_l ? -0.125 : 0.375;
    for (int e = tid; e < nrows * r; e += THREADS) {
      const int at = (e / r * ldm + e % r) * PL;
#pragma unroll
      for (int p = 0; p < PL; ++p) Yc[at + p] += c1 * buf0[at + p] + c2 * buf1[at + p];
    }
    __syncthreads();
    return;
  }
  const int bottom = times_l ? r : r + nrows;  // rows that are eliminated
  const int ty = tid >> 4, tx = tid & 15;
  for (int j0 = 0; j0 < r; j0 += NB) {
    const int nb = min(NB, r - j0), j1 = j0 + nb;
    // the panel's diagonal block, lower triangle; the unit matrix where the last panel is narrower
    double D[NB][NB][PL], inv[NB];
#pragma unroll
    for (int i = 0; i < NB; ++i)
#pragma unroll
      for (int k = 0; k <= i; ++k) {
        if (i < nb) {
          ld<PL>(D[i][k], A + ((j0 + i) * ldm + j0 + k) * PL);
        } else {
#pragma unroll
          for (int p = 0; p < PL; ++p) D[i][k][p] = i == k && p == 0 ? 1.0 : 0.0;
        }
      }
    bool bad = false;
#pragma unroll
    for (int j = 0; j < NB; ++j) {
      double d = D[j][j][0];
      if (!(d > 0.0)) {
        bad = true;
        d = 1e-300;
      }
      inv[j] = rsqrt(d);
      D[j][j][0] = d * inv[j];
      if (PL == 2) D[j][j][PL - 1] = 0.0;
#pragma unroll
      for (int i = j + 1; i < NB; ++i)
#pragma unroll
        for (int p = 0; p < PL; ++p) D[i][j][p] *= inv[j];
#pragma unroll
      for (int i = j + 1; i < NB; ++i)
#pragma unroll
        for (int k = j + 1; k <= i; ++k) sub_conj<PL>(D[i][k], D[i][j], D[k][j]);
    }
    if (bad && tid == 0 && status) atomicOr(status, 1);
    // the rows below, one thread each: v L^{-dagger}
    for (int i = j1 + tid; i < bottom; i += THREADS) {
      double v[NB][PL];
      double* row = A + (i * ldm + j0) * PL;
#pragma unroll
      for (int j = 0; j < NB; ++j) {
        if (j < nb) {
          ld<PL>(v[j], row + j * PL);
#pragma unroll
          for (int k = 0; k < j; ++k) sub_conj<PL>(v[j], v[k], D[j][k]);
#pragma unroll
          for (int p = 0; p < PL; ++p) v[j][p] *= inv[j];
          st<PL>(row + j * PL, v[j]);
        }
      }
    }
    __syncthreads();
    if (tid == 0) {  // everyone has read the diagonal block
#pragma unroll
      for (int i = 0; i < NB; ++i)
#pragma unroll
        for (int k = 0; k <= i; ++k)
          if (i < nb) st<PL>(A + ((j0 + i) * ldm + j0 + k) * PL, D[i][k]);
    }
    // trailing update (a full panel: after a narrow one nothing is left): rows i and i + 16, columns k <= i
    for (int i = j1 + ty; i < bottom; i += 32) {
      const int i2 = i + 16;
      const bool two = i2 < bottom;
      double a[NB][PL], b[NB][PL];
#pragma unroll
      for (int t = 0; t < NB; ++t) {
        ld<PL>(a[t], A + (i * ldm + j0 + t) * PL);
        if (two) ld<PL>(b[t], A + (i2 * ldm + j0 + t) * PL);
      }
      const int last = min(two ? i2 : i, r - 1), end1 = min(i, r - 1);
      for (int k = j1 + tx; k <= last; k += 16) {
        double* p1 = A + (i * ldm + k) * PL;
        double* p2 = A + (i2 * ldm + k) * PL;
        double x[PL] = {}, y[PL] = {};
        if (k <= end1) ld<PL>(x, p1);
        if (two) ld<PL>(y, p2);
        const double* col = A + (k * ldm + j0) * PL;
#pragma unroll
        for (int t = 0; t < NB; ++t) {
          double c[PL];
          ld<PL>(c, col + t * PL);
          sub_conj<PL>(x, a[t], c);
          if (two) sub_conj<PL>(y, b[t], c);
        }
        if (k <= end1) st<PL>(p1, x);
        if (two) st<PL>(p2, y);
      }
    }
    __syncthreads();
  }
  if (times_l) {
    rows_times<PL, true>(Yc, A, r, ldm, nrows, buf0);
    __syncthreads();
    for (int e = tid; e < nrows * r; e += THREADS) {
      const int at = (e / r * ldm + e % r) * PL;
#pragma unroll
      for (int p = 0; p < PL; ++p) Yc[at + p] = buf0[at + p];
    }
    __syncthreads();
  }
}

}  // namespace cholr
}  // namespace rr
