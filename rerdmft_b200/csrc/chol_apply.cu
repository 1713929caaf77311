// Y L^{-dagger} or Y L for the Cholesky factor L of a small Gram matrix M = L L^dagger, in one launch
// (the CholeskyQR steps of the occupied-orbital recovery).
//
// Every CTA loads M, factors it and applies the factor to its own few rows of Y: the factorisation is a serial
// chain that one SM has to walk in any case, so walking it on all SMs costs nothing, and neither the inverse
// factor nor a product with it are needed.  Y's rows stand below M's in shared memory and are eliminated along
// with them: what the elimination leaves of a row y is y L^{-dagger}.
//
// Bound: that chain (X2C, r = 80, 400 rows: 44 us against 171 + 8 us for the one-CTA factor with inverse and the product
// with it, 17 us near the identity; real, r = 40, 400 rows: 13 and 11 us against 48 + 16).  A panel of NB columns (8 real, 4 complex) costs every thread the factorisation of
// the panel's diagonal block, done redundantly in registers without a barrier, then one row of the panel, then a
// rank-NB update of the trailing part with two rows a thread: 2 barriers per NB columns.
//
// Where M is near the identity (the second CholeskyQR pass; the weights of an idempotent density) the symmetric
// factors M^{-1/2} and M^{1/2} take the place of the triangular ones: with E = M - 1 the series
// 1 - E/2 + 3/8 E^2 and 1 + E/2 - E^2/8, whose next terms 5/16 E^3 and 1/16 E^3 are below 2e-17 for
// ||E||_inf <= kNearNorm.  Two products of the CTA's rows with E replace the chain.
#include <algorithm>

#include "chol.cuh"

namespace rr {

namespace {

constexpr int THREADS = 256;
constexpr int kMaxSmem = 227 * 1024;
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

// Shared memory: M (r x r), the CTA's rows of Y and two buffers of as many rows, pitch ldm = r | 1 elements (a
// column spreads over all banks).
template <int PL>
__global__ void __launch_bounds__(THREADS, 1) chol_apply_kernel(const double* M, int r, const double* Y, int64_t n, int rows,
                                                                int times_l, double* out, int* status) {
  extern __shared__ __align__(16) double A[];
  constexpr int NB = Panel<PL>::NB;
  const int ldm = r | 1, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  double* Yc = A + static_cast<int64_t>(r) * ldm * PL;
  double* buf0 = Yc + rows * ldm * PL;
  double* buf1 = buf0 + rows * ldm * PL;
  const int64_t row0 = static_cast<int64_t>(blockIdx.x) * rows;
  const int nrows = static_cast<int>(min(static_cast<int64_t>(rows), n - row0));

  const double near = kNearNorm / r;
  bool far = false;
  for (int i = warp; i < r + nrows; i += THREADS / 32) {
    const double* src = i < r ? M + static_cast<int64_t>(i) * r * PL : Y + (row0 + i - r) * r * PL;
#pragma unroll 4
    for (int k = lane; k < r; k += 32) {
      double v[PL];
      ld<PL>(v, src + k * PL);
      st<PL>(A + (i * ldm + k) * PL, v);
      if (i < r) {
        far |= !(fabs(v[0] - (i == k ? 1.0 : 0.0)) <= near);
        if (PL == 2) far |= !(fabs(v[PL - 1]) <= near);
      }
    }
  }
  if (!__syncthreads_or(far)) {
    for (int i = tid; i < r; i += THREADS) A[(i * ldm + i) * PL] -= 1.0;
    __syncthreads();
    rows_times<PL, false>(Yc, A, r, ldm, nrows, buf0);
    __syncthreads();
    rows_times<PL, false>(buf0, A, r, ldm, nrows, buf1);
    __syncthreads();
    const double c1 = times_l ? 0.5 : -0.5, c2 = times_l ? -0.125 : 0.375;
    for (int e = tid; e < nrows * r; e += THREADS) {
      const int row = e / r, c = e - row * r, at = (row * ldm + c) * PL;
      double v[PL];
#pragma unroll
      for (int p = 0; p < PL; ++p) v[p] = Yc[at + p] + (c1 * buf0[at + p] + c2 * buf1[at + p]);
      st<PL>(out + ((row0 + row) * r + c) * PL, v);
    }
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
    if (bad && tid == 0 && blockIdx.x == 0) atomicOr(status, 1);
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
  const double* res = Yc;
  if (times_l) {
    rows_times<PL, true>(Yc, A, r, ldm, nrows, buf0);
    __syncthreads();
    res = buf0;
  }
  for (int e = tid; e < nrows * r; e += THREADS) {
    const int row = e / r, c = e - row * r;
    double v[PL];
    ld<PL>(v, res + (row * ldm + c) * PL);
    st<PL>(out + ((row0 + row) * r + c) * PL, v);
  }
}

}  // namespace

bool chol_apply(const double* M, int64_t r, const double* Y, int64_t n, bool cplx, bool times_l, double* out, int* status,
                cudaStream_t s) {
  if (r <= 0 || n <= 0) return true;
  const int PL = cplx ? 2 : 1;
  const int64_t rows = (n + sm_count_current() - 1) / sm_count_current();
  const int64_t smem = static_cast<int64_t>(sizeof(double)) * PL * (r | 1) * (r + 3 * rows);
  if (smem > kMaxSmem) return false;
  static std::atomic<bool> attr[kMaxDevices];
  once_per_device(attr, [] {
    RR_CUDA(cudaFuncSetAttribute(chol_apply_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmem));
    RR_CUDA(cudaFuncSetAttribute(chol_apply_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmem));
  });
  const unsigned grid = static_cast<unsigned>((n + rows - 1) / rows);
  if (cplx)
    chol_apply_kernel<2><<<grid, THREADS, smem, s>>>(M, static_cast<int>(r), Y, n, static_cast<int>(rows), times_l, out, status);
  else
    chol_apply_kernel<1><<<grid, THREADS, smem, s>>>(M, static_cast<int>(r), Y, n, static_cast<int>(rows), times_l, out, status);
  RR_LAUNCH_CHECK();
  return true;
}

}  // namespace rr
