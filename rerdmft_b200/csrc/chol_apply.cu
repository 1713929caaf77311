// Y L^{-dagger} or Y L for the Cholesky factor L of a small Gram matrix M = L L^dagger, in one launch (the CholeskyQR steps
// of the occupied-orbital recovery): every CTA loads M, factors it and applies the factor to its own few rows of Y
// (chol_rows.cuh).  The factorisation is a serial chain that one SM has to walk in any case, so walking it on all SMs
// costs nothing.
//
// X2C, r = 80, 400 rows: 44 us against 171 + 8 us for the one-CTA factor with inverse and the product with it, 17 us near
// the identity; real, r = 40, 400 rows: 13 and 11 us against 48 + 16.
#include <algorithm>

#include "chol.cuh"
#include "chol_rows.cuh"

namespace rr {

namespace {

using namespace cholr;

constexpr int kMaxSmem = 227 * 1024;

// Shared memory: M (r x r), the CTA's rows of Y and two buffers of as many rows, pitch ldm = r | 1 elements (a
// column spreads over all banks).
template <int PL>
__global__ void __launch_bounds__(THREADS, 1) chol_apply_kernel(const double* M, int r, const double* Y, int64_t n, int rows,
                                                                int times_l, double* out, int* status) {
  extern __shared__ __align__(16) double A[];
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
  chol_rows<PL>(A, r, ldm, nrows, buf0, buf1, times_l != 0, far, blockIdx.x == 0 ? status : nullptr);
  for (int e = tid; e < nrows * r; e += THREADS) {
    const int row = e / r, c = e - row * r;
    double v[PL];
    ld<PL>(v, Yc + (row * ldm + c) * PL);
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
