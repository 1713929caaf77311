// The occupied-orbital recovery of recovery.cu in one launch, for matrices that fit one CTA's shared memory four at a
// time (n <= 79 real, 56 complex): the same steps in the same order, on plain FP64 FMA tiles.
//
// What it replaces is a chain of 17 - 25 launches of 2 - 6 us each with 2 - 4 us between them, none of which has work for
// more than a few SMs at these sizes.  Bound here: one SM's FP64 pipe (64 FMA per cycle; a 64 x 64 x 64 real product takes
// 4.1 k of them) and, below n of about 30, barriers and latencies.  Whole Fock builds on device arrays, the launches / this
// kernel, us: real n = 12 158 / 96, 24 177 / 108, 48 225 / 138, 64 191 / 145, 72 190 / 173, 84 212 / 215; X2C nl = 12 199 / 155,
// 24 217 / 205, 29 242 / 240; four components nl = 10 315 / 280.  The limit of 200 KB lies where the two meet.
#include <algorithm>
#include <cmath>

#include "chol_rows.cuh"
#include "ri_store.cuh"

namespace rr {

namespace {

using namespace cholr;

constexpr int kMaxSmem = 200 * 1024;

enum : int { kOk = 0, kNotConverged = 1, kNoRoom = 2 };

// Pitch (elements) of the square buffers: odd, so that a column spreads over the banks.
__host__ __device__ inline int64_t small_pitch(int64_t n, int64_t n_eff) { return (n > n_eff ? n : n_eff) | 1; }

// Strides (elements) of a stored matrix as a factor: (row, column) = row * r + column * c; conj: its conjugate.
struct Factor {
  const double* p;
  int r, c;
  bool conj;
};
__device__ __forceinline__ Factor plain(const double* p, int pitch) { return Factor{p, pitch, 1, false}; }
__device__ __forceinline__ Factor dagger(const double* p, int pitch) { return Factor{p, 1, pitch, true}; }

// C (pitch ldc) = alpha A B for A of M x K, B of K x N.  4 x 4 (complex 2 x 2) outputs a thread, columns a stride apart so
// that a warp reads consecutive ones.  Inlined into each use: as one shared copy, with generic
// loads and run-time strides, the kernel took 30 us instead of 24 at n = 24 and a quarter longer at n = 64.
template <int PL>
__device__ __forceinline__ void product(int M, int N, int K, const Factor A, const Factor B, double alpha, double* C, int64_t ldc) {
  constexpr int TM = PL == 1 ? 4 : 2, TN = TM;
  const int ntm = (M + TM - 1) / TM, ntn = (N + TN - 1) / TN;
  const double sa = A.conj ? -1.0 : 1.0, sb = B.conj ? -1.0 : 1.0;
  for (int tile = threadIdx.x; tile < ntm * ntn; tile += THREADS) {
    const int tm = tile / ntn, tn = tile - tm * ntn;
    const double *pa[TM], *pb[TN];
#pragma unroll
    for (int i = 0; i < TM; ++i) pa[i] = A.p + min(tm * TM + i, M - 1) * A.r * PL;
#pragma unroll
    for (int j = 0; j < TN; ++j) pb[j] = B.p + min(tn + j * ntn, N - 1) * B.c * PL;
    double acc[TM][TN][PL] = {};
#pragma unroll 2
    for (int k = 0; k < K; ++k) {
      double a[TM][PL], b[TN][PL];
#pragma unroll
      for (int i = 0; i < TM; ++i) ld<PL>(a[i], pa[i] + k * A.c * PL);
#pragma unroll
      for (int j = 0; j < TN; ++j) ld<PL>(b[j], pb[j] + k * B.r * PL);
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) {
          if constexpr (PL == 1) {
            acc[i][j][0] = fma(a[i][0], b[j][0], acc[i][j][0]);
          } else {
            const double ai = sa * a[i][PL - 1], bi = sb * b[j][PL - 1];
            acc[i][j][0] = fma(a[i][0], b[j][0], fma(-ai, bi, acc[i][j][0]));
            acc[i][j][PL - 1] = fma(a[i][0], bi, fma(ai, b[j][0], acc[i][j][PL - 1]));
          }
        }
    }
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < TN; ++j)
        if (tm * TM + i < M && tn + j * ntn < N) {
#pragma unroll
          for (int q = 0; q < PL; ++q) C[((tm * TM + i) * ldc + tn + j * ntn) * PL + q] = alpha * acc[i][j][q];
        }
  }
  __syncthreads();
}

// rows x cols of a packed global matrix into pitch ldp.
template <int PL>
__device__ __forceinline__ void stage(double* dst, const double* src, int rows, int cols, int ldp) {
  for (int e = threadIdx.x; e < rows * cols; e += THREADS) {
    const int i = e / cols, j = e - i * cols;
    double v[PL];
#pragma unroll
    for (int p = 0; p < PL; ++p) v[p] = src[static_cast<int64_t>(e) * PL + p];  // a caller's complex array may be 8-byte aligned
    st<PL>(dst + (i * ldp + j) * PL, v);
  }
}

__device__ __forceinline__ double block_reduce(double v, bool max_of, double* red) {
  for (int o = 16; o > 0; o >>= 1) {
    const double w = __shfl_xor_sync(0xffffffffu, v, o);
    v = max_of ? fmax(v, w) : v + w;
  }
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  v = red[0];
  for (int w = 1; w < THREADS / 32; ++w) v = max_of ? fmax(v, red[w]) : v + red[w];
  return v;
}

// Entry idx of the fixed pseudo-random test matrix (fill_test_matrix_kernel of recovery.cu).
__device__ __forceinline__ double test_entry(int64_t idx) {
  uint64_t z = static_cast<uint64_t>(idx) + 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  z ^= z >> 31;
  return static_cast<double>(z >> 11) * (2.0 / 9007199254740992.0) - 1.0;
}

// ct (r x n) = F^dagger X^dagger of recovery.cu; result[0] = r, result[1] = kOk, kNotConverged or kNoRoom (r too
// large a part of n_eff for the shared memory: nothing written).
template <int PL>
__global__ void __launch_bounds__(THREADS, 1) recover_small_kernel(const double* X, const double* S, const double* D, int n, int n_eff,
                                                                   double scale, int weighted, double* ct, int* result, int* status) {
  extern __shared__ __align__(16) double sm[];
  __shared__ double red[THREADS / 32];
  const int ldp = static_cast<int>(small_pitch(n, n_eff)), cap = max(n, n_eff) * ldp * PL, tid = threadIdx.x;
  double *b0 = sm, *b1 = sm + cap, *b2 = b1 + cap, *b3 = b2 + cap;

  // P_eff = Z^dagger D Z scale, Z = S X
  stage<PL>(b0, S, n, n, ldp);
  stage<PL>(b1, X, n, n_eff, ldp);
  __syncthreads();
  product<PL>(n, n_eff, n, plain(b0, ldp), plain(b1, ldp), 1.0, b2, ldp);
  stage<PL>(b0, D, n, n, ldp);
  __syncthreads();
  product<PL>(n, n_eff, n, plain(b0, ldp), plain(b2, ldp), 1.0, b3, ldp);
  product<PL>(n_eff, n_eff, n, dagger(b2, ldp), plain(b3, ldp), scale, b0, ldp);
  for (int e = tid; e < n_eff * n_eff; e += THREADS) {
    const int i = e / n_eff, j = e - i * n_eff, at = (i * ldp + j) * PL;
    b1[at] = 2.0 * b0[at] - (i == j ? 1.0 : 0.0);
    if (PL == 2) b1[at + PL - 1] = 2.0 * b0[at + PL - 1];
  }
  __syncthreads();

  // Newton-Schulz sign iteration: A in b1, A^2 in b2
  double trace = 0.0;
  bool converged = false;
  for (int it = 0; it < 100; ++it) {
    product<PL>(n_eff, n_eff, n_eff, plain(b1, ldp), plain(b1, ldp), 1.0, b2, ldp);
    double off = 0.0, rows = 0.0, tr = 0.0;
    for (int i = tid >> 5; i < n_eff; i += THREADS / 32) {
      double rs = 0.0;
      for (int j = tid & 31; j < n_eff; j += 32) {
        const double re = b2[(i * ldp + j) * PL], im = PL == 2 ? b2[(i * ldp + j) * PL + PL - 1] : 0.0;
        const double d = re - (i == j ? 1.0 : 0.0);
        off = fmax(off, PL == 2 ? sqrt(d * d + im * im) : fabs(d));
        rs += PL == 2 ? sqrt(re * re + im * im) : fabs(re);
        if (i == j) tr += b1[(i * ldp + j) * PL];
      }
      for (int o = 16; o > 0; o >>= 1) rs += __shfl_xor_sync(0xffffffffu, rs, o);
      rows = fmax(rows, rs);
    }
    off = block_reduce(off, true, red);
    rows = block_reduce(rows, true, red);
    trace = block_reduce(tr, false, red);
    if (it == 0 && rows > 2.5) {  // ||A||_2 <= sqrt(||A^2||_inf): into the convergence region
      const double f = 1.0 / sqrt(rows);
      for (int e = tid; e < n_eff * n_eff; e += THREADS) {
        double* p = b1 + (e / n_eff * ldp + e % n_eff) * PL;
#pragma unroll
        for (int q = 0; q < PL; ++q) p[q] *= f;
      }
      __syncthreads();
      continue;
    }
    if (off < 1e-13) {
      converged = true;
      break;
    }
    product<PL>(n_eff, n_eff, n_eff, plain(b1, ldp), plain(b2, ldp), 1.0, b3, ldp);
    for (int e = tid; e < n_eff * n_eff; e += THREADS) {
      const int at = (e / n_eff * ldp + e % n_eff) * PL;
#pragma unroll
      for (int q = 0; q < PL; ++q) b1[at + q] = 1.5 * b1[at + q] - 0.5 * b3[at + q];
    }
    __syncthreads();
    if (off < 1e-10) {
      converged = true;
      break;
    }
  }
  const double half = rint(0.5 * (n_eff + trace));
  const int r = converged ? static_cast<int>(fmax(0.0, fmin(static_cast<double>(n_eff), half))) : 0;
  const int ldr = r | 1;
  const bool room = static_cast<int64_t>(r + 3 * n_eff) * ldr * PL <= 2 * static_cast<int64_t>(cap);
  if (tid == 0) {
    result[0] = r;
    result[1] = !converged ? kNotConverged : !room ? kNoRoom : kOk;
  }
  if (r == 0 || !room) return;

  // CholeskyQR2 of Y = Pi G, Pi = (1 + A) / 2
  double *M = b2, *Y = M + r * ldr * PL, *w0 = Y + n_eff * ldr * PL, *w1 = w0 + n_eff * ldr * PL;
  for (int e = tid; e < n_eff * n_eff; e += THREADS) {
    const int i = e / n_eff, j = e - i * n_eff;
    double* p = b1 + (i * ldp + j) * PL;
    p[0] = 0.5 * (p[0] + (i == j ? 1.0 : 0.0));
    if (PL == 2) p[PL - 1] *= 0.5;
  }
  for (int e = tid; e < n_eff * r; e += THREADS) {
#pragma unroll
    for (int q = 0; q < PL; ++q) w0[(e / r * ldr + e % r) * PL + q] = test_entry(static_cast<int64_t>(e) * PL + q);
  }
  __syncthreads();
  product<PL>(n_eff, r, n_eff, plain(b1, ldp), plain(w0, ldr), 1.0, Y, ldr);
  const double near = kNearNorm / r;
  for (int pass = 0; pass < (weighted ? 3 : 2); ++pass) {
    if (pass == 2) product<PL>(n_eff, r, n_eff, plain(b0, ldp), plain(Y, ldr), 1.0, w0, ldr);  // F = Q (Q^dagger P_eff Q)^{1/2}
    product<PL>(r, r, n_eff, dagger(Y, ldr), plain(pass == 2 ? w0 : Y, ldr), 1.0, M, ldr);
    bool far = false;
    for (int e = tid; e < r * r; e += THREADS) {
      double v[PL];
      ld<PL>(v, M + (e / r * ldr + e % r) * PL);
      far |= !(fabs(v[0] - (e / r == e % r ? 1.0 : 0.0)) <= near);
      if (PL == 2) far |= !(fabs(v[PL - 1]) <= near);
    }
    chol_rows<PL>(M, r, ldr, n_eff, w0, w1, pass == 2, far, status);
  }
  stage<PL>(b0, X, n, n_eff, ldp);
  __syncthreads();
  product<PL>(r, n, n_eff, dagger(Y, ldr), dagger(b0, ldp), 1.0, ct, n);
}

}  // namespace

bool recover_small_fits(int64_t n, int64_t n_eff, bool cplx) {
  if (n > 256 || n_eff > 256) return false;
  return static_cast<int64_t>(sizeof(double)) * 4 * std::max(n, n_eff) * small_pitch(n, n_eff) * (cplx ? 2 : 1) <= kMaxSmem;
}

void recover_small_launch(rr_ri_store* h, const double* X, const double* S, const double* D, int64_t n, int64_t n_eff, double scale,
                          bool cplx, bool weighted, double* ct, cudaStream_t s) {
  const int64_t smem = static_cast<int64_t>(sizeof(double)) * 4 * std::max(n, n_eff) * small_pitch(n, n_eff) * (cplx ? 2 : 1);
  static std::atomic<bool> attr[kMaxDevices];
  once_per_device(attr, [] {
    RR_CUDA(cudaFuncSetAttribute(recover_small_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmem));
    RR_CUDA(cudaFuncSetAttribute(recover_small_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmem));
  });
  h->solver_a.ensure(32);
  auto k = cplx ? recover_small_kernel<2> : recover_small_kernel<1>;
  k<<<1, THREADS, smem, s>>>(X, S, D, static_cast<int>(n), static_cast<int>(n_eff), scale, weighted, ct,
                             reinterpret_cast<int*>(h->solver_a.p), h->status.p + 1);
  RR_LAUNCH_CHECK();
}

bool recover_small_finish(rr_ri_store* h, cudaStream_t s, int64_t* r) {
  int got[2] = {0, 0};
  RR_CUDA(cudaMemcpyAsync(got, h->solver_a.p, sizeof(got), cudaMemcpyDeviceToHost, s));
  host_wait(h, s);
  if (got[1] == kNoRoom) return false;
  RR_REQUIRE(got[1] == kOk, RR_ERR_SOLVER,
             "occupied recovery: an eigenvalue of X^dagger(SPS)X sits at the 0.5 threshold (sign iteration did not converge)");
  *r = got[0];
  return true;
}

}  // namespace rr
