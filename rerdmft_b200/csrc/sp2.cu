// The density step's purification in two launches instead of about eighty.
//
// sp2_kernel: all SP2 steps in one cooperative launch.  A step of an n x n matrix is one product X X (16 x 16 tiles of the
// upper triangle dealt out to the CTAs, FP64 mma.sync m8n8k4: tcgen05 has no FP64 kind) whose epilogue applies the step and writes both triangles,
// then one grid barrier.  X is Hermitian, so both operands of a tile are rows of X.  The choice between X^2 and
// 2 X - X^2 needs tr X and tr X^2 = ||X||_F^2 of the matrix being squared, which its writers left as per-tile
// partials: every CTA adds all of them in the same order and comes to the same choice.
// Bound: latency (the barrier, one L2 round trip for the rows, a chain of n / 8 mma).  n = 160: 4.4 us a step
// against 15 us for product, split-K reduction and step kernel, and no host check every fourth step.
//
// ritz_kernel: the extreme eigenvalues of a 32 x 32 generalized problem on one CTA: Cholesky reduction
// (chol_rows.cuh), Householder tridiagonalisation by one warp (only the moduli of the off-diagonals matter), multisection on Sturm
// counts (Barth, Martin, Wilkinson, "Calculation of the eigenvalues of a symmetric tridiagonal matrix by the method of bisection",
// Numer. Math. 9, 1967), 32 points a pass, one warp for either end.  80 us (n = 160, real) against 320 us for the library's sygvd.
#include <algorithm>
#include <vector>

#include "chol_rows.cuh"
#include "sp2.cuh"

namespace rr {

namespace {

constexpr int TILE = 16, SP2_THREADS = 256;
constexpr int kSp2Smem = 200 * 1024;
constexpr int kMaxTiles = (kSp2MaxReal / TILE) * (kSp2MaxReal / TILE + 1) / 2;
constexpr int kMaxGroupCtas = 1184;  // of one launch
constexpr unsigned kBarrierPolls = 1u << 21;  // about a second

struct Sp2Args {
  const double* F;
  const double* b;
  double *X, *Y;
  double* part;       // two sets of (tr, fro) per tile
  unsigned* bar;      // zeroed counter, expiry flag
  double* outcome;
  double nocc;
  int n, kc, max_steps, sure;
};

// All CTAs past their k-th arrival; false after kBarrierPolls polls of any CTA.
__device__ __forceinline__ bool grid_barrier(unsigned* bar, unsigned target, int* ok) {
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    atomicAdd(bar, 1u);
    unsigned seen = 0, polls = 0;
    bool good = true;
    do {
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(bar) : "memory");
      if (++polls > kBarrierPolls || (polls % 1024 == 0 && *reinterpret_cast<volatile unsigned*>(bar + 1))) {
        good = false;
        break;
      }
    } while (seen < target);
    if (!good) atomicExch(bar + 1, 1u);
    __threadfence();
    *ok = good;
  }
  __syncthreads();
  return *ok != 0;
}

__device__ __forceinline__ void dmma(double (&c)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n" : "+d"(c[0]), "+d"(c[1]) : "d"(a), "d"(b));
}

// Tile (i0, j0) of X X^dagger: rows i0 .. and j0 .. of X staged kc columns at a time (pitch kc + 4: 8 rows x 4 columns of a
// fragment spread over the banks), planes (re, im) apart.  Warp w: 8 x 8 sub-tile w & 3, half w >> 2 of each chunk; the
// halves are added through `red`.  out[16][17][PL] in shared memory.
template <int PL>
__device__ __forceinline__ void square_tile(const double* X, int n, int kc, int i0, int j0, double* sm, double* red, double* out) {
  const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31, pitch = kc + 4;
  const int sr = (w & 1) * 8, sc = ((w >> 1) & 1) * 8, half = w >> 2;
  double* sa = sm;
  double* sb = sm + PL * TILE * pitch;
  double re[2][2] = {}, im[2][2] = {};
  for (int k0 = 0; k0 < n; k0 += kc) {
    const int kn = min(kc, n - k0), kp = (kn + 7) / 8 * 8;
    __syncthreads();
    // warp w: rows w and w + 8 of either operand, four rows' loads in flight for each of its columns
    constexpr int NW = SP2_THREADS / 32, NROW = 2 * TILE / NW;
    const double* src[NROW];
    double* dst[NROW];
    bool live[NROW];
#pragma unroll
    for (int q = 0; q < NROW; ++q) {
      const int r = w + NW * q, row = r < TILE ? i0 + r : j0 + r - TILE;
      live[q] = row < n;
      dst[q] = (r < TILE ? sa : sb) + (r % TILE) * pitch;
      src[q] = X + (static_cast<int64_t>(live[q] ? row : 0) * n + k0) * PL;
    }
#pragma unroll 4
    for (int k = lane; k < kp; k += 32) {
      double v[NROW][PL];
#pragma unroll
      for (int q = 0; q < NROW; ++q) {
        const bool in = live[q] && k < kn;
        if constexpr (PL == 1) {
          v[q][0] = in ? src[q][k] : 0.0;
        } else {
          const double2 d = in ? *reinterpret_cast<const double2*>(src[q] + 2 * k) : make_double2(0.0, 0.0);
          v[q][0] = d.x;
          v[q][PL - 1] = d.y;
        }
      }
#pragma unroll
      for (int q = 0; q < NROW; ++q) {
        dst[q][k] = v[q][0];
        if (PL == 2) dst[q][TILE * pitch + k] = v[q][PL - 1];
      }
    }
    __syncthreads();
    const double* a = sa + (sr + (lane >> 2)) * pitch + (lane & 3);
    const double* b = sb + (sc + (lane >> 2)) * pitch + (lane & 3);
    const int steps = kp / 8;  // pairs of 4 columns: this warp's half of each pair
    auto mac = [&](int t, double (&r0)[2], double (&r1)[2]) {
      const int k = t * 8 + half * 4;
      if constexpr (PL == 1) {
        dmma(r0, a[k], b[k]);
      } else {  // x conj(y)
        const double ar = a[k], ai = a[TILE * pitch + k], br = b[k], bi = b[TILE * pitch + k];
        dmma(r0, ar, br);
        dmma(r1, ai, bi);
        dmma(im[0], ai, br);
        dmma(im[1], -ar, bi);
      }
    };
#pragma unroll 2
    for (int t = 0; t + 1 < steps; t += 2) {  // two chains of sums
      mac(t, re[0], re[1]);
      mac(t + 1, re[1], re[0]);
    }
    if (steps & 1) mac(steps - 1, re[0], re[1]);
  }
  const int r = sr + (lane >> 2), c = sc + 2 * (lane & 3);
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    re[0][q] += re[1][q];
    im[0][q] += im[1][q];
  }
  if (half) {
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      red[(r * 17 + c + q) * PL] = re[0][q];
      if (PL == 2) red[(r * 17 + c + q) * PL + PL - 1] = im[0][q];
    }
  }
  __syncthreads();
  if (!half) {
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      out[(r * 17 + c + q) * PL] = re[0][q] + red[(r * 17 + c + q) * PL];
      if (PL == 2) out[(r * 17 + c + q) * PL + PL - 1] = im[0][q] + red[(r * 17 + c + q) * PL + PL - 1];
    }
  }
  __syncthreads();
}

// (a, b) summed over the CTA, in every thread.
__device__ __forceinline__ void cta_sum2(double& a, double& b, double* red) {
  for (int o = 16; o > 0; o >>= 1) {
    a += __shfl_xor_sync(0xffffffffu, a, o);
    b += __shfl_xor_sync(0xffffffffu, b, o);
  }
  __syncthreads();
  if ((threadIdx.x & 31) == 0) {
    red[2 * (threadIdx.x >> 5)] = a;
    red[2 * (threadIdx.x >> 5) + 1] = b;
  }
  __syncthreads();
  a = red[0];
  b = red[1];
  for (int w = 1; w < SP2_THREADS / 32; ++w) {
    a += red[2 * w];
    b += red[2 * w + 1];
  }
}

// Upper-triangle tile t of nt x nt.
__device__ __forceinline__ void tile_at(int t, int nt, int& i0, int& j0) {
  int ti = 0;
  while (t >= nt - ti) {
    t -= nt - ti;
    ++ti;
  }
  i0 = ti * TILE;
  j0 = (ti + t) * TILE;
}

// X is indexed by element (i n + j) PL; Hermitian to the last bit (both triangles are written from one value).
template <int PL>
__device__ __forceinline__ void sp2_body(const Sp2Args& g, int me, int ctas, double* sm) {
  __shared__ double red[TILE * 17 * PL], tile[TILE * 17 * PL], sums[2 * SP2_THREADS / 32];
  __shared__ int ok;
  const int n = g.n, tid = threadIdx.x, nt = (n + TILE - 1) / TILE, tiles = nt * (nt + 1) / 2;
  unsigned arrivals = 0;
  double* part[2] = {g.part, g.part + 2 * kMaxTiles};  // (tr, ||.||_F^2) per tile: the sums do not depend on ctas

  // X = (hi - F) / (hi - lo), upper triangle and its mirror
  {
    const double lo = g.b[0], hi = g.b[1], inv = 1.0 / fmax(hi - lo, 1e-300);
    for (int t = me; t < tiles; t += ctas) {
      int i0, j0;
      tile_at(t, nt, i0, j0);
      const int i = i0 + tid / TILE, j = j0 + tid % TILE;
      double tr = 0.0, fro = 0.0;
      if (i < n && j < n && i <= j) {
        const int64_t e = static_cast<int64_t>(i) * n + j, m = static_cast<int64_t>(j) * n + i;
        const double re = ((i == j ? hi : 0.0) - g.F[e * PL]) * inv, im = PL == 2 && i != j ? -g.F[e * PL + PL - 1] * inv : 0.0;
        g.X[e * PL] = re;
        g.X[m * PL] = re;
        if (PL == 2) {
          g.X[e * PL + PL - 1] = im;
          g.X[m * PL + PL - 1] = -im;
        }
        fro = (i == j ? 1.0 : 2.0) * (re * re + im * im);
        if (i == j) tr = re;
      }
      cta_sum2(tr, fro, sums);
      if (tid == 0) {
        part[0][2 * t] = tr;
        part[0][2 * t + 1] = fro;
      }
    }
  }
  if (!grid_barrier(g.bar, arrivals += ctas, &ok)) {
    if (me == 0 && tid == 0) g.outcome[0] = 2.0;
    return;
  }

  const double tol = fmax(1.0, g.nocc);
  double *cur = g.X, *nxt = g.Y;
  double result = 1.0, t1 = 0.0, t2 = 0.0;
  int step = 0;
  for (; step < g.max_steps; ++step) {
    // tr X and tr X^2 of the matrix about to be squared
    const volatile double* pin = part[step & 1];
    t1 = t2 = 0.0;
    for (int i = tid; i < tiles; i += SP2_THREADS) {
      t1 += pin[2 * i];
      t2 += pin[2 * i + 1];
    }
    cta_sum2(t1, t2, sums);
    const bool square = fabs(t2 - g.nocc) < fabs(2.0 * t1 - t2 - g.nocc);
    for (int t = me; t < tiles; t += ctas) {
      int i0, j0;
      tile_at(t, nt, i0, j0);
      double tr = 0.0, fro = 0.0;
      square_tile<PL>(cur, n, g.kc, i0, j0, sm, red, tile);
      const int r = tid / TILE, c = tid % TILE, i = i0 + r, j = j0 + c;
      if (i < n && j < n && i <= j) {
        const int64_t e = (static_cast<int64_t>(i) * n + j) * PL, m = (static_cast<int64_t>(j) * n + i) * PL;
        double v[PL];
#pragma unroll
        for (int q = 0; q < PL; ++q) {
          const double x2 = tile[(r * 17 + c) * PL + q];
          v[q] = square ? x2 : 2.0 * cur[e + q] - x2;
        }
        if (PL == 2 && i == j) v[PL - 1] = 0.0;
        nxt[e] = v[0];
        nxt[m] = v[0];
        double sq = v[0] * v[0];
        if (PL == 2) {
          nxt[e + PL - 1] = v[PL - 1];
          nxt[m + PL - 1] = i == j ? 0.0 : -v[PL - 1];
          sq += v[PL - 1] * v[PL - 1];
        }
        fro = (i == j ? 1.0 : 2.0) * sq;
        if (i == j) tr = v[0];
      }
      cta_sum2(tr, fro, sums);
      if (tid == 0) {
        part[(step + 1) & 1][2 * t] = tr;
        part[(step + 1) & 1][2 * t + 1] = fro;
      }
    }
    if (!grid_barrier(g.bar, arrivals += ctas, &ok)) {
      result = 2.0;
      break;
    }
    double* x = cur;
    cur = nxt;
    nxt = x;
    // idempotency of the matrix just squared: |tr X - tr X^2| = |sum lambda (1 - lambda)|
    if (fabs(t1 - t2) < 1e-11 * tol && fabs(t1 - g.nocc) < 1e-6) {
      result = 0.0;
      break;
    }
    // every eigenvalue of X in [0, 1] makes tr X^2 <= tr X
    if (!g.sure && t2 > t1 + 1e-9 * tol) break;
  }
  if (result == 0.0 && cur != g.X) {
    const int64_t cnt = static_cast<int64_t>(n) * n * PL;
    for (int64_t e = me * static_cast<int64_t>(SP2_THREADS) + tid; e < cnt; e += static_cast<int64_t>(ctas) * SP2_THREADS) g.X[e] = cur[e];
  }
  if (me == 0 && tid == 0) {
    g.outcome[0] = result;
    g.outcome[1] = t1;
    g.outcome[2] = t2;
    g.outcome[3] = step + 1;
  }
}

template <int PL>
__global__ void __launch_bounds__(SP2_THREADS, 1) sp2_kernel(const Sp2Args g) {
  extern __shared__ __align__(16) double sm[];
  sp2_body<PL>(g, blockIdx.x, gridDim.x, sm);
}

// Independent complex problems side by side: CTA b works on problem of[b], as one of its ctas from first on.
struct Sp2Entry {
  Sp2Args a;
  int first, ctas;
};
__global__ void __launch_bounds__(SP2_THREADS, 1) sp2_group_kernel(const Sp2Entry* tab, const int* of) {
  extern __shared__ __align__(16) double sm[];
  const Sp2Entry e = tab[of[blockIdx.x]];
  sp2_body<2>(e.a, blockIdx.x - e.first, e.ctas, sm);
}

// ---------------------------------------------------------------- Ritz values

using cholr::THREADS;

template <int PL>
__global__ void __launch_bounds__(THREADS, 1) ritz_kernel(const double* T, const double* M, double* b) {
  constexpr int K = kRitz, LD = K | 1;
  extern __shared__ __align__(16) double sm[];
  __shared__ int bad;
  __shared__ double diag[K], off2[K], ends[2];
  double *A = sm, *U = A + K * LD * PL, *w0 = U + K * LD * PL, *w1 = w0 + K * LD * PL;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) bad = 0;
  // U <- T L^{-dagger}, then U <- U^dagger L^{-dagger} = (L^{-1} T L^{-dagger})^dagger
  for (int pass = 0; pass < 2; ++pass) {
    for (int e = tid; e < K * K; e += THREADS) {
      const int i = e / K, j = e % K;
#pragma unroll
      for (int q = 0; q < PL; ++q) {
        A[(i * LD + j) * PL + q] = M[e * PL + q];
        if (pass == 0) U[(i * LD + j) * PL + q] = T[e * PL + q];
        else w0[(i * LD + j) * PL + q] = (q ? -1.0 : 1.0) * U[(j * LD + i) * PL + q];
      }
    }
    __syncthreads();
    if (pass == 1) {
      for (int e = tid; e < K * LD * PL; e += THREADS) U[e] = w0[e];
      __syncthreads();
    }
    cholr::chol_rows<PL>(A, K, LD, K, w0, w1, false, true, &bad);
  }
  if (bad) return;  // (uniform: written before chol_rows' last barrier)
  if (warp == 0) {
    // lane i owns row i of the Hermitian U (upper and lower halves averaged)
    for (int j = 0; j < K; ++j) {
#pragma unroll
      for (int q = 0; q < PL; ++q)
        w0[(lane * LD + j) * PL + q] = 0.5 * (U[(lane * LD + j) * PL + q] + (q ? -1.0 : 1.0) * U[(j * LD + lane) * PL + q]);
    }
    __syncwarp();
    double* H = w0;
    double* v = w1;          // reflector
    double* w = w1 + K * PL;
    for (int k = 0; k < K - 1; ++k) {
      const bool in = lane > k;
      double x[PL];
      double s = 0.0;
#pragma unroll
      for (int q = 0; q < PL; ++q) {
        x[q] = in ? H[(lane * LD + k) * PL + q] : 0.0;
        s += x[q] * x[q];
      }
      for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      if (lane == 0) off2[k] = s;
      if (k == K - 2) break;
      // v = x + phase(x_0) |x| e_1
      const double nrm = sqrt(s);
      double x0[PL], m0 = 0.0;
#pragma unroll
      for (int q = 0; q < PL; ++q) {
        x0[q] = __shfl_sync(0xffffffffu, x[q], k + 1);
        m0 += x0[q] * x0[q];
      }
      m0 = sqrt(m0);
      if (lane == k + 1) {
#pragma unroll
        for (int q = 0; q < PL; ++q) x[q] += nrm * (m0 > 0.0 ? x0[q] / m0 : (q ? 0.0 : 1.0));
      }
      const double vv = 2.0 * nrm * (nrm + m0), beta = vv > 0.0 ? 2.0 / vv : 0.0;
#pragma unroll
      for (int q = 0; q < PL; ++q) v[lane * PL + q] = x[q];
      __syncwarp();
      double p[PL] = {};
      if (in) {
        for (int j = k + 1; j < K; ++j) {
          const double* h = H + (lane * LD + j) * PL;
          if constexpr (PL == 1) {
            p[0] = fma(h[0], v[j], p[0]);
          } else {
            p[0] = fma(h[0], v[2 * j], fma(-h[1], v[2 * j + 1], p[0]));
            p[1] = fma(h[0], v[2 * j + 1], fma(h[1], v[2 * j], p[1]));
          }
        }
      }
      double vp = 0.0;
#pragma unroll
      for (int q = 0; q < PL; ++q) {
        p[q] *= beta;
        vp += x[q] * p[q];
      }
      for (int o = 16; o > 0; o >>= 1) vp += __shfl_xor_sync(0xffffffffu, vp, o);
#pragma unroll
      for (int q = 0; q < PL; ++q) {
        p[q] -= 0.5 * beta * vp * x[q];
        w[lane * PL + q] = p[q];
      }
      __syncwarp();
      if (in) {  // H -= v w^dagger + w v^dagger
        for (int j = k + 1; j < K; ++j) {
          double* h = H + (lane * LD + j) * PL;
          if constexpr (PL == 1) {
            h[0] -= x[0] * w[j] + p[0] * v[j];
          } else {
            h[0] -= x[0] * w[2 * j] + x[1] * w[2 * j + 1] + p[0] * v[2 * j] + p[1] * v[2 * j + 1];
            h[1] -= x[1] * w[2 * j] - x[0] * w[2 * j + 1] + p[1] * v[2 * j] - p[0] * v[2 * j + 1];
          }
        }
      }
      __syncwarp();
    }
    diag[lane] = H[(lane * LD + lane) * PL];
  }
  __syncthreads();
  if (warp < 2) {  // warp 0: the smallest eigenvalue (first x with a count of 1), warp 1: the largest (count K)
    double lo = diag[lane], hi = lo;
    {
      const double e0 = lane > 0 ? sqrt(off2[lane - 1]) : 0.0, e1 = lane + 1 < K ? sqrt(off2[lane]) : 0.0;
      lo -= e0 + e1;
      hi += e0 + e1;
    }
    for (int o = 16; o > 0; o >>= 1) {
      lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
      hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    }
    const double tiny = 1e-290, stop = 1e-13 * fmax(fabs(lo), fabs(hi));
    const int want = warp == 0 ? 1 : K;
    for (int it = 0; it < 12 && hi - lo > stop; ++it) {
      const double x = lo + (hi - lo) * (lane + 1) * (1.0 / 33.0);
      double q = diag[0] - x;
      int cnt = q < 0.0;
      for (int i = 1; i < K; ++i) {
        if (fabs(q) < tiny) q = -tiny;
        q = diag[i] - x - off2[i - 1] / q;
        cnt += q < 0.0;
      }
      const unsigned reach = __ballot_sync(0xffffffffu, cnt >= want);
      const int first = reach ? __ffs(reach) - 1 : 32;
      const double nlo = first > 0 ? __shfl_sync(0xffffffffu, x, first - 1) : lo;
      const double nhi = first < 32 ? __shfl_sync(0xffffffffu, x, first & 31) : hi;
      lo = nlo;
      hi = nhi;
    }
    if (lane == 0) ends[warp] = 0.5 * (lo + hi);
  }
  __syncthreads();
  if (tid == 0) {
    const double lo = ends[0], hi = ends[1], spread = hi - lo;
    if (!(spread >= 0.0) || !isfinite(lo) || !isfinite(hi)) return;
    const double m = 0.1 * spread + 1e-12 * fmax(fabs(lo), fabs(hi));
    const double nlo = fmax(b[0], lo - m), nhi = fmin(b[1], hi + m);
    if (nhi > nlo) {
      b[0] = nlo;
      b[1] = nhi;
    }
  }
}

}  // namespace

namespace {

Sp2Args make_args(const Sp2Problem& q, bool cplx, bool sure, int max_steps) {
  const int PL = cplx ? 2 : 1;
  Sp2Args g{};
  g.F = q.F;
  g.b = q.b;
  g.X = q.X;
  g.Y = q.Y;
  g.part = q.scratch;
  g.bar = reinterpret_cast<unsigned*>(q.scratch + 4 * kMaxTiles);
  g.outcome = q.outcome;
  g.nocc = q.nocc;
  g.n = static_cast<int>(q.n);
  g.max_steps = max_steps;
  g.sure = sure;
  const int kfit = kSp2Smem / static_cast<int>(sizeof(double)) / (2 * TILE * PL) - 4;
  g.kc = std::min<int>(static_cast<int>(round_up(q.n, 8)), kfit / 8 * 8);
  return g;
}
int smem_of(const Sp2Args& g, int PL) { return static_cast<int>(sizeof(double)) * 2 * TILE * PL * (g.kc + 4); }
int tiles_of(int64_t n) {
  const int nt = static_cast<int>((n + TILE - 1) / TILE);
  return nt * (nt + 1) / 2;
}

}  // namespace

int64_t sp2_scratch_doubles() { return 4 * kMaxTiles + 32; }

int64_t sp2_workspace_doubles(int64_t n, bool cplx) {
  return std::max<int64_t>(8 * n * n * (cplx ? 2 : 1) + 6 * kScfRedCtas, sp2_scratch_doubles() + 4);
}

void sp2_run_group(const Sp2Problem* p, int count, const std::function<const void*(const void*, size_t)>& put, cudaStream_t s) {
  static std::atomic<bool> attr[kMaxDevices];
  once_per_device(attr, [] {
    RR_CUDA(cudaFuncSetAttribute(sp2_group_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSp2Smem));
  });
  // at most half as many problems a launch as CTAs fit the GPU at once; CTAs in proportion to a step's work
  for (int p0 = 0; p0 < count;) {
    int smem = 0, many = 0, per_sm = 0, room = 0;
    std::vector<Sp2Entry> tab;
    std::vector<double> work;
    double all = 0.0;
    while (p0 + many < count) {
      Sp2Entry e{};
      e.a = make_args(p[p0 + many], true, true, 120);
      const int need = std::max(smem, smem_of(e.a, 2));
      RR_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, sp2_group_kernel, SP2_THREADS, need));
      const int fits = std::min(per_sm * sm_count_current(), kMaxGroupCtas);
      if (many > 0 && many + 1 > fits / 2) break;
      room = fits;
      smem = need;
      tab.push_back(e);
      work.push_back(static_cast<double>(tiles_of(e.a.n)) * e.a.n);
      all += work.back();
      ++many;
    }
    std::vector<int> of;
    for (int i = 0; i < many; ++i) {
      const int share = static_cast<int>((room - many) * (work[i] / all));
      tab[i].first = static_cast<int>(of.size());
      tab[i].ctas = std::max(1, std::min(1 + share, tiles_of(tab[i].a.n)));
      of.insert(of.end(), tab[i].ctas, i);
      RR_CUDA(cudaMemsetAsync(tab[i].a.bar, 0, 2 * sizeof(unsigned), s));
    }
    const Sp2Entry* dt = static_cast<const Sp2Entry*>(put(tab.data(), sizeof(Sp2Entry) * tab.size()));
    const int* dof = static_cast<const int*>(put(of.data(), sizeof(int) * of.size()));
    void* args[] = {&dt, &dof};
    RR_CUDA(cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(sp2_group_kernel), dim3(static_cast<unsigned>(of.size())),
                                        dim3(SP2_THREADS), args, smem, s));
    RR_LAUNCH_CHECK();
    p0 += many;
  }
}

void sp2_run(const double* F, int64_t n, double nocc, bool cplx, const double* b, bool sure, int max_steps, double* X, double* Y,
             double* scratch, double* outcome, cudaStream_t s) {
  const int PL = cplx ? 2 : 1;
  static std::atomic<bool> attr[kMaxDevices];
  once_per_device(attr, [] {
    RR_CUDA(cudaFuncSetAttribute(sp2_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSp2Smem));
    RR_CUDA(cudaFuncSetAttribute(sp2_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSp2Smem));
  });
  Sp2Args g = make_args(Sp2Problem{F, b, X, Y, scratch, outcome, nocc, n}, cplx, sure, max_steps);
  const int smem = smem_of(g, PL), grid = std::max(1, std::min(tiles_of(n), sm_count_current()));
  RR_CUDA(cudaMemsetAsync(g.bar, 0, 2 * sizeof(unsigned), s));
  void* args[] = {&g};
  RR_CUDA(cudaLaunchCooperativeKernel(cplx ? reinterpret_cast<const void*>(sp2_kernel<2>) : reinterpret_cast<const void*>(sp2_kernel<1>),
                                      dim3(grid), dim3(SP2_THREADS), args, smem, s));
  RR_LAUNCH_CHECK();
}

void ritz_interval(const double* T, const double* M, bool cplx, double* b, cudaStream_t s) {
  const int smem = static_cast<int>(sizeof(double)) * 4 * kRitz * (kRitz | 1) * (cplx ? 2 : 1);
  static std::atomic<bool> attr[kMaxDevices];
  once_per_device(attr, [] {
    RR_CUDA(cudaFuncSetAttribute(ritz_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, 4 * kRitz * (kRitz | 1) * 16));
  });
  if (cplx) ritz_kernel<2><<<1, THREADS, smem, s>>>(T, M, b);
  else ritz_kernel<1><<<1, THREADS, smem, s>>>(T, M, b);
  RR_LAUNCH_CHECK();
}

}  // namespace rr
