// FP64 products on the INT8 tensor cores (tcgen05 kind::i8): every FP64 operand is scaled by a power of two
// per row and cut into eight signed base-256 digits, the digit planes are multiplied exactly in INT32
// (Ozaki, Ogita, Oishi, Rump, "Error-free transformations of matrix multiplication", Numer. Algorithms 59,
// 2012; balanced digits instead of their floating-point slices), and the eight anti-diagonals of plane
// products are recombined in FP64.
//
//   x = 2^(e - 63) v,  1.005 |x| < 2^e,  v = round(x 2^(63 - e)) = sum_i D_i 256^(7 - i),  D_i in [-128, 127]
//   sum_k x_k y_k = 2^(ex + ey - 126) sum_{i + j <= 7} 256^(14 - i - j) sum_k Dx_i Dy_j  + truncation
//
// The 36 plane pairs with i + j <= 7 are kept.  Dropped: the rounding of v, 2^-64 of 2^e, and the pairs of
// weight 256^6 and below, for K terms of unrelated operands about sqrt(7 K) 74^2 2^-78 of 2^(ex + ey).  Where
// an operand meets itself (the diagonal of a symmetric product) the pair (4, 4) does not average out: its sum
// of squares is formed beside the digits (HalfOut::sq) and added by the caller.  Rows of different functions that coincide beyond
// digit 4 (equal functions) keep it, kk 74^2 2^-78 of 2^(ea + eb): J and K of 128 functions, equal in pairs, kk = 25600, off by 2^-49.0 of
// sqrt(K_aa K_bb) at most, against 2^-49.8 on DMMA; of 128 different ones 2^-50.5 against 2^-49.9.
// INT32 holds 8 K 2^14 for K <= kOzMaxK.
#pragma once

#include <cuda.h>

#include <cmath>
#include <cstdint>

#include "rr_common.cuh"

namespace rr {
namespace oz {

constexpr int kDigits = 8;
constexpr int kBM = 128;       // output rows of a tile (TMEM lanes)
constexpr int kBN = 64;        // widest output column tile: kDigits * kBN = 512 TMEM columns
constexpr int kBK = 32;        // K bytes of one MMA and of one pipeline stage
constexpr int64_t kOzMaxK = 16256;  // longest INT32 accumulation, a multiple of kBK below 2^14
constexpr int kExpBad = 30000;      // exponent of a row that holds a NaN or an infinity: its products are NaN
constexpr int kExpZero = -500;      // exponent of a zero row, and the least exponent (resolution 2^-563)

// Digit planes in the order the tensor cores read them: tiles of `rt` rows (128; 64 for coefficient operands,
// the last of those only as tall as its column tile), K blocks of 32 bytes, planes, and inside a plane of a
// block the core matrices of 8 rows x 16 bytes, the two of one row group adjacent.  One tile's K block is
// contiguous over all planes, so a stage is one bulk copy.
struct Planes {
  uint8_t* p = nullptr;
  int64_t rows = 0, k = 0;
  int rt = kBM;
  __host__ __device__ int64_t kblocks() const { return (k + kBK - 1) / kBK; }
  __host__ __device__ int64_t tile_bytes() const { return kblocks() * kDigits * rt * kBK; }
  __host__ __device__ int64_t bytes() const { return (rows + rt - 1) / rt * tile_bytes(); }
  // Rows of the tile that row r is in (coefficient operands: the last tile is as tall as its rows, in 16s).
  __host__ __device__ int tile_rows(int64_t r) const {
    if (rt == kBM) return kBM;
    const int64_t left = (rows + 15) / 16 * 16 - r / rt * rt;
    return left < rt ? static_cast<int>(left) : rt;
  }
  // Byte (row r, k) of plane 0; plane d is d * tile_rows(r) * kBK further.
  __host__ __device__ int64_t at(int64_t r, int64_t kk) const {
    const int64_t i = r % rt, j = kk % kBK;
    return r / rt * tile_bytes() + kk / kBK * (static_cast<int64_t>(kDigits) * tile_rows(r) * kBK) + i / 8 * 256 +
           j / 16 * 128 + i % 8 * 16 + j % 16;
  }
};

// Where the coefficient rows of a conversion product come from: column (output) c of the product is row c
// of a real matrix, element k.
//   kind 0: src[c * ld + k]                                          (rows x K, row-major)
//   kind 1: src[k * ld + c]                                          (K x rows, row-major)
//   kind 2: c < 2 per: pair c / 2 of complex rows: part (c & 1) of src[(c / 2) * ld + off + k], zero for
//           pairs >= rows; per = the padded pair count                (complex, interleaved)
//   kind 3: c < per: Re src[k * ld + c], else Im src[k * ld + c - per], rows offset off in k
//   kind 4: row c of [Re c; Im c] (c even: pair c/2) or [-Im c; Re c] (c odd) over k < 2 half:
//           k < half: row k of the complex K x nt matrix src, else row k - half
struct CoefSrc {
  const double* src = nullptr;
  int64_t ld = 0, off = 0;
  int kind = 0;
  int64_t rows = 0;  // valid rows (pairs for kind 2)
  int64_t half = 0;
};

// Digits of `count` coefficient rows of K elements into pl at rows [row0, row0 + count) (and zero rows up to the end
// of pl); scale[row0 + c] = 2^(e - 35) of the row's exponent (a NaN for a row that is not finite), norm[row0 + c] the 2-norms (rounded up; of the complex row for kinds 2 and 3).
void digitize_rows(const CoefSrc& c, int64_t count, int64_t K, const Planes& pl, int64_t row0, double* scale, double* norm,
                   cudaStream_t s);

// Columns of a three-centre tensor: cscale[P n + a] = 2^(e - 35) for the exponent of column a of B^P, cnorm[a] >= max_P
// ||B^P[:, a]||_2, pnorm[P] >= max_a of it; flag is set when B holds a NaN, an infinity or a value beyond 1e140.
struct ColumnStats {
  double *cscale = nullptr, *cnorm = nullptr, *pnorm = nullptr;
  int* flag = nullptr;
};
// Statistics of the whole tensor and, with pl, its digit planes: row P n + a, byte q.
void digitize_columns(const double* B, int64_t pitch, int64_t n, int64_t naux, const Planes* pl, const ColumnStats& st,
                      cudaStream_t s);
// Digit planes of the aux rows P0 .. P0 + naux from known exponents; row (P - P0) n + a.
void digitize_range(const double* B, int64_t pitch, int64_t n, int64_t P0, int64_t naux, const Planes& pl, const double* cscale,
                    cudaStream_t s);

// Exponents of the half-transformed rows: e[a] for |sum_q B^P[q][a] c[q]|, every P and every coefficient row of norm
// at most max(norm[0 .. nnorm)).  scale[a] = 2^(e - 35) (padded to a multiple of 64 entries), tinv[a] = 2^(31 - e),
// sq[a] = 0, rowmax[a] = 0, mag[a] = 0 (kMagNever where e is no magnitude: a zero row or one that is not finite).
constexpr unsigned long long kMagNever = 1ull << 62;
struct RowScales {
  int* e = nullptr;
  double *scale = nullptr, *tinv = nullptr, *rowmax = nullptr;
  unsigned long long *sq = nullptr, *mag = nullptr;
};
void row_scales(const double* cnorm, int64_t n, const double* norm, int64_t nnorm, const RowScales& out, cudaStream_t s);
// The same for the MO transform: entry P per + j from pnorm[P] and the norm of coefficient column j (max over the ntab
// norm tables norm + t * nstride; the second half of them with pnorm1).
void pair_scales(const double* pnorm0, const double* pnorm1, int64_t naux, const double* norm, int64_t per, int64_t ntab,
                 int64_t nstride, double* scale, double* tinv, cudaStream_t s);

// Half-transform: T[(P, a)][c] = sum_q B^P[q][a] coef[c][q], the result as digit planes.
struct HalfOut {
  int mode = 0;  // 0: real exchange planes, 1: complex exchange planes, 2: MO planes
  // mode 0 / 1: planes at row a, byte P period + j, inverse row scale tinv[a]; mode 1: two flavours of 2 period columns
  // (pair j, part) each, four plane sets Re, Im, (Re - Im) / 2, (Re + Im) / 2 (null: not wanted).  sq[a] +=
  // the squares of digit 4 of the row (of Re and Im), mag[a] += the squares of its top 16 bits.
  int64_t period = 0;
  Planes t;                 // shape of every plane set
  uint8_t* pl[2][4] = {};
  const double* tinv[2] = {nullptr, nullptr};
  unsigned long long *sq[2] = {nullptr, nullptr}, *mag[2] = {nullptr, nullptr};
  // mode 2: row Pl per + c % per, byte (c / per) chi + koff + a with Pl = P - P0, inverse scale tinv[0][Pl per + c % per]
  int64_t per = 0, chi = 0, koff = 0;
  int64_t tile_bytes = 0;  // filled by half_product
  bool quad = false;
};
// Aux rows P0 .. P0 + naux of the tensor; b: digit planes whose row 0 is aux row Pb (row (P - Pb) n + a).
void half_product(const Planes& b, int64_t Pb, int64_t n, int64_t P0, int64_t naux, const double* cscale,
                  const Planes& coef, const double* coef_scale, int64_t ncol, const HalfOut& out, int* err, cudaStream_t s);

// Rows of exchange planes whose exponent, a Cauchy-Schwarz bound, lies too far above their values: a product of two rows
// a, b of kk terms drops about sqrt(7 kk) 74^2 2^-78 of 2^(ea + eb), which is measured against sqrt(K_aa K_bb), K_aa = sum T_a^2,
// so its part grows with the square of rho = 2^e / sqrt(K_aa).  A row with rho^2 above refit_limit(kk) (that part above
// 2^-50; kk = 64000 FP64 additions in a row leave about 2^-45) gets its true exponent: its T is formed again in FP64 and cut anew, and rho
// is at most 2.01.  Such rows are rare (rho at the limits' sizes: at most 6.6 of 8.6 for n = 400, naux = 1600, 40 orbitals of the benchmark's
// recipe, 7.9 of 9.7 for its four components; 3.5 of 13 for water and CO / cc-pVDZ at their SCF orbitals): nearly
// dependent functions with large cancelling coefficients, functions far from every occupied orbital.
inline double refit_limit(int64_t kk) {
  const double r = 49664.0 / sqrt(7.0 * static_cast<double>(kk));
  return r < 256.0 ? r : 256.0;
}
struct RefitRows {
  const double* B = nullptr;  // the flavour's tensor, rows of n x n
  int64_t pitch = 0, n = 0;
  CoefSrc c;                  // its coefficients (kinds 0 - 2), as digitize_rows took them
  uint8_t* pl[4] = {};        // its plane sets (HalfOut)
  RowScales row;
};
// All flavours of a build (r coefficient rows or pairs, planes of shape (n, naux period)), after its half-transforms.
void refit_rows(const RefitRows* f, int nf, int64_t naux, int64_t r, int64_t period, cudaStream_t s);

// A list of products C_p[i][j] = sum_k A_p[i][k] B_p[j][k] of digit planes, one launch.
struct Prod {
  Planes a, b;
  const double *sa = nullptr, *sb = nullptr;  // row scales of a and of b (b's padded to a multiple of 16)
  int64_t M = 0, N = 0, K = 0;
  int sym = 0;           // tiles that touch the upper triangle only
  int negate_odd = 0;    // odd output columns negated (conjugate of an interleaved complex result)
  int splits = 1;        // K ranges of at most kOzMaxK
  int64_t kchunk = 0;
  double* out = nullptr; // split s at out + s * sstride; row i at i * ldo
  int64_t ldo = 0, sstride = 0;
};
constexpr int kMaxProds = 32;
// Fills splits and kchunk of every product so that the list has several items per SM; returns nothing else.
void plan_products(Prod* p, int count);
void run_products(const Prod* p, int count, int* err, cudaStream_t s);

}  // namespace oz
}  // namespace rr
