// FP64 products on the INT8 tensor cores: kernels and host side of oz.cuh.
//
// oz_gemm_kernel: a persistent CTA per SM walks 128 x 64 output tiles of a list of products of digit planes.
// One warp brings 32 K bytes of all eight planes of both operands (48 KB a stage, four stages; the planes lie in
// memory as the tensor cores read them, so a stage is one bulk copy of 32 KB and one of 16); one thread issues
// the MMAs: plane i of A meets the planes 0 .. 7 - i of B, stacked in shared memory, in one wide MMA
// whose output columns start at anti-diagonal i.  Eight anti-diagonals x 64 columns are the 512 TMEM columns,
// and a plane of A is read from shared memory once or twice a K step instead of 8 - i times.  Sixteen epilogue
// warps drain TMEM into FP64 registers (eight INT32 anti-diagonals -> two INT64 -> one double), free it for the
// next tile's MMAs, then scale and store: FP64, or the digit planes of the result for the next product.
//
// Bound, more than one column tile: the tensor pipe as these MMAs drive it.  A step of 128 x 64 x 32 takes 1668 cycles, with
// the copies and without them (clock64 around 508 steps of 144 tiles): 5660 INT8 MAC per cycle and SM of the nominal 8192 (1152 cycles),
// 3.3 P operations/s on 148 SMs at 1965 MHz, where cuBLAS' INT8 GEMM of 8192^3 reaches 3.0; divided by the 36 plane pairs, 91 TF/s of
// FP64 products.  Half-transforms of one column tile (up to 64 orbitals) stream the tensor's planes at 4.4 TB/s and are bound by that.  Against
// the DMMA kernels: n = 400, naux = 1600, nocc = 40: half-transform 773 -> 484 us (2.1 GB of planes read), SYRK 443 -> 199 us; four
// components nl = 200, ns = 600, naux = 1000, 40 spinors: half-transforms 5.7 -> 2.7 ms, exchange blocks 15.2 -> 4.9 ms; MO transform
// n = 400, naux = 1600: 16.9 -> 7.3 ms.
//
// digitize_columns_kernel: the three-centre tensor to digit planes, one pass over HBM (the tile of 32 columns
// stays in shared memory between the search for its largest magnitudes and the conversion).
#include <cuda.h>

#include <algorithm>
#include <vector>

#include "oz.cuh"
#include "umma.cuh"

namespace rr {
namespace oz {
namespace {

constexpr int ERR_OZ_FULL = 1 << 17, ERR_OZ_EMPTY = 1 << 18, ERR_OZ_TFULL = 1 << 19, ERR_OZ_TEMPTY = 1 << 20,
              ERR_OZ_DONE = 1 << 21;

constexpr int STAGES = 4;
constexpr int A_PLANE = kBM * kBK;             // 4 KB
constexpr int A_BYTES = kDigits * A_PLANE;     // 32 KB
constexpr int B_BYTES = kDigits * kBN * kBK;   // 16 KB
constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
constexpr int BAR_OFF = STAGES * STAGE_BYTES;
constexpr int SMEM_BYTES = BAR_OFF + 256 + 1024;
constexpr int EPI_WARPS = 16;  // four per group of 32 TMEM lanes, each with up to 16 columns in two units of eight
constexpr int GEMM_THREADS = 32 * (EPI_WARPS + 2);
constexpr int kKeepBytes = 220 * 1024;  // column tile of digitize_columns_kernel
static_assert(SMEM_BYTES <= 232448, "shared memory per CTA");

// ---- tcgen05 kind::i8 ----
// Instruction descriptor: S32 accumulator (2 at bit 4), signed 8-bit A and B (1 at bits 7 and 10), N / 8 at bit
// 17, M / 16 at bit 24; both operands K-major.
__device__ __forceinline__ uint32_t idesc_s8(int n) {
  return (2u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>(n >> 3) << 17) |
         (static_cast<uint32_t>(kBM >> 4) << 24);
}

__device__ __forceinline__ void umma_i8(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                        uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n}\n" ::"r"(d_tmem),
      "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(0u), "r"(0u), "r"(0u), "r"(0u)
      : "memory");
}

// K-major operand without swizzle: core matrices of 8 rows x 16 bytes, the next along K 128 bytes on (leading
// byte offset), the next 8 rows 256 bytes on (stride byte offset); descriptor version 1, layout type 0.
__device__ __forceinline__ uint64_t sdesc_cores(uint32_t smem_addr) {
  return static_cast<uint64_t>((smem_addr >> 4) & 0x3FFFu) | (static_cast<uint64_t>(128u >> 4) << 16) |
         (static_cast<uint64_t>(256u >> 4) << 32) | (static_cast<uint64_t>(1u) << 46);
}

// The MMAs of one stage (32 K bytes), nt columns a plane: pieces of at most 256 columns, multiples of 16 (nt is
// one).
__device__ __forceinline__ void issue_stage(uint32_t tmem, uint32_t stage, int nt, bool first) {
  const uint64_t a0 = sdesc_cores(stage), b0 = sdesc_cores(stage + A_BYTES);
#pragma unroll
  for (int i = 0; i < kDigits; ++i) {
    const uint64_t a = a0 + (static_cast<uint64_t>(i * A_PLANE) >> 4);
    const int n = nt * (kDigits - i);
    const uint32_t acc = (first && i == 0) ? 0u : 1u;
    const int n0 = n <= 256 ? n : (n / 2 + 15) / 16 * 16;
    umma_i8(tmem + nt * i, a, b0, idesc_s8(n0), acc);
    if (n > n0) umma_i8(tmem + nt * i + n0, a, b0 + (static_cast<uint64_t>(n0 * kBK) >> 4), idesc_s8(n - n0), acc);
  }
}

// Four columns of the eight anti-diagonals, load and wait in one statement (the values exist after the wait).
__device__ __forceinline__ void tmem_ld_diag(uint32_t t, uint32_t nt, int (&r)[kDigits][4]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%32];\n"
      "tcgen05.ld.sync.aligned.32x32b.x4.b32 {%4,%5,%6,%7}, [%33];\n"
      "tcgen05.ld.sync.aligned.32x32b.x4.b32 {%8,%9,%10,%11}, [%34];\n"
      "tcgen05.ld.sync.aligned.32x32b.x4.b32 {%12,%13,%14,%15}, [%35];\n"
      "tcgen05.ld.sync.aligned.32x32b.x4.b32 {%16,%17,%18,%19}, [%36];\n"
      "tcgen05.ld.sync.aligned.32x32b.x4.b32 {%20,%21,%22,%23}, [%37];\n"
      "tcgen05.ld.sync.aligned.32x32b.x4.b32 {%24,%25,%26,%27}, [%38];\n"
      "tcgen05.ld.sync.aligned.32x32b.x4.b32 {%28,%29,%30,%31}, [%39];\n"
      "tcgen05.wait::ld.sync.aligned;\n"
      : "=r"(r[0][0]), "=r"(r[0][1]), "=r"(r[0][2]), "=r"(r[0][3]), "=r"(r[1][0]), "=r"(r[1][1]), "=r"(r[1][2]),
        "=r"(r[1][3]), "=r"(r[2][0]), "=r"(r[2][1]), "=r"(r[2][2]), "=r"(r[2][3]), "=r"(r[3][0]), "=r"(r[3][1]),
        "=r"(r[3][2]), "=r"(r[3][3]), "=r"(r[4][0]), "=r"(r[4][1]), "=r"(r[4][2]), "=r"(r[4][3]), "=r"(r[5][0]),
        "=r"(r[5][1]), "=r"(r[5][2]), "=r"(r[5][3]), "=r"(r[6][0]), "=r"(r[6][1]), "=r"(r[6][2]), "=r"(r[6][3]),
        "=r"(r[7][0]), "=r"(r[7][1]), "=r"(r[7][2]), "=r"(r[7][3])
      : "r"(t), "r"(t + nt), "r"(t + 2 * nt), "r"(t + 3 * nt), "r"(t + 4 * nt), "r"(t + 5 * nt), "r"(t + 6 * nt),
        "r"(t + 7 * nt)
      : "memory");
}

// Integer <-> FP64 conversions through the mantissa of 2^52 (+ 2^51): additions on the FP64 pipe. 
__device__ __forceinline__ double from_s32(int v) {
  return __hiloint2double(0x43300000, v ^ static_cast<int>(0x80000000u)) - 4503601774854144.0;  // 2^52 + 2^31
}
__device__ __forceinline__ double from_u32(uint32_t v) {
  return __hiloint2double(0x43300000, static_cast<int>(v)) - 4503599627370496.0;
}
// hi 2^32 + lo for |hi|, |lo| < 2^58 with at most two roundings of 2^-53 of the result: three signed words, so
// that a small sum has no large parts that cancel.
__device__ __forceinline__ double join96(int64_t hi, int64_t lo) {
  const int64_t h = hi + (lo >> 32);
  const int mid = static_cast<int>(h), top = static_cast<int>(h >> 32) + (mid < 0 ? 1 : 0);
  return fma(from_s32(top), 18446744073709551616.0, fma(from_s32(mid), 4294967296.0, from_u32(static_cast<uint32_t>(lo))));
}
// round(x s) for |x s| < 2^63 / 1.004, given s 2^-32: the upper word by rounding, the lower one from the exact remainder.
__device__ __forceinline__ int64_t to_s64(double x, double s32) {
  constexpr double kMagic = 6755399441055744.0;  // 2^52 + 2^51
  const double t1 = fma(x, s32, kMagic);
  const double t2 = fma(fma(x, s32, kMagic - t1), 4294967296.0, kMagic);
  const uint32_t lo = static_cast<uint32_t>(__double2loint(t2));
  const uint32_t hi = static_cast<uint32_t>(__double2loint(t1)) + static_cast<uint32_t>(__double2hiint(t2)) - 0x43380000u;
  return static_cast<int64_t>((static_cast<uint64_t>(hi) << 32) | lo);
}

// First column of this warp's unit u (0, 1): units of eight are dealt out to the four column groups, in adjacent
// pairs where a store needs sixteen columns; at or beyond nt: none.
template <int MODE>
__device__ __forceinline__ int unit_col(int group, int u) {
  return MODE == 1 ? 16 * group + 8 * u : 8 * (group + 4 * u);
}

// Drains this warp's 32 rows of its units into w[]: the exact INT64 sums of the upper and the lower four
// anti-diagonals, joined in FP64.
template <int MODE>
__device__ __forceinline__ void drain(uint32_t tmem_row, int nt, int group, double* w) {
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const int col = unit_col<MODE>(group, u);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      if (col < nt) {
        int r[kDigits][4];
        tmem_ld_diag(tmem_row + col + 4 * h, static_cast<uint32_t>(nt), r);
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          const int64_t hi = static_cast<int64_t>(r[0][t]) * (1 << 24) + static_cast<int64_t>(r[1][t]) * (1 << 16) +
                             static_cast<int64_t>(r[2][t]) * (1 << 8) + r[3][t];
          const int64_t lo = static_cast<int64_t>(r[4][t]) * (1 << 24) + static_cast<int64_t>(r[5][t]) * (1 << 16) +
                             static_cast<int64_t>(r[6][t]) * (1 << 8) + r[7][t];
          w[8 * u + 4 * h + t] = join96(hi, lo);
        }
      } else {
#pragma unroll
        for (int t = 0; t < 4; ++t) w[8 * u + 4 * h + t] = 0.0;
      }
    }
  }
}

// 2^e as a double for e in the normal range (clamped); NaN for the mark of a non-finite row.
__device__ __forceinline__ double pow2i(int e) {
  e = max(-1022, min(1023, e));
  return __longlong_as_double(static_cast<int64_t>(e + 1023) << 52);
}
__device__ __forceinline__ double scale_of(int e, int shift) {
  return e >= kExpBad ? __longlong_as_double(0x7FF8000000000000ll) : pow2i(e + shift);
}
constexpr int kRowShift = -35;  // a result is w 2^(ex + ey - 70): half of it with either row

// Balanced base-256 digits of v: bytes of (v + 0x80..80) ^ 0x80..80, least significant first.
__device__ __forceinline__ uint64_t digit_bytes(int64_t v) {
  return (static_cast<uint64_t>(v) + 0x8080808080808080ull) ^ 0x8080808080808080ull;
}

// Four 32-bit words to their byte columns: out[b] = byte b of in[0..3].
__device__ __forceinline__ void transpose4(const uint32_t* in, uint32_t* out) {
  const uint32_t a = __byte_perm(in[0], in[1], 0x5140), b = __byte_perm(in[2], in[3], 0x5140);
  const uint32_t c = __byte_perm(in[0], in[1], 0x7362), d = __byte_perm(in[2], in[3], 0x7362);
  out[0] = __byte_perm(a, b, 0x5410);
  out[1] = __byte_perm(a, b, 0x7632);
  out[2] = __byte_perm(c, d, 0x5410);
  out[3] = __byte_perm(c, d, 0x7632);
}

// Digits of eight values x 2^32 (|x| < 2^31 / 1.004): out[plane] = their bytes, plane 0 most significant.
__device__ __forceinline__ void digits8(const double* x, uint2* out) {
  uint32_t lo[8], hi[8];
#pragma unroll
  for (int t = 0; t < 8; ++t) {
    const uint64_t u = digit_bytes(to_s64(x[t], 1.0));
    lo[t] = static_cast<uint32_t>(u);
    hi[t] = static_cast<uint32_t>(u >> 32);
  }
  uint32_t p[4], q[4];
  transpose4(lo, p);
  transpose4(lo + 4, q);
#pragma unroll
  for (int b = 0; b < 4; ++b) out[7 - b] = make_uint2(p[b], q[b]);
  transpose4(hi, p);
  transpose4(hi + 4, q);
#pragma unroll
  for (int b = 0; b < 4; ++b) out[3 - b] = make_uint2(p[b], q[b]);
}

struct Bars {
  uint64_t *full, *empty, *tfull, *tempty, *done;
  uint32_t* tmem_slot;
  __device__ explicit Bars(unsigned char* smem) {
    full = reinterpret_cast<uint64_t*>(smem + BAR_OFF);
    empty = full + STAGES;
    tfull = empty + STAGES;
    tempty = tfull + 1;
    done = tempty + 1;
    tmem_slot = reinterpret_cast<uint32_t*>(done + 1);
  }
};

// ---------------------------------------------------------------- the product kernel

struct Item {
  int p, m0, n0, nt, k0, k1, split;
};

struct ProdDev {
  const uint8_t *a, *b;
  int64_t a_tile, b_tile;  // bytes of a 128-row tile of A, of a 128- or 64-row tile of B
  int b_rt;                // rows of B's tiles
  int mt0, row0;           // first row tile, first valid row
  int M, N, K;
  int tn, ntl;     // column tiles, width of the last one
  int sym, negate_odd, kchunk;
  const double *sa, *sb;  // row scales 2^(e - 35) of A and of B (padded to whole column tiles)
  double* out;
  int64_t ldo, sstride;
};

// Items are ordered by segments: every product's full column tiles, then every product's narrow last column tiles,
// so that the short items fill the end of the launch.
struct Seg {
  int item0, p, narrow, tiles;
};

struct GemmArgs {
  ProdDev p[kMaxProds];
  Seg seg[2 * kMaxProds];
  int segs, items;
};

// One product whose result leaves as digit planes (half-transforms).
struct HalfArgs {
  ProdDev p;
  int items, n, Pl0;  // Pl0: aux row of the planes that is aux row P0 of the tensor
  int64_t P0;
  HalfOut o;
};
__device__ __forceinline__ const ProdDev& prod_of(const GemmArgs& g, int p) { return g.p[p]; }
__device__ __forceinline__ const ProdDev& prod_of(const HalfArgs& g, int) { return g.p; }
__device__ __forceinline__ Item item_of(const ProdDev& d, int p, int m, int n, int split) {
  Item t;
  t.p = p;
  t.split = split;
  t.m0 = (m + d.mt0) * kBM;
  t.n0 = n * kBN;
  t.nt = n == d.tn - 1 ? d.ntl : kBN;
  t.k0 = split * d.kchunk;
  t.k1 = min(d.K, t.k0 + d.kchunk);
  return t;
}

// Work item -> product, tile and K range; tiles of one K range are consecutive.
__device__ __forceinline__ Item decode(const GemmArgs& g, int item) {
  int i = 0;
  while (i + 1 < g.segs && g.seg[i + 1].item0 <= item) ++i;
  const Seg s = g.seg[i];
  const ProdDev& d = g.p[s.p];
  const int local = item - s.item0, split = local / s.tiles;
  int tile = local - split * s.tiles, m = 0, n;
  const int wide = d.tn - (d.ntl < kBN ? 1 : 0);  // full column tiles
  if (s.narrow) {
    m = tile;
    n = d.tn - 1;
  } else if (d.sym) {  // row tile m keeps the column tiles that reach row 128 m: n >= 2 m
    while (tile >= wide - 2 * m) {
      tile -= wide - 2 * m;
      ++m;
    }
    n = 2 * m + tile;
  } else {
    m = tile / wide;
    n = tile - m * wide;
  }
  return item_of(d, s.p, m, n, split);
}

// Half-transforms: the column tiles of a row tile are consecutive (they share the tensor through L2).
__device__ __forceinline__ Item decode(const HalfArgs& g, int item) {
  const int m = item / g.p.tn;
  return item_of(g.p, 0, m, item - m * g.p.tn, 0);
}

// Byte (row r, k) of plane 0 of 128-row tiles (Planes::at).
__device__ __forceinline__ int64_t left_at(int64_t tile_bytes, uint32_t r, uint32_t k) {
  return (r >> 7) * tile_bytes + static_cast<int64_t>(k >> 5) * A_BYTES + ((r & 127) >> 3) * 256 + ((k >> 4) & 1) * 128 +
         (r & 7) * 16 + (k & 15);
}

// Eight column scales from column c (a multiple of eight).
__device__ __forceinline__ void load8(const double* p, double* v) {
#pragma unroll
  for (int i = 0; i < 8; i += 2) {
    const double2 d = __ldg(reinterpret_cast<const double2*>(p + i));
    v[i] = d.x;
    v[i + 1] = d.y;
  }
}

// w sa sb to the FP64 output of one row.
__device__ __forceinline__ void store_f64(const ProdDev& d, const Item& t, int row, int group, double sa, const double* w) {
  double* out = d.out + t.split * d.sstride + row * d.ldo + t.n0;
  const double odd = d.negate_odd ? -1.0 : 1.0;
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const int c = unit_col<3>(group, u);
    if (c < t.nt && t.n0 + c < d.N) {
      double sb[8], y[8];
      load8(d.sb + t.n0 + c, sb);  // padded to whole tiles
#pragma unroll
      for (int i = 0; i < 8; ++i) y[i] = w[8 * u + i] * sa * ((i & 1) ? odd * sb[i] : sb[i]);
      double* o = out + c;
      if (t.n0 + c + 8 <= d.N && (reinterpret_cast<uintptr_t>(o) & 31) == 0) {
#pragma unroll
        for (int i = 0; i < 8; i += 4)
          asm volatile("st.global.v4.f64 [%0], {%1,%2,%3,%4};\n" ::"l"(o + i), "d"(y[i]), "d"(y[i + 1]), "d"(y[i + 2]),
                       "d"(y[i + 3])
                       : "memory");
      } else {
#pragma unroll
        for (int i = 0; i < 8; ++i)
          if (t.n0 + c + i < d.N) o[i] = y[i];
      }
    }
  }
}

__device__ __forceinline__ unsigned square_sum(uint2 d) {
  return static_cast<unsigned>(__dp4a(static_cast<int>(d.x), static_cast<int>(d.x),
                                      __dp4a(static_cast<int>(d.y), static_cast<int>(d.y), 0)));
}

// Squares of the top 16 bits of eight values, from their two leading digit planes.
__device__ __forceinline__ unsigned long long top_square_sum(uint2 a, uint2 b) {
  const int ax = static_cast<int>(a.x), ay = static_cast<int>(a.y), bx = static_cast<int>(b.x), by = static_cast<int>(b.y);
  const int aa = __dp4a(ax, ax, __dp4a(ay, ay, 0)), ab = __dp4a(ax, bx, __dp4a(ay, by, 0)), bb = __dp4a(bx, bx, __dp4a(by, by, 0));
  return static_cast<unsigned long long>(aa * 65536ll + ab * 512ll + bb);
}

// Four lanes x four 64-bit values to their transpose: lane i gets the values that the quad's lanes hold at i.
__device__ __forceinline__ void quad_transpose(uint64_t (&v)[4], int lane) {
  const bool b0 = lane & 1, b1 = lane & 2;
  const uint64_t r0 = __shfl_xor_sync(0xffffffffu, b0 ? v[0] : v[1], 1), r1 = __shfl_xor_sync(0xffffffffu, b0 ? v[2] : v[3], 1);
  if (b0) { v[0] = r0; v[2] = r1; }
  else { v[1] = r0; v[3] = r1; }
  const uint64_t r2 = __shfl_xor_sync(0xffffffffu, b1 ? v[0] : v[2], 2), r3 = __shfl_xor_sync(0xffffffffu, b1 ? v[1] : v[3], 2);
  if (b1) { v[0] = r2; v[1] = r3; }
  else { v[2] = r2; v[3] = r3; }
}

// What a lane needs to know of its row before the tile is done.
struct RowInfo {
  bool live;
  int a;            // half-transforms: column of B
  int64_t P;        // and aux row
  int64_t Pl;       // counted from the launch's first
  double sa;        // row scale 2^(e - 35); exchange planes: flavour 0's times 2^(31 - rexp)
  double sa1;       // flavour 1's
};

template <int MODE, class Args>
__device__ __forceinline__ RowInfo row_info(const Args& g, const ProdDev& d, int row) {
  RowInfo r{};
  r.live = row >= d.row0 && row < d.M;
  if (!r.live) return r;
  r.sa = __ldg(d.sa + row);
  if constexpr (MODE != 3) {
    const int Pp = row / g.n;
    r.a = row - Pp * g.n;
    r.Pl = Pp - g.Pl0;
    r.P = g.P0 + r.Pl;
    if constexpr (MODE == 1) r.sa1 = r.sa * __ldg(g.o.tinv[1] + r.a);
    if constexpr (MODE != 2) r.sa *= __ldg(g.o.tinv[0] + r.a);
  }
  return r;
}

// The digits of the tile's values: to_s64's argument is value 2^(31 - e) for the result's row exponent e.
template <int MODE>
__device__ __forceinline__ void store_planes(const HalfArgs& g, const Item& t, const RowInfo& r, int group, int lane,
                                             const double* w) {
  const HalfOut& o = g.o;
  const double* sb = g.p.sb + t.n0;
  if constexpr (MODE == 0) {
    unsigned sq = 0;
    unsigned long long mag = 0;
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int c = unit_col<0>(group, u);
      if (r.live && c < t.nt && t.n0 + c < o.period) {
        double y[8];
        uint2 d[kDigits];
        load8(sb + c, y);
#pragma unroll
        for (int i = 0; i < 8; ++i) y[i] *= w[8 * u + i] * r.sa;
        digits8(y, d);
        uint8_t* dst = o.pl[0][0] + left_at(o.tile_bytes, r.a, static_cast<uint32_t>(r.P * o.period) + t.n0 + c);
#pragma unroll
        for (int p = 0; p < kDigits; ++p) *reinterpret_cast<uint2*>(dst + p * A_PLANE) = d[p];
        sq += square_sum(d[4]);
        mag += top_square_sum(d[0], d[1]);
      }
    }
    if (sq) atomicAdd(o.sq[0] + r.a, static_cast<unsigned long long>(sq));
    if (mag) atomicAdd(o.mag[0] + r.a, mag);
  } else if constexpr (MODE == 1) {
    const int c = t.n0 + unit_col<1>(group, 0), fcols = 2 * static_cast<int>(o.period);
    if (r.live && unit_col<1>(group, 0) < t.nt && c < 2 * fcols) {
      const int fl = c >= fcols ? 1 : 0;
      const int pair = (c - fl * fcols) / 2;
      const double rs = fl ? r.sa1 : r.sa;
      double re[8], im[8], y[8];
      uint2 d[kDigits];
      unsigned sq = 0;
      unsigned long long mag = 0;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const double2 s2 = __ldg(reinterpret_cast<const double2*>(sb + unit_col<1>(group, 0)) + i);
        re[i] = w[2 * i] * rs * s2.x;
        im[i] = w[2 * i + 1] * rs * s2.y;
      }
      const int64_t at = left_at(o.tile_bytes, r.a, static_cast<uint32_t>(r.P * o.period) + pair);
#pragma unroll
      for (int v = 0; v < 4; ++v) {
        uint8_t* base = o.pl[fl][v];
        if (!base) continue;
        // (Re -+ Im) / 2: never longer than the complex value
#pragma unroll
        for (int i = 0; i < 8; ++i) y[i] = v == 0 ? re[i] : v == 1 ? im[i] : 0.5 * (v == 2 ? re[i] - im[i] : re[i] + im[i]);
        digits8(y, d);
#pragma unroll
        for (int p = 0; p < kDigits; ++p) *reinterpret_cast<uint2*>(base + at + p * A_PLANE) = d[p];
        if (v < 2) {
          sq += square_sum(d[4]);
          mag += top_square_sum(d[0], d[1]);
        }
      }
      if (sq) atomicAdd(o.sq[fl] + r.a, static_cast<unsigned long long>(sq));
      if (mag) atomicAdd(o.mag[fl] + r.a, mag);
    }
  } else {
    // result row (Pl, c % per), K byte (c / per) chi + koff + a
    const uint32_t per = static_cast<uint32_t>(o.per), k0 = static_cast<uint32_t>(o.koff) + r.a;
    const double* ti = o.tinv[0];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int c = unit_col<2>(group, u);
      if (c >= t.nt || t.n0 + c >= g.p.N) continue;  // (uniform over the warp)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        uint64_t v[4];
        uint32_t orow[4], kk[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int col = t.n0 + c + 4 * h + i;
          const uint32_t blk = col >= static_cast<int>(per) ? 1 : 0;  // at most two blocks of `per` columns
          const bool ok = r.live && col < g.p.N;
          orow[i] = static_cast<uint32_t>(r.Pl) * per + col - blk * per;
          kk[i] = k0 + blk * static_cast<uint32_t>(o.chi);
          v[i] = ok ? digit_bytes(to_s64(w[8 * u + 4 * h + i] * r.sa, __ldg(sb + c + 4 * h + i) * __ldg(ti + orow[i]))) : 0;
        }
        if (o.quad) {
          // bytes of four K's of one row at a time: a quad of lanes holds four consecutive K's
          quad_transpose(v, lane);
          const uint32_t lo[4] = {static_cast<uint32_t>(v[0]), static_cast<uint32_t>(v[1]), static_cast<uint32_t>(v[2]),
                                  static_cast<uint32_t>(v[3])};
          const uint32_t hi[4] = {static_cast<uint32_t>(v[0] >> 32), static_cast<uint32_t>(v[1] >> 32),
                                  static_cast<uint32_t>(v[2] >> 32), static_cast<uint32_t>(v[3] >> 32)};
          uint32_t pl[4], ph[4];
          transpose4(lo, pl);
          transpose4(hi, ph);
          const int i = lane & 3;
          const uint32_t ro = i == 0 ? orow[0] : i == 1 ? orow[1] : i == 2 ? orow[2] : orow[3];
          const uint32_t ko = (i == 0 ? kk[0] : i == 1 ? kk[1] : i == 2 ? kk[2] : kk[3]) - i;
          if (r.live && t.n0 + c + 4 * h + i < g.p.N) {
            uint8_t* dst = o.pl[0][0] + left_at(o.tile_bytes, ro, ko);
#pragma unroll
            for (int b = 0; b < 4; ++b) {
              *reinterpret_cast<uint32_t*>(dst + (7 - b) * A_PLANE) = pl[b];
              *reinterpret_cast<uint32_t*>(dst + (3 - b) * A_PLANE) = ph[b];
            }
          }
        } else {
#pragma unroll
          for (int i = 0; i < 4; ++i)
            if (r.live && t.n0 + c + 4 * h + i < g.p.N) {
              uint8_t* dst = o.pl[0][0] + left_at(o.tile_bytes, orow[i], kk[i]);
#pragma unroll
              for (int p = 0; p < kDigits; ++p) dst[p * A_PLANE] = static_cast<uint8_t>(v[i] >> (8 * (7 - p)));
            }
        }
      }
    }
  }
}

// MODE 0 / 1 / 2: HalfOut::mode; 3: FP64 results.
template <int MODE, class Args>
__global__ void __launch_bounds__(GEMM_THREADS, 1) oz_gemm_kernel(const __grid_constant__ Args g, int* err) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const Bars bar(smem);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) { mbar_init(&bar.full[s], 1); mbar_init(&bar.empty[s], 1); }
    mbar_init(bar.tfull, 1);
    mbar_init(bar.tempty, EPI_WARPS);
    mbar_init(bar.done, 1);
    fence_barrier_init();
  }
  if (warp == 0) {
    tmem_alloc(bar.tmem_slot, kDigits * kBN);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *bar.tmem_slot;
  bool dead = false;

  if (warp == EPI_WARPS) {
    if (lane == 0) {  // TMA producer
      uint32_t q = 0;
      for (int item = blockIdx.x; item < g.items && !dead; item += gridDim.x) {
        const Item t = decode(g, item);
        const ProdDev& d = prod_of(g, t.p);
        const uint8_t* pa = d.a + t.m0 / kBM * d.a_tile;
        const uint8_t* pb = d.b + t.n0 / d.b_rt * d.b_tile + (t.n0 % d.b_rt) * kBK;
        const uint32_t brow = static_cast<uint32_t>(t.nt * kBK), bytes = A_BYTES + kDigits * brow;
        for (int k = t.k0; k < t.k1; k += kBK, ++q) {
          const int s = q % STAGES;
          if (q >= STAGES && !mbar_wait(&bar.empty[s], ((q / STAGES) & 1) ^ 1, err, ERR_OZ_EMPTY, dead)) break;
          unsigned char* st = smem + s * STAGE_BYTES;
          const int64_t kb = k / kBK;
          mbar_arrive_expect_tx(&bar.full[s], bytes);
          tma_load_1d(st, pa + kb * A_BYTES, A_BYTES, &bar.full[s]);
          if (d.b_rt == kBM) {  // half a 128-row tile: a run per plane
            for (int p = 0; p < kDigits; ++p)
              tma_load_1d(st + A_BYTES + p * brow, pb + kb * A_BYTES + p * A_PLANE, brow, &bar.full[s]);
          } else {
            tma_load_1d(st + A_BYTES, pb + kb * kDigits * brow, kDigits * brow, &bar.full[s]);
          }
        }
      }
    }
  } else if (warp == EPI_WARPS + 1) {
    if (lane == 0) {  // MMA issuer
      uint32_t q = 0, j = 0;
      for (int item = blockIdx.x; item < g.items; item += gridDim.x, ++j) {
        const Item t = decode(g, item);
        if (j > 0) mbar_wait(bar.tempty, (j - 1) & 1, err, ERR_OZ_TEMPTY, dead);
        tc_fence_after();
        for (int k = t.k0; k < t.k1; k += kBK, ++q) {
          const int s = q % STAGES;
          mbar_wait(&bar.full[s], (q / STAGES) & 1, err, ERR_OZ_FULL, dead);
          tc_fence_after();
          if (!dead) issue_stage(tmem, smem_u32(smem) + s * STAGE_BYTES, t.nt, k == t.k0);
          umma_commit(&bar.empty[s]);
        }
        umma_commit(bar.tfull);
        if (dead) break;
      }
      umma_commit(bar.done);
    }
  } else if (warp < EPI_WARPS) {
    const uint32_t tmem_row = tmem + (static_cast<uint32_t>((warp & 3) * 32) << 16);
    uint32_t j = 0;
    for (int item = blockIdx.x; item < g.items; item += gridDim.x, ++j) {
      const Item t = decode(g, item);
      const ProdDev& d = prod_of(g, t.p);
      const int group = warp >> 2;
      const int row = t.m0 + 32 * (warp & 3) + lane;
      const RowInfo r = row_info<MODE>(g, d, row);  // before the wait: its loads are back when the tile is done
      // (the vote also reconverges the warp after the last item's stores)
      const bool ok = __all_sync(0xffffffffu, mbar_wait(bar.tfull, j & 1, err, ERR_OZ_TFULL, dead));
      tc_fence_after();
      double w[16];
      if (ok) drain<MODE>(tmem_row, t.nt, group, w);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar.tempty);
      if (!ok) break;
      if constexpr (MODE == 3) {
        if (r.live) store_f64(d, t, row, group, r.sa, w);
      } else {
        store_planes<MODE>(g, t, r, group, lane, w);
      }
    }
  }
  __syncthreads();
  if (warp == 0) {
    bool ddead = false;
    mbar_wait(bar.done, 0, err, ERR_OZ_DONE, ddead);
    tc_fence_after();
    tmem_dealloc(tmem, kDigits * kBN);
  }
}

// ---------------------------------------------------------------- digits, norms, exponents

__device__ __forceinline__ double coef_at(const CoefSrc& c, int64_t r, int64_t k) {
  switch (c.kind) {
    case 0: return c.src[r * c.ld + k];
    case 1: return c.src[k * c.ld + r];
    case 2: return r / 2 < c.rows ? c.src[((r / 2) * c.ld + c.off + k) * 2 + (r & 1)] : 0.0;
    case 3: {
      const int64_t j = r < c.rows ? r : r - c.rows;
      return c.src[((c.off + k) * c.ld + j) * 2 + (r < c.rows ? 0 : 1)];
    }
    default: {
      const bool im = (k >= c.half) != ((r & 1) != 0);
      const double v = c.src[((k < c.half ? k : k - c.half) * c.ld + r / 2) * 2 + (im ? 1 : 0)];
      return (r & 1) && k < c.half ? -v : v;
    }
  }
}

// Exponent e >= kExpZero with 1.005 x < 2^e for a magnitude x (eight balanced digits end at 127.498 / 128 of
// 2^63); kExpBad when it is not finite.
__device__ __forceinline__ int exponent_of(double x) {
  x *= 1.005;
  if (!(x <= 1.7976931348623157e308)) return kExpBad;
  if (x == 0.0) return kExpZero;
  return max(kExpZero, ilogb(x) + 1);
}

// 2-norm bound from the largest magnitude and the sum of squares (which may have left the normal range).
__device__ __forceinline__ double norm_bound(double mx, double sum, int64_t n) {
  return mx > 1e-140 && mx < 1e140 ? sqrt(sum) * (1.0 + 1e-10) : mx * sqrt(static_cast<double>(n));
}

// fmax that keeps a NaN.
__device__ __forceinline__ double nan_max(double a, double b) { return a != a || b != b ? a + b : fmax(a, b); }

// One CTA of 128 threads per coefficient row; rows at or beyond `valid` are zero rows (padding).
__global__ void __launch_bounds__(128) digitize_rows_kernel(const CoefSrc c, int64_t valid, int64_t K, const Planes pl,
                                                            int64_t row0, double* scale, double* norm) {
  __shared__ double red[3][4];
  const int64_t r = blockIdx.x;
  const int tid = threadIdx.x, warp = tid >> 5;
  const bool live = r < valid;
  // the other part of a complex row
  const int64_t mate = c.kind == 2 ? r ^ 1 : c.kind == 3 ? (r < c.rows ? r + c.rows : r - c.rows) : -1;
  double mx = 0.0, mo = 0.0, sum = 0.0;
  if (live) {
#pragma unroll 4
    for (int64_t k = tid; k < K; k += 128) {
      const double v = coef_at(c, r, k), o = mate >= 0 ? coef_at(c, mate, k) : 0.0;
      mx = nan_max(mx, fabs(v));
      mo = nan_max(mo, fabs(o));
      sum += v * v + o * o;
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    mx = nan_max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    mo = nan_max(mo, __shfl_xor_sync(0xffffffffu, mo, o));
    sum += __shfl_xor_sync(0xffffffffu, sum, o);
  }
  if ((tid & 31) == 0) { red[0][warp] = mx; red[1][warp] = mo; red[2][warp] = sum; }
  __syncthreads();
  mx = nan_max(nan_max(red[0][0], red[0][1]), nan_max(red[0][2], red[0][3]));
  mo = nan_max(nan_max(red[1][0], red[1][1]), nan_max(red[1][2], red[1][3]));
  sum = (red[2][0] + red[2][1]) + (red[2][2] + red[2][3]);
  const int e = exponent_of(mx);
  const double sc = e >= kExpBad ? 0.0 : pow2i(31 - e);
  const int64_t pstride = static_cast<int64_t>(pl.tile_rows(row0 + r)) * kBK;
  uint8_t* base = pl.p + pl.at(row0 + r, 0);
  const int64_t kblock = kDigits * pstride;
  for (int64_t k = tid; k < pl.kblocks() * kBK; k += 128) {
    const double v = live && k < K ? coef_at(c, r, k) : 0.0;
    const uint64_t u = digit_bytes(to_s64(e >= kExpBad ? 0.0 : v, sc));
    uint8_t* dst = base + k / kBK * kblock + (k / 16 % 2) * 128 + k % 16;
#pragma unroll
    for (int p = 0; p < kDigits; ++p) dst[p * pstride] = static_cast<uint8_t>(u >> (8 * (7 - p)));
  }
  if (tid == 0) {
    scale[row0 + r] = scale_of(e, kRowShift);
    norm[row0 + r] = norm_bound(nan_max(mx, mo), sum, 2 * K);
  }
}

__device__ __forceinline__ void atomic_max_nonneg(double* addr, double v) {
  // IEEE order of non-negative doubles equals the order of their bit patterns; a NaN bound orders above all
  atomicMax(reinterpret_cast<unsigned long long*>(addr), static_cast<unsigned long long>(__double_as_longlong(v)));
}

// Columns (P, a) of the three-centre tensor, 32 a CTA: statistics and, with pl.p, digit planes (row P n + a
// minus R0, byte q).  KEEP: the tile stays in shared memory between the two passes over it; otherwise (large n)
// the second pass reads it again.  Bandwidth-bound: 8 bytes read and 8 written per element.
template <bool KEEP, bool STATS>
__global__ void __launch_bounds__(256) digitize_columns_kernel(const double* B, int64_t pitch, int64_t n, int64_t R0, int64_t rows,
                                                               const Planes pl, double* cscale, double* cnorm,
                                                               double* pnorm, int* flag) {
  extern __shared__ double tile[];  // KEEP: [n][32]
  __shared__ double smx[8][32], ssum[8][32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t Rl = blockIdx.x * 32LL + lane, R = R0 + Rl;
  const bool live = Rl < rows;
  const int64_t P = live ? R / n : 0, a = live ? R - P * n : 0;
  const double* p = B + P * pitch + a;
  int e = 0;
  if (STATS || KEEP) {
    double mx = 0.0, sum = 0.0;
    // each warp the q that it converts below: chunks of 32
    for (int64_t q0 = warp * 32; q0 < n; q0 += 256) {
      const int m = static_cast<int>(min(static_cast<int64_t>(32), n - q0));
#pragma unroll 16
      for (int t = 0; t < m; ++t) {
        const double v = live ? __ldg(p + (q0 + t) * n) : 0.0;
        if (KEEP) tile[(q0 + t) * 32 + lane] = v;
        if (STATS) {
          mx = nan_max(mx, fabs(v));
          sum += v * v;
        }
      }
    }
    if (STATS) {
      smx[warp][lane] = mx;
      ssum[warp][lane] = sum;
      __syncthreads();
      mx = smx[0][lane];
      sum = ssum[0][lane];
      for (int w = 1; w < 8; ++w) {
        mx = nan_max(mx, smx[w][lane]);
        sum += ssum[w][lane];
      }
      e = exponent_of(mx);
      if (warp == 0 && live) {
        if (!(mx < 1e140)) *flag = 1;
        cscale[R] = scale_of(e, kRowShift);
        if (mx < 1e140) {
          const double nb = norm_bound(mx, sum, n);
          atomic_max_nonneg(cnorm + a, nb);
          atomic_max_nonneg(pnorm + P, nb);
        }
      }
    }
  }
  if (!pl.p || !live) return;
  // 2^(31 - e), from the scale 2^(e - 35) where the exponents are known already
  const double sc = STATS ? (e >= kExpBad ? 0.0 : pow2i(31 - e)) : 0.0625 / cscale[R];
  for (int64_t q0 = warp * 32; q0 < n; q0 += 256) {
    uint32_t w[kDigits][8];
#pragma unroll
    for (int t4 = 0; t4 < 8; ++t4) {
      uint32_t lo[4], hi[4], o[4];
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const int64_t q = q0 + 4 * t4 + t;
        const double v = q < n ? (KEEP ? tile[q * 32 + lane] : __ldg(p + q * n)) : 0.0;
        const uint64_t u = digit_bytes(to_s64(v, sc));
        lo[t] = static_cast<uint32_t>(u);
        hi[t] = static_cast<uint32_t>(u >> 32);
      }
      transpose4(lo, o);
#pragma unroll
      for (int b = 0; b < 4; ++b) w[7 - b][t4] = o[b];
      transpose4(hi, o);
#pragma unroll
      for (int b = 0; b < 4; ++b) w[3 - b][t4] = o[b];
    }
    uint8_t* dst = pl.p + pl.at(Rl, q0);
#pragma unroll
    for (int d = 0; d < kDigits; ++d) {
      *reinterpret_cast<uint4*>(dst + d * A_PLANE) = make_uint4(w[d][0], w[d][1], w[d][2], w[d][3]);
      *reinterpret_cast<uint4*>(dst + d * A_PLANE + 128) = make_uint4(w[d][4], w[d][5], w[d][6], w[d][7]);
    }
  }
}

// Row scales of a half-transform's result, their exponents, the inverse scales its digits are cut with, and zeroes
// for the digit squares.
__global__ void row_scales_kernel(const double* cnorm, int64_t n, const double* norm, int64_t nnorm, const RowScales out) {
  __shared__ double red[32];
  double m = 0.0;
  for (int64_t i = threadIdx.x; i < nnorm; i += blockDim.x) m = nan_max(m, norm[i]);
  for (int o = 16; o > 0; o >>= 1) m = nan_max(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
  __syncthreads();
  m = red[0];
  for (int w = 1; w < static_cast<int>(blockDim.x >> 5); ++w) m = nan_max(m, red[w]);
  const int64_t padded = round_up_dev(n, 64);
  for (int64_t a = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; a < padded;
       a += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int e = a < n ? exponent_of(cnorm[a] * m) : kExpZero;
    out.scale[a] = scale_of(e, kRowShift);
    if (a >= n) continue;
    out.e[a] = e;
    out.tinv[a] = e >= kExpBad ? 0.0 : pow2i(31 - e);
    out.sq[a] = 0;
    out.rowmax[a] = 0.0;
    out.mag[a] = e >= kExpBad || e <= kExpZero ? kMagNever : 0;
  }
}

constexpr int kRefitWarps = 8, kRefitRows = 16;
struct RefitFlavour {
  const double *B, *c;  // coefficient (j, q): part p at c + j cj + q cq + p
  int64_t pitch, cj, cq, tile_bytes;
  int n;
  uint8_t* pl[4];
  RowScales row;
};
struct RefitArgs {
  RefitFlavour f[4];
  int nf, r;
  int64_t naux, period;
  double need;          // rows with mag below this
};

__device__ __forceinline__ void dmma_8x8x4(double (&c)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n" : "+d"(c[0]), "+d"(c[1]) : "d"(a), "d"(b));
}

// PHASE 0: rowmax = the largest magnitude of every row concerned; 1: its digits at the exponent of that.  A CTA collects the rows
// concerned of 256 at a time; a warp forms T of one aux row for 16 of them and 8 MT coefficient rows at a time on FP64 MMAs (tcgen05
// has no FP64 kind), fragments straight from global memory: neighbouring rows share sectors of B, the coefficients lie in L2.
// Bound: the launch where no row is concerned, the latency of the fragments for a few rows, the FP64 pipe for all of them.
// J and K of n = 400, naux = 1600, 40 orbitals with 0 / 1 / 10 / 100 / 399 such rows: 1.01 / 1.15 / 1.16 / 1.98 / 4.45 ms; four
// components nl = 200, ns = 600, naux = 1000, 40 spinors, 0 / 1 / 10 / 300 of a flavour: 8.1 / 8.6 / 8.7 / 18.3 ms.  Fock builds without
// such rows, two launches more and the sums in the half-transform's epilogue: 1080 -> 1092 us (n = 400), 1925 -> 1929 us (X2C nl = 200),
// 10251 -> 10288 us (four components).
template <int PHASE, int PARTS>
__global__ void __launch_bounds__(32 * kRefitWarps, 2) refit_kernel(const __grid_constant__ RefitArgs g) {
  constexpr int MT = PARTS == 1 ? 5 : 3, SETS = PARTS == 1 ? 1 : 4;
  __shared__ int list[32 * kRefitWarps], total;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, lr = lane >> 2, lc = lane & 3;
  const int64_t warps = static_cast<int64_t>(gridDim.x) * kRefitWarps, me = static_cast<int64_t>(blockIdx.x) * kRefitWarps + warp;
  int64_t seen = 0;  // items dealt out so far
  for (int fi = 0; fi < g.nf; ++fi) {
    const RefitFlavour& f = g.f[fi];
    const int n = f.n;
    for (int row0 = 0; row0 < n; row0 += 32 * kRefitWarps) {
      const bool mine = row0 + tid < n && static_cast<double>(f.row.mag[row0 + tid]) < g.need;
      if (!__syncthreads_or(mine)) continue;
      if (tid == 0) total = 0;
      __syncthreads();
      for (int w = 0; w < kRefitWarps; ++w) {  // in the order of the rows
        if (w == warp) {
          const unsigned vote = __ballot_sync(0xffffffffu, mine);
          if (mine) list[total + __popc(vote & ((1u << lane) - 1))] = row0 + tid;
          __syncwarp();
          if (lane == 0) total += __popc(vote);
        }
        __syncthreads();
      }
      const int count = total, groups = (count + kRefitRows - 1) / kRefitRows;
      const int64_t items = static_cast<int64_t>(groups) * g.naux;
      for (int64_t it = (me + warps - seen % warps) % warps; it < items; it += warps) {
        const int gr = static_cast<int>(it / g.naux) * kRefitRows;
        const int64_t P = it % g.naux;
        if (P == 0 && lane < kRefitRows && gr + lane < count) {
          const int a = list[gr + lane];
          if (PHASE == 0) {
            f.row.sq[a] = 0;
          } else {
            const int e = exponent_of(f.row.rowmax[a]);
            f.row.e[a] = e;
            f.row.scale[a] = scale_of(e, kRowShift);
          }
        }
        const double *b0 = f.B + P * f.pitch + list[min(gr + lr, count - 1)], *b1 = f.B + P * f.pitch + list[min(gr + 8 + lr, count - 1)];
        // this lane's results: rows (list) gr + 8 t + 2 lc + q, coefficient rows j0 + 8 m + lr
        double mx[2][2] = {};
        int e[2][2];
        unsigned long long sq[2][2] = {};
#pragma unroll
        for (int t = 0; t < 2; ++t)
#pragma unroll
          for (int q = 0; q < 2; ++q)
            e[t][q] = PHASE ? exponent_of(f.row.rowmax[list[min(gr + 8 * t + 2 * lc + q, count - 1)]]) : 0;
        for (int j0 = 0; j0 < g.r; j0 += 8 * MT) {
          double acc[MT][PARTS][2][2] = {};
          const double* cp[MT];
#pragma unroll
          for (int m = 0; m < MT; ++m) cp[m] = f.c + min(j0 + 8 * m + lr, g.r - 1) * f.cj;
#pragma unroll 4
          for (int q0 = 0; q0 < n; q0 += 4) {
            const int64_t q = min(q0 + lc, n - 1);
            const bool in = q0 + lc < n;
            const double x0 = in ? b0[q * n] : 0.0, x1 = in ? b1[q * n] : 0.0;
#pragma unroll
            for (int m = 0; m < MT; ++m)
#pragma unroll
              for (int p = 0; p < PARTS; ++p) {
                const double v = cp[m][q * f.cq + p];
                dmma_8x8x4(acc[m][p][0], v, x0);
                dmma_8x8x4(acc[m][p][1], v, x1);
              }
          }
#pragma unroll
          for (int m = 0; m < MT; ++m) {
            const int j = j0 + 8 * m + lr;
            if (j >= g.r) continue;
#pragma unroll
            for (int t = 0; t < 2; ++t)
#pragma unroll
              for (int q = 0; q < 2; ++q) {
                const double re = acc[m][0][t][q], im = acc[m][PARTS - 1][t][q];
                if constexpr (PHASE == 0) {
                  mx[t][q] = fmax(mx[t][q], fmax(fabs(re), fabs(im)));
                } else {
                  const int at = gr + 8 * t + 2 * lc + q;
                  if (at >= count) continue;
                  const double s32 = pow2i(31 - e[t][q]);
                  const int64_t off = left_at(f.tile_bytes, list[at], static_cast<uint32_t>(P * g.period + j));
#pragma unroll
                  for (int v = 0; v < SETS; ++v) {
                    if (!f.pl[v]) continue;
                    const double y = v == 0 ? re : v == 1 ? im : 0.5 * (v == 2 ? re - im : re + im);
                    const uint64_t d = digit_bytes(to_s64(y, s32));
#pragma unroll
                    for (int p = 0; p < kDigits; ++p) f.pl[v][off + p * A_PLANE] = static_cast<uint8_t>(d >> (8 * (7 - p)));
                    const int d4 = static_cast<int8_t>(d >> 24);
                    if (v < 2) sq[t][q] += static_cast<unsigned long long>(d4 * d4);
                  }
                }
              }
          }
        }
#pragma unroll
        for (int t = 0; t < 2; ++t)
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            for (int o = 4; o < 32; o <<= 1) {
              if (PHASE == 0) mx[t][q] = fmax(mx[t][q], __shfl_xor_sync(0xffffffffu, mx[t][q], o));
              else sq[t][q] += __shfl_xor_sync(0xffffffffu, sq[t][q], o);
            }
            const int at = gr + 8 * t + 2 * lc + q;
            if (lr == 0 && at < count) {
              if (PHASE == 0) atomic_max_nonneg(f.row.rowmax + list[at], mx[t][q]);
              else atomicAdd(f.row.sq + list[at], sq[t][q]);
            }
          }
      }
      seen += items;
      __syncthreads();  // the list is written again
    }
  }
}

__global__ void pair_scales_kernel(const double* pnorm0, const double* pnorm1, int64_t naux, const double* norm, int64_t per,
                                   int64_t ntab, int64_t nstride, double* scale, double* tinv) {
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < naux * per;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t P = i / per, j = i - P * per;
    double m = 0.0;
    for (int64_t t = 0; t < ntab; ++t) {
      const double pn = pnorm1 && t >= ntab / 2 ? pnorm1[P] : pnorm0[P];
      m = nan_max(m, pn * norm[t * nstride + j]);
    }
    const int e = exponent_of(m);
    scale[i] = scale_of(e, kRowShift);
    tinv[i] = e >= kExpBad ? 0.0 : pow2i(31 - e);
  }
}

int grid1(int64_t count, int block) {
  return static_cast<int>(std::max<int64_t>(1, std::min<int64_t>((count + block - 1) / block, 16LL * sm_count_current())));
}

template <int MODE, class Args>
void launch_gemm(const Args& g, int* err, cudaStream_t s) {
  auto kern = oz_gemm_kernel<MODE, Args>;
  static std::atomic<bool> attr[kMaxDevices];
  once_per_device(attr, [&] { RR_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES)); });
  kern<<<std::min(g.items, sm_count_current()), GEMM_THREADS, SMEM_BYTES, s>>>(g, err);
  RR_LAUNCH_CHECK();
}

template <bool KEEP, bool STATS>
void launch_columns(const double* B, int64_t pitch, int64_t n, int64_t R0, int64_t rows, const Planes& pl, double* cscale,
                    double* cnorm, double* pnorm, int* flag, cudaStream_t s) {
  auto kern = digitize_columns_kernel<KEEP, STATS>;
  const int smem = KEEP ? static_cast<int>(n * 32 * sizeof(double)) : 0;
  if (KEEP) RR_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kKeepBytes));
  kern<<<static_cast<unsigned>((rows + 31) / 32), 256, smem, s>>>(B, pitch, n, R0, rows, pl, cscale, cnorm, pnorm, flag);
  RR_LAUNCH_CHECK();
}

}  // namespace

void digitize_rows(const CoefSrc& c, int64_t count, int64_t K, const Planes& pl, int64_t row0, double* scale, double* norm,
                   cudaStream_t s) {
  // with the padding rows up to the end of the planes
  digitize_rows_kernel<<<static_cast<unsigned>(pl.rows - row0), 128, 0, s>>>(c, count, K, pl, row0, scale, norm);
  RR_LAUNCH_CHECK();
}

void digitize_columns(const double* B, int64_t pitch, int64_t n, int64_t naux, const Planes* pl, const ColumnStats& st,
                      cudaStream_t s) {
  RR_CUDA(cudaMemsetAsync(st.cnorm, 0, sizeof(double) * n, s));
  RR_CUDA(cudaMemsetAsync(st.pnorm, 0, sizeof(double) * naux, s));
  RR_CUDA(cudaMemsetAsync(st.flag, 0, sizeof(int), s));
  const Planes none;
  if (pl && n * 32 * static_cast<int64_t>(sizeof(double)) <= kKeepBytes) {
    launch_columns<true, true>(B, pitch, n, 0, naux * n, *pl, st.cscale, st.cnorm, st.pnorm, st.flag, s);
  } else {
    launch_columns<false, true>(B, pitch, n, 0, naux * n, pl ? *pl : none, st.cscale, st.cnorm, st.pnorm, st.flag, s);
  }
}

void digitize_range(const double* B, int64_t pitch, int64_t n, int64_t P0, int64_t naux, const Planes& pl, const double* cscale,
                    cudaStream_t s) {
  launch_columns<false, false>(B, pitch, n, P0 * n, naux * n, pl, const_cast<double*>(cscale), nullptr, nullptr, nullptr, s);
}

void row_scales(const double* cnorm, int64_t n, const double* norm, int64_t nnorm, const RowScales& out, cudaStream_t s) {
  row_scales_kernel<<<grid1(n, 256), 256, 0, s>>>(cnorm, n, norm, nnorm, out);
  RR_LAUNCH_CHECK();
}

void refit_rows(const RefitRows* f, int nf, int64_t naux, int64_t r, int64_t period, cudaStream_t s) {
  RR_REQUIRE(nf >= 1 && nf <= 4, RR_ERR_ARG, "oz: flavour count");
  RefitArgs g{};
  const bool pairs = f[0].c.kind == 2;
  for (int i = 0; i < nf; ++i) {
    RefitFlavour& d = g.f[i];
    const CoefSrc& c = f[i].c;
    RR_REQUIRE(c.kind <= 2 && (c.kind == 2) == pairs, RR_ERR_STATE, "oz: coefficient kinds");
    d.B = f[i].B;
    d.pitch = f[i].pitch;
    d.c = c.kind == 2 ? c.src + 2 * c.off : c.src;
    d.cj = c.kind == 0 ? c.ld : c.kind == 1 ? 1 : 2 * c.ld;
    d.cq = c.kind == 0 ? 1 : c.kind == 1 ? c.ld : 2;
    d.tile_bytes = Planes{nullptr, f[i].n, naux * period, kBM}.tile_bytes();
    d.n = static_cast<int>(f[i].n);
    for (int v = 0; v < 4; ++v) d.pl[v] = f[i].pl[v];
    d.row = f[i].row;
  }
  g.nf = nf;
  g.naux = naux;
  g.r = static_cast<int>(r);
  g.period = period;
  g.need = 1073741824.0 / refit_limit(naux * period);  // mag is K_aa in units of 2^(2 e - 30)
  const int grid = 2 * sm_count_current(), threads = 32 * kRefitWarps;
  if (pairs) {
    refit_kernel<0, 2><<<grid, threads, 0, s>>>(g);
    refit_kernel<1, 2><<<grid, threads, 0, s>>>(g);
  } else {
    refit_kernel<0, 1><<<grid, threads, 0, s>>>(g);
    refit_kernel<1, 1><<<grid, threads, 0, s>>>(g);
  }
  RR_LAUNCH_CHECK();
}

void pair_scales(const double* pnorm0, const double* pnorm1, int64_t naux, const double* norm, int64_t per, int64_t ntab,
                 int64_t nstride, double* scale, double* tinv, cudaStream_t s) {
  pair_scales_kernel<<<grid1(naux * per, 256), 256, 0, s>>>(pnorm0, pnorm1, naux, norm, per, ntab, nstride, scale, tinv);
  RR_LAUNCH_CHECK();
}

void half_product(const Planes& b, int64_t Pb, int64_t n, int64_t P0, int64_t naux, const double* cscale,
                  const Planes& coef, const double* coef_scale, int64_t ncol, const HalfOut& out, int* err, cudaStream_t s) {
  RR_REQUIRE(n >= 1 && n <= kOzMaxK && ncol >= 1 && b.rows < (1LL << 31), RR_ERR_ARG, "oz: product size");
  if (naux == 0) return;
  HalfArgs g{};
  // complex planes: column tiles in multiples of 32, so that a warp's half holds whole groups of eight pairs
  const int64_t padded = round_up(ncol, out.mode == 1 ? 32 : 16), r0 = (P0 - Pb) * n, r1 = r0 + naux * n;
  RR_REQUIRE(coef.rows == padded && coef.rt == kBN && b.rt == kBM && b.rows >= r1 && b.k == n && coef.k == n, RR_ERR_STATE,
             "oz: operand shapes");
  ProdDev& d = g.p;
  d.a = b.p;
  d.a_tile = b.tile_bytes();
  d.b = coef.p;
  d.b_tile = coef.tile_bytes();
  d.b_rt = kBN;
  d.row0 = static_cast<int>(r0);
  d.mt0 = static_cast<int>(r0 / kBM);
  d.M = static_cast<int>(r1); d.N = static_cast<int>(ncol); d.K = static_cast<int>(n);
  d.tn = static_cast<int>((padded + kBN - 1) / kBN);
  d.ntl = static_cast<int>(padded - static_cast<int64_t>(d.tn - 1) * kBN);
  d.kchunk = static_cast<int>(round_up(n, kBK));
  d.sa = cscale + Pb * n;
  d.sb = coef_scale;
  g.items = static_cast<int>((r1 + kBM - 1) / kBM - d.mt0) * d.tn;
  g.n = static_cast<int>(n);
  g.P0 = P0;
  g.Pl0 = static_cast<int>(P0 - Pb);
  g.o = out;
  g.o.tile_bytes = out.t.tile_bytes();
  // whole quads of lanes hold four consecutive K bytes of one aux row
  g.o.quad = n % 4 == 0 && out.koff % 4 == 0 && out.chi % 4 == 0;
  if (out.mode == 0) launch_gemm<0>(g, err, s);
  else if (out.mode == 1) launch_gemm<1>(g, err, s);
  else launch_gemm<2>(g, err, s);
}

namespace {

// Output tiles of a product: full column tiles and narrow last ones.
struct TileCount {
  int64_t wide = 0, narrow = 0;
  int ntl = 0;
};
TileCount tile_count(const Prod& p) {
  TileCount t;
  const int64_t tm = (p.M + kBM - 1) / kBM, tn = (p.N + kBN - 1) / kBN;
  t.ntl = static_cast<int>(round_up(p.N - (tn - 1) * kBN, 16));
  const int64_t wide = tn - (t.ntl < kBN ? 1 : 0);
  for (int64_t m = 0; m < tm; ++m) {
    if (!p.sym) {
      t.wide += wide;
      t.narrow += tn - wide;
    } else {
      t.wide += std::max<int64_t>(0, wide - 2 * m);
      t.narrow += 2 * m <= tn - 1 ? tn - wide : 0;
    }
  }
  return t;
}

}  // namespace

void plan_products(Prod* p, int count) {
  // One K range length for the whole list, the one whose items, dealt out in their order, end soonest: cost of an
  // item = its K steps (a step of 64 columns 1, narrower ones from 0.35 on: the A planes are read all the same)
  // plus about two steps for the drain.
  const int sms = sm_count_current();
  TileCount tc[kMaxProds];
  int64_t kmax = 1;
  for (int i = 0; i < count; ++i) {
    tc[i] = tile_count(p[i]);
    kmax = std::max(kmax, p[i].K);
  }
  double best = 0.0;
  int64_t best_len = 0;
  std::vector<double> diff(static_cast<size_t>(sms) + 1);
  for (int64_t parts = (kmax + kOzMaxK - 1) / kOzMaxK, tried = 0; tried < 24; ++tried) {
    const int64_t len = round_up((kmax + parts - 1) / parts, kBK);
    if (tried > 0 && len < 512) break;
    std::fill(diff.begin(), diff.end(), 0.0);
    double all = 0.0;
    int64_t at = 0;
    for (int narrow = 0; narrow < 2; ++narrow)
      for (int i = 0; i < count; ++i) {
        const int64_t splits = (p[i].K + len - 1) / len, n = (narrow ? tc[i].narrow : tc[i].wide) * splits;
        const double c = static_cast<double>((p[i].K + splits - 1) / splits) / kBK *
                             (narrow ? 0.35 + 0.65 * tc[i].ntl / kBN : 1.0) + 2.0;
        all += c * static_cast<double>(n / sms);
        const int64_t rem = n % sms, end = at + rem;
        diff[at] += c;
        diff[std::min<int64_t>(end, sms)] -= c;
        if (end > sms) { diff[0] += c; diff[end - sms] -= c; }
        at = end % sms;
      }
    double worst = 0.0, run = 0.0;
    for (int c = 0; c < sms; ++c) worst = std::max(worst, run += diff[c]);
    if (best_len == 0 || all + worst < best) { best = all + worst; best_len = len; }
    parts += std::max<int64_t>(1, parts / 8);
  }
  for (int i = 0; i < count; ++i) {
    const int64_t splits = std::max<int64_t>(1, (p[i].K + best_len - 1) / best_len);
    p[i].kchunk = round_up((p[i].K + splits - 1) / splits, kBK);
    p[i].splits = static_cast<int>((p[i].K + p[i].kchunk - 1) / p[i].kchunk);
  }
}

void run_products(const Prod* p, int count, int* err, cudaStream_t s) {
  RR_REQUIRE(count >= 1 && count <= kMaxProds, RR_ERR_ARG, "oz: product count");
  GemmArgs g{};
  int items = 0;
  for (int i = 0; i < count; ++i) {
    const Prod& q = p[i];
    RR_REQUIRE(q.kchunk > 0 && q.kchunk <= kOzMaxK && q.kchunk % kBK == 0 && q.a.k == q.K && q.b.k == q.K &&
                   q.a.rt == kBM && q.a.rows >= q.M && q.b.rows >= q.N,
               RR_ERR_STATE, "oz: operand shapes");
    RR_REQUIRE(q.M < (1LL << 31) && q.K < (1LL << 31), RR_ERR_ARG, "oz: product size");
    ProdDev& d = g.p[i];
    d.a = q.a.p; d.b = q.b.p;
    d.a_tile = q.a.tile_bytes(); d.b_tile = q.b.tile_bytes();
    d.b_rt = q.b.rt;
    d.M = static_cast<int>(q.M); d.N = static_cast<int>(q.N); d.K = static_cast<int>(q.K);
    d.tn = static_cast<int>((q.N + kBN - 1) / kBN);
    d.ntl = static_cast<int>(round_up(q.N - static_cast<int64_t>(d.tn - 1) * kBN, 16));
    d.sym = q.sym; d.negate_odd = q.negate_odd;
    d.kchunk = static_cast<int>(q.kchunk);
    d.sa = q.sa; d.sb = q.sb;
    d.out = q.out; d.ldo = q.ldo; d.sstride = q.sstride;
  }
  for (int narrow = 0; narrow < 2; ++narrow)
    for (int i = 0; i < count; ++i) {
      const TileCount t = tile_count(p[i]);
      const int64_t tiles = narrow ? t.narrow : t.wide;
      if (tiles == 0) continue;
      g.seg[g.segs++] = Seg{items, i, narrow, static_cast<int>(tiles)};
      items += static_cast<int>(tiles) * p[i].splits;
    }
  g.items = items;
  if (items == 0) return;
  launch_gemm<3>(g, err, s);
}

}  // namespace oz
}  // namespace rr
