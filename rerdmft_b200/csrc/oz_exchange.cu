// The exchange of the FP64 Fock builds and the FP64 MO transforms as products of digit planes on the INT8
// tensor cores (oz.cuh): scratch layout, product lists, and the kernels that finish their split-K sums.
#include <algorithm>

#include "mo_store.cuh"
#include "oz.cuh"
#include "oz_paths.cuh"

namespace rr {

namespace {

using oz::kDigits;

// Byte sub-buffers of the handle's digit scratch.
struct Carve {
  DevBuf<uint8_t>& buf;
  int64_t used = 0;
  explicit Carve(DevBuf<uint8_t>& b) : buf(b) {}
  int64_t take(int64_t bytes) {
    const int64_t at = used;
    used += round_up(std::max<int64_t>(bytes, 16), 256);
    return at;
  }
  // false when the device has no room (the caller keeps the FP64 path, which may need less)
  bool commit() {
    if (static_cast<int64_t>(buf.n) >= used) return true;
    try {
      buf.alloc(static_cast<size_t>(used));
    } catch (const Error& e) {
      if (e.code != RR_ERR_CUDA) throw;
      cudaGetLastError();
      return false;
    }
    return true;
  }
  template <typename T>
  T* at(int64_t off) const { return reinterpret_cast<T*>(buf.p + off); }
};

// Planes of a left operand (128-row tiles) and of a coefficient operand.
oz::Planes left(uint8_t* p, int64_t rows, int64_t k) { return oz::Planes{p, rows, k, oz::kBM}; }
oz::Planes coefs(uint8_t* p, int64_t rows, int64_t k) { return oz::Planes{p, rows, k, oz::kBN}; }
int64_t left_bytes(int64_t rows, int64_t k) { return left(nullptr, rows, k).bytes(); }
int64_t coef_bytes(int64_t rows, int64_t k) { return coefs(nullptr, rows, k).bytes(); }
// Zeroes the last, partly filled K block before the planes are written: a product of the planes with themselves
// reads all of it.
void clear_tail(const oz::Planes& p, cudaStream_t s) {
  if (p.k % oz::kBK == 0) return;
  const int64_t blk = static_cast<int64_t>(kDigits) * oz::kBM * oz::kBK;
  RR_CUDA(cudaMemset2DAsync(p.p + (p.kblocks() - 1) * blk, static_cast<size_t>(p.tile_bytes()), 0, static_cast<size_t>(blk),
                            static_cast<size_t>((p.rows + oz::kBM - 1) / oz::kBM), s));
}

int grid_of(int64_t count) { return static_cast<int>(std::max<int64_t>(1, std::min<int64_t>((count + 255) / 256, 1184))); }

// Aux rows whose digit planes are at most 64 MB: what one range digitizes into scratch, to be read back from L2.
int64_t range_rows(int64_t naux, int64_t n) {
  return std::max<int64_t>(1, std::min<int64_t>(naux, (64LL << 20) / (kDigits * n * round_up(n, oz::kBK))));
}

// Calls f(P0, count, planes, aux row of the planes' row 0) over tensor t: once with the resident planes, else range
// by range with planes made in `scratch`.
template <class F>
void over_planes(rr_ri_store* h, int t, int64_t n, uint8_t* scratch, cudaStream_t s, F&& f) {
  auto& z = h->oz[t];
  const int64_t naux = h->naux;
  if (z.planes) {
    f(int64_t{0}, naux, left(z.planes, naux * n, n));
    return;
  }
  const int64_t pc = range_rows(naux, n);
  for (int64_t P0 = 0; P0 < naux; P0 += pc) {
    const int64_t cnt = std::min(pc, naux - P0);
    const oz::Planes b = left(scratch, cnt * n, n);
    oz::digitize_range(h->B[t].p, h->pitch[t], n, P0, cnt, b, z.cscale, s);
    f(P0, cnt, b);
  }
}
// Scratch bytes over_planes needs.
int64_t over_bytes(rr_ri_store* h, int t, int64_t n) {
  return h->oz[t].planes ? 0 : left_bytes(range_rows(h->naux, n) * n, n);
}

// One allocation for the row scales of n rows.
int64_t row_bytes(int64_t n) { return (8 * 5 + 4) * round_up(n, 64); }
oz::RowScales rows_at(double* p, int64_t n) {
  const int64_t np = round_up(n, 64);
  oz::RowScales r;
  r.scale = p;
  r.tinv = p + np;
  r.sq = reinterpret_cast<unsigned long long*>(p + 2 * np);
  r.mag = r.sq + np;
  r.rowmax = p + 4 * np;
  r.e = reinterpret_cast<int*>(p + 5 * np);
  return r;
}

// The digit pair (4, 4) of a row with itself: sq 2^(2 e - 78).
__device__ __forceinline__ double square_term(const unsigned long long* sq, const int* rexp, int64_t a) {
  return scalbn(static_cast<double>(sq[a]), 2 * rexp[a] - 78);
}

// K = sum over the K ranges of the upper-triangle products, both triangles.
__global__ void sum_symmetric_kernel(double* K, const double* part, int splits, int64_t sstride, int64_t ldo, int64_t n,
                                     const unsigned long long* sq, const int* rexp) {
  for (int64_t idx = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; idx < n * n;
       idx += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t a = idx / n, b = idx % n;
    if (a > b) continue;
    double v = 0.0;
    for (int s = 0; s < splits; ++s) v += part[s * sstride + a * ldo + b];
    if (a == b) v += square_term(sq, rexp, a);
    K[a * n + b] = v;
    K[b * n + a] = v;
  }
}

// One exchange block (f, u) of the relativistic builds, from three products:
//   f == u:  Re K = P0 + P1 (symmetric, upper triangles), Im K = P2 - P2^T (P2 = Re^T Im)
//   f != u:  Re K = P0 + P1, Im K = 4 P2 - P0 + P1        (4 P2 = (Re - Im)^T (Re + Im), Gauss)
struct BlockDev {
  const double* p[3];
  int splits[3];
  int64_t sstride[3], ldo[3];
  int64_t of, ou, ff, fu;
  const double* j;  // Coulomb block added on the diagonal (or null)
  const unsigned long long* sq;  // diag: digit squares and exponents of the flavour
  const int* rexp;
  int diag;
};
struct BlockList {
  BlockDev b[10];
  int count;
};

__device__ __forceinline__ double sum_splits(const BlockDev& b, int w, int64_t r, int64_t c) {
  double v = 0.0;
  const double* p = b.p[w] + r * b.ldo[w] + c;
  for (int s = 0; s < b.splits[w]; ++s) v += p[s * b.sstride[w]];
  return v;
}

// G (complex ntot x ntot) block (f, u) = sgn K (+ J), and for f != u the conjugate block (u, f).
__global__ void place_blocks_kernel(const __grid_constant__ BlockList l, double* G, int64_t ntot, double sgn) {
  const BlockDev& b = l.b[blockIdx.y];
  for (int64_t idx = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; idx < b.ff * b.fu;
       idx += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t r = idx / b.fu, c = idx % b.fu;
    double re, im;
    if (b.diag) {
      if (r > c) continue;  // written with (c, r)
      re = sum_splits(b, 0, r, c) + sum_splits(b, 1, r, c);
      if (r == c) re += square_term(b.sq, b.rexp, r);
      im = r == c ? 0.0 : sum_splits(b, 2, r, c) - sum_splits(b, 2, c, r);
    } else {
      const double p0 = sum_splits(b, 0, r, c), p1 = sum_splits(b, 1, r, c);
      re = p0 + p1;
      im = 4.0 * sum_splits(b, 2, r, c) - p0 + p1;
    }
    re *= sgn;
    im *= sgn;
    double* g = G + ((b.of + r) * ntot + b.ou + c) * 2;
    double* t = G + ((b.ou + c) * ntot + b.of + r) * 2;
    t[0] = re + (b.j ? b.j[c * b.fu + r] : 0.0);
    t[1] = -im;
    g[0] = re + (b.j ? b.j[idx] : 0.0);
    g[1] = im;
  }
}

}  // namespace

namespace {

// Column statistics and digit planes of tensor t (n x n rows); synchronises s.
void oz_prepare(rr_ri_store* h, int t, int64_t n, cudaStream_t s) {
  auto& z = h->oz[t];
  if (h->naux == 0 || n < kOzMinDim || n > oz::kOzMaxK || h->naux * n >= (1LL << 31)) {
    z.made = true;
    return;
  }
  Carve c(z.stats);
  const int64_t o_cs = c.take(8 * h->naux * n), o_cn = c.take(8 * n), o_pn = c.take(8 * h->naux), o_flag = c.take(4);
  if (!c.commit()) return;  // no room now
  size_t free_b = 0, total_b = 0;
  RR_CUDA(cudaMemGetInfo(&free_b, &total_b));
  const int64_t bytes = left_bytes(h->naux * n, n);
  Carve cp(z.buf);
  cp.take(bytes);
  const bool keep = static_cast<double>(bytes) <= 0.25 * static_cast<double>(free_b) && cp.commit();  // else: ranges
  z.cscale = c.at<double>(o_cs);
  z.cnorm = c.at<double>(o_cn);
  z.pnorm = c.at<double>(o_pn);
  int* flag = c.at<int>(o_flag);
  const oz::Planes pl = left(keep ? z.buf.p : nullptr, h->naux * n, n);
  oz::digitize_columns(h->B[t].p, h->pitch[t], n, h->naux, keep ? &pl : nullptr,
                       oz::ColumnStats{z.cscale, z.cnorm, z.pnorm, flag}, s);
  int bad = 0;
  RR_CUDA(cudaMemcpyAsync(&bad, flag, sizeof(int), cudaMemcpyDeviceToHost, s));
  RR_CUDA(cudaStreamSynchronize(s));
  z.ok = bad == 0;
  z.made = true;
  if (z.ok) {
    z.planes = keep ? z.buf.p : nullptr;
  } else {
    z.stats.release();
    z.buf.release();
  }
}

// Every store, for release_idle_planes.
struct StoreList {
  std::mutex mu;
  std::vector<rr_ri_store*> all;
};
StoreList& stores() {
  static StoreList* l = new StoreList();  // never destroyed: handles may outlive static destructors
  return *l;
}

}  // namespace

bool release_idle_planes(int device) noexcept {
  bool any = false;
  StoreList& l = stores();
  std::lock_guard<std::mutex> lock(l.mu);
  for (rr_ri_store* h : l.all) {
    std::lock_guard<std::mutex> own(h->oz_mu);
    if (h->oz_users > 0 || h->oz_pinned || h->ctx.device != device) continue;
    for (auto& z : h->oz)
      if (z.planes) {
        z.planes = nullptr;
        z.buf.release();  // (waits for the products queued on it)
        any = true;
      }
  }
  return any;
}

OzUse::OzUse(rr_ri_store* h, cudaStream_t s) : h_(h) {
  if (h->oz_off) {
    h_ = nullptr;
    return;
  }
  cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
  RR_CUDA(cudaStreamIsCapturing(s, &capture));
  const bool captured = capture != cudaStreamCaptureStatusNone;
  {
    std::lock_guard<std::mutex> lock(h->oz_mu);
    ++h->oz_users;
    if (captured) h->oz_pinned = true;
  }
  try {
    std::lock_guard<std::mutex> lock(h->oz_making);
    ok = true;
    for (int t = 0; t < h->ntens; ++t) {
      if (!h->oz[t].made && !captured) oz_prepare(h, t, t ? h->ns : h->n, s);
      ok = ok && h->oz[t].ok;
    }
  } catch (...) {
    std::lock_guard<std::mutex> lock(h->oz_mu);
    --h->oz_users;
    throw;
  }
}

OzUse::~OzUse() {
  if (!h_) return;
  std::lock_guard<std::mutex> lock(h_->oz_mu);
  --h_->oz_users;
}

bool oz_exchange_nonrel(rr_ri_store* h, const double* Ct, int64_t ldct, bool ct_transposed, int64_t nocc, double* K,
                        cudaStream_t s) {
  const int64_t n = h->n, naux = h->naux;
  const int64_t per = round_up(nocc, 8), ncp = round_up(per, 16), kk = naux * per, ldo = round_up(n, 4);
  if (kk >= (1LL << 31)) return false;
  oz::Prod pr;
  pr.M = n; pr.N = n; pr.K = kk; pr.sym = 1;
  oz::plan_products(&pr, 1);
  Carve c(h->ozbuf);
  const int64_t o_coef = c.take(coef_bytes(ncp, n)), o_cs = c.take(8 * ncp), o_norm = c.take(8 * ncp),
                o_row = c.take(row_bytes(n)), o_t = c.take(left_bytes(n, kk)),
                o_part = c.take(8 * pr.splits * n * ldo), o_b = c.take(over_bytes(h, 0, n));
  if (!c.commit()) return false;
  const oz::Planes coef = coefs(c.at<uint8_t>(o_coef), ncp, n), T = left(c.at<uint8_t>(o_t), n, kk);
  double *cs = c.at<double>(o_cs), *norm = c.at<double>(o_norm);
  const oz::RowScales row = rows_at(c.at<double>(o_row), n);
  oz::CoefSrc src;
  src.src = Ct; src.ld = ldct; src.kind = ct_transposed ? 1 : 0;
  oz::digitize_rows(src, nocc, n, coef, 0, cs, norm, s);
  oz::row_scales(h->oz[0].cnorm, n, norm, ncp, row, s);
  oz::HalfOut out;
  out.mode = 0;
  out.period = per;
  out.t = T;
  out.pl[0][0] = T.p;
  out.tinv[0] = row.tinv;
  out.sq[0] = row.sq;
  out.mag[0] = row.mag;
  clear_tail(T, s);
  over_planes(h, 0, n, c.at<uint8_t>(o_b), s, [&](int64_t P0, int64_t cnt, const oz::Planes& b) {
    oz::half_product(b, P0, n, P0, cnt, h->oz[0].cscale, coef, cs, per, out, h->status.p, s);
  });
  oz::RefitRows rf;
  rf.B = h->B[0].p; rf.pitch = h->pitch[0]; rf.n = n;
  rf.c = src;
  rf.pl[0] = T.p;
  rf.row = row;
  oz::refit_rows(&rf, 1, naux, nocc, per, s);
  prof_mark(h, 2, s);
  pr.a = T; pr.b = T;
  pr.sa = row.scale; pr.sb = row.scale;
  pr.out = c.at<double>(o_part);
  pr.ldo = ldo; pr.sstride = n * ldo;
  oz::run_products(&pr, 1, h->status.p, s);
  sum_symmetric_kernel<<<grid_of(n * n), 256, 0, s>>>(K, pr.out, pr.splits, pr.sstride, ldo, n, row.sq, row.e);
  RR_LAUNCH_CHECK();
  return true;
}

bool oz_exchange_rel(rr_ri_store* h, int nf, const int64_t* off, const int64_t* fs, const int* tens, int64_t ntot,
                     const double* Ct, int64_t r, double* const* J, cudaEvent_t j_ready, double* G, double sgn,
                     cudaStream_t s) {
  const int64_t naux = h->naux;
  const int64_t per = round_up(std::max<int64_t>(r, 1), 8), kk = naux * per;
  if (r == 0 || kk >= (1LL << 31) || nf < 2 || nf > 4) return false;
  // two flavours per tensor, side by side
  for (int f = 0; f < nf; f += 2)
    if (f + 1 >= nf || tens[f] != tens[f + 1] || fs[f] != fs[f + 1]) return false;
  const OzUse use(h, s);
  if (!use.ok) return false;
  const int ng = nf / 2;
  const int64_t ncol = 4 * per, ncp = round_up(ncol, 32);

  oz::Prod pr[30];
  int np = 0;
  for (int f = 0; f < nf; ++f)
    for (int u = f; u < nf; ++u)
      for (int w = 0; w < 3; ++w) {
        oz::Prod& p = pr[np++];
        p.M = fs[f]; p.N = fs[u]; p.K = kk;
        p.sym = f == u && w < 2;
      }
  oz::plan_products(pr, np);

  Carve c(h->ozbuf);
  int64_t o_coef[2], o_cs[2], o_norm[2], o_row[4], o_t[4][4], o_part[30], o_b[2];
  for (int g = 0; g < ng; ++g) {
    o_coef[g] = c.take(coef_bytes(ncp, fs[2 * g]));
    o_cs[g] = c.take(8 * ncp);
    o_norm[g] = c.take(8 * ncp);
    o_b[g] = c.take(over_bytes(h, tens[2 * g], fs[2 * g]));
  }
  for (int f = 0; f < nf; ++f) {
    o_row[f] = c.take(row_bytes(fs[f]));
    for (int v = 0; v < 4; ++v) {
      const bool want = v < 2 || (v == 2 ? f + 1 < nf : f > 0);
      o_t[f][v] = want ? c.take(left_bytes(fs[f], kk)) : -1;
    }
  }
  for (int i = 0; i < np; ++i) {
    pr[i].ldo = round_up(pr[i].N, 4);
    pr[i].sstride = pr[i].M * pr[i].ldo;
    o_part[i] = c.take(8 * pr[i].splits * pr[i].sstride);
  }
  if (!c.commit()) return false;
  oz::RowScales row[4];
  oz::RefitRows rf[4];
  for (int f = 0; f < nf; ++f) row[f] = rows_at(c.at<double>(o_row[f]), fs[f]);

  for (int g = 0; g < ng; ++g) {
    const int f0 = 2 * g, t = tens[f0];
    const int64_t n = fs[f0];
    const oz::Planes coef = coefs(c.at<uint8_t>(o_coef[g]), ncp, n);
    double *cs = c.at<double>(o_cs[g]), *norm = c.at<double>(o_norm[g]);
    oz::HalfOut out;
    out.mode = 1;
    out.period = per;
    out.t = left(nullptr, n, kk);
    for (int k = 0; k < 2; ++k) {
      const int f = f0 + k;
      oz::CoefSrc src;
      src.src = Ct; src.ld = ntot; src.off = off[f]; src.kind = 2; src.rows = r;
      oz::digitize_rows(src, 2 * per, n, coef, k * 2 * per, cs, norm, s);
      for (int v = 0; v < 4; ++v) out.pl[k][v] = o_t[f][v] >= 0 ? c.at<uint8_t>(o_t[f][v]) : nullptr;
      out.tinv[k] = row[f].tinv;
      out.sq[k] = row[f].sq;
      out.mag[k] = row[f].mag;
      rf[f].B = h->B[t].p; rf[f].pitch = h->pitch[t]; rf[f].n = n;
      rf[f].c = src;
      for (int v = 0; v < 4; ++v) rf[f].pl[v] = out.pl[k][v];
      rf[f].row = row[f];
    }
    for (int k = 0; k < 2; ++k)
      oz::row_scales(h->oz[t].cnorm, n, norm + k * 2 * per, 2 * per, row[f0 + k], s);
    for (int k = 0; k < 2; ++k)
      for (int v = 0; v < 4; ++v)
        if (out.pl[k][v]) clear_tail(left(out.pl[k][v], n, kk), s);
    over_planes(h, t, n, c.at<uint8_t>(o_b[g]), s, [&](int64_t P0, int64_t cnt, const oz::Planes& b) {
      oz::half_product(b, P0, n, P0, cnt, h->oz[t].cscale, coef, cs, ncol, out, h->status.p, s);
    });
  }
  oz::refit_rows(rf, nf, naux, r, per, s);
  prof_mark(h, 2, s);

  auto planes = [&](int f, int v) { return left(c.at<uint8_t>(o_t[f][v]), fs[f], kk); };
  BlockList bl{};
  int i = 0;
  int64_t most = 1;
  for (int f = 0; f < nf; ++f)
    for (int u = f; u < nf; ++u) {
      BlockDev& b = bl.b[bl.count++];
      b.of = off[f]; b.ou = off[u]; b.ff = fs[f]; b.fu = fs[u];
      b.diag = f == u;
      b.sq = row[f].sq;
      b.rexp = row[f].e;
      b.j = f == u && J ? J[tens[f]] : nullptr;
      most = std::max(most, b.ff * b.fu);
      for (int w = 0; w < 3; ++w, ++i) {
        const int va = f == u ? (w == 1 ? 1 : 0) : w, vb = f == u ? (w == 0 ? 0 : 1) : (w == 2 ? 3 : w);
        pr[i].a = planes(f, va);
        pr[i].b = planes(u, vb);
        pr[i].sa = row[f].scale;
        pr[i].sb = row[u].scale;
        pr[i].out = c.at<double>(o_part[i]);
        b.p[w] = pr[i].out;
        b.splits[w] = pr[i].splits;
        b.sstride[w] = pr[i].sstride;
        b.ldo[w] = pr[i].ldo;
      }
    }
  oz::run_products(pr, np, h->status.p, s);
  if (J && j_ready) RR_CUDA(cudaStreamWaitEvent(s, j_ready, 0));
  place_blocks_kernel<<<dim3(grid_of(most), bl.count), 256, 0, s>>>(bl, G, ntot, sgn);
  RR_LAUNCH_CHECK();
  return true;
}

namespace {

// Aux rows of one range of an MO transform: the digit planes of the intermediate (and of B where they are made here)
// stay below 96 MB, so that the products read them from L2.
int64_t mo_range(int64_t naux, int64_t bytes_per_row) {
  return std::max<int64_t>(1, std::min<int64_t>(naux, (96LL << 20) / std::max<int64_t>(bytes_per_row, 1)));
}

// A range of at most `most` aux rows whose two launches (n rows an aux row, n columns) fill their last round of tiles: a CTA
// walks whole tiles, and 75 rows of n = 400 are 1645 of them, 11.1 a CTA, 74 rows 1624, 10.97.  n = 400, naux = 1600: 8.0 ->
// 7.6 ms.  (Not for the four-component transform: its five launches of different shapes gain nothing, 5.13 / 5.17 ms.)
int64_t mo_even_range(int64_t naux, int64_t most, int64_t n) {
  if (most >= naux) return most;
  const int64_t sms = sm_count_current();
  int64_t best = most;
  double best_cost = 0.0;
  for (int64_t pc = std::max<int64_t>(1, most - most / 4); pc <= most; ++pc) {
    const int64_t tiles = (pc * n + oz::kBM - 1) / oz::kBM * ((n + oz::kBN - 1) / oz::kBN);
    const double cost = static_cast<double>((tiles + sms - 1) / sms) / static_cast<double>(pc);
    if (best_cost == 0.0 || cost <= best_cost) {
      best_cost = cost;
      best = pc;
    }
  }
  return best;
}

// out[P] = C^T B^P C for device C (n x n).
bool mo_real(const double* B, int64_t pitch, int64_t n, int64_t naux, const double* cscale, const double* pnorm, const uint8_t* resident,
             const double* C, double* out, Carve& c, int* err, cudaStream_t s) {
  const int64_t ncp = round_up(n, 16), per_row = kDigits * n * round_up(n, oz::kBK);
  const int64_t pc = mo_even_range(naux, mo_range(naux, resident ? per_row : 2 * per_row), n);
  const int64_t o_coef = c.take(coef_bytes(ncp, n)), o_cs = c.take(8 * ncp), o_norm = c.take(8 * ncp),
                o_row = c.take(16 * naux * n), o_y = c.take(left_bytes(pc * n, n)),
                o_b = c.take(resident ? 0 : left_bytes(pc * n, n));
  if (!c.commit()) return false;
  const oz::Planes coef = coefs(c.at<uint8_t>(o_coef), ncp, n);
  double *cs = c.at<double>(o_cs), *norm = c.at<double>(o_norm), *scale = c.at<double>(o_row), *tinv = scale + naux * n;
  oz::CoefSrc src;
  src.src = C; src.ld = n; src.kind = 1;
  oz::digitize_rows(src, n, n, coef, 0, cs, norm, s);
  oz::pair_scales(pnorm, nullptr, naux, norm, n, 1, ncp, scale, tinv, s);
  for (int64_t P0 = 0; P0 < naux; P0 += pc) {
    const int64_t cnt = std::min(pc, naux - P0);
    oz::Planes b = left(const_cast<uint8_t*>(resident), naux * n, n);
    if (!resident) {
      b = left(c.at<uint8_t>(o_b), cnt * n, n);
      oz::digitize_range(B, pitch, n, P0, cnt, b, cscale, s);
    }
    const oz::Planes Y = left(c.at<uint8_t>(o_y), cnt * n, n);
    oz::HalfOut o;
    o.mode = 2;
    o.t = Y;
    o.pl[0][0] = Y.p;
    o.tinv[0] = tinv + P0 * n;
    o.per = n;
    oz::half_product(b, resident ? 0 : P0, n, P0, cnt, cscale, coef, cs, n, o, err, s);
    oz::Prod p;
    p.a = Y; p.b = coef;
    p.sa = scale + P0 * n; p.sb = cs;
    p.M = cnt * n; p.N = n; p.K = n;
    p.kchunk = round_up(n, oz::kBK);
    p.out = out + P0 * n * n;
    p.ldo = n;
    oz::run_products(&p, 1, err, s);
  }
  return true;
}

}  // namespace

bool oz_mo_build_nonrel(rr_ri_store* ri, const double* Cd, rr_mo_store* m, cudaStream_t s) {
  if (!oz_worth(ri->naux, ri->n, ri->n)) return false;
  const OzUse use(ri, s);
  if (!use.ok) return false;
  auto& z = ri->oz[0];
  Carve c(m->ozbuf);
  return mo_real(ri->B[0].p, ri->pitch[0], ri->n, ri->naux, z.cscale, z.pnorm, z.planes, Cd, m->B.p, c, ri->status.p, s);
}

bool oz_mo_build_ukb(rr_ri_store* ri, const double* cd, int64_t nt, rr_mo_store* m, cudaStream_t s) {
  const int64_t nl = ri->n, ns = ri->ns, naux = ri->naux, nu = 2 * nl + 2 * ns;
  const int64_t off[4] = {0, nl, 2 * nl, 2 * nl + ns}, fs[4] = {nl, nl, ns, ns};
  const int tens[4] = {0, 0, 1, 1};
  if (2 * nu > oz::kOzMaxK || nt == 0 || naux == 0) return false;
  const OzUse use(ri, s);
  if (!use.ok) return false;
  const int64_t nc = 2 * nt, ncp = round_up(nc, 16);
  int64_t made = 0;
  for (int t = 0; t < 2; ++t)
    if (!ri->oz[t].planes) made += left_bytes(t ? ns : nl, t ? ns : nl);
  const int64_t pc = mo_range(naux, kDigits * nt * round_up(2 * nu, oz::kBK) + made);
  Carve c(m->ozbuf);
  int64_t o_coef[4], o_b[2];
  for (int f = 0; f < 4; ++f) o_coef[f] = c.take(coef_bytes(ncp, fs[f]));
  for (int t = 0; t < 2; ++t) {
    const int64_t n = t ? ns : nl;
    o_b[t] = c.take(ri->oz[t].planes ? 0 : left_bytes(pc * n, n));
  }
  const int64_t o_cs = c.take(8 * 5 * ncp), o_norm = c.take(8 * 5 * ncp), o_row = c.take(16 * naux * nt),
                o_cc = c.take(coef_bytes(ncp, 2 * nu)), o_y = c.take(left_bytes(pc * nt, 2 * nu));
  if (!c.commit()) return false;
  double *cs = c.at<double>(o_cs), *norm = c.at<double>(o_norm), *scale = c.at<double>(o_row), *tinv = scale + naux * nt;
  oz::Planes coef[4];
  for (int f = 0; f < 4; ++f) {
    coef[f] = coefs(c.at<uint8_t>(o_coef[f]), ncp, fs[f]);
    oz::CoefSrc src;
    src.src = cd; src.ld = nt; src.off = off[f]; src.kind = 3; src.rows = nt;
    oz::digitize_rows(src, nc, fs[f], coef[f], 0, cs + f * ncp, norm + f * ncp, s);
  }
  const oz::Planes cc = coefs(c.at<uint8_t>(o_cc), ncp, 2 * nu);
  oz::CoefSrc src;
  src.src = cd; src.ld = nt; src.kind = 4; src.half = nu;
  oz::digitize_rows(src, nc, 2 * nu, cc, 0, cs + 4 * ncp, norm + 4 * ncp, s);
  oz::pair_scales(ri->oz[0].pnorm, ri->oz[1].pnorm, naux, norm, nt, 4, ncp, scale, tinv, s);
  for (int64_t P0 = 0; P0 < naux; P0 += pc) {
    const int64_t cnt = std::min(pc, naux - P0);
    const oz::Planes Y = left(c.at<uint8_t>(o_y), cnt * nt, 2 * nu);
    oz::Planes b[2];
    for (int t = 0; t < 2; ++t) {
      const int64_t n = t ? ns : nl;
      b[t] = left(ri->oz[t].planes, naux * n, n);
      if (ri->oz[t].planes) continue;
      b[t] = left(c.at<uint8_t>(o_b[t]), cnt * n, n);
      oz::digitize_range(ri->B[t].p, ri->pitch[t], n, P0, cnt, b[t], ri->oz[t].cscale, s);
    }
    for (int f = 0; f < 4; ++f) {
      oz::HalfOut o;
      o.mode = 2;
      o.t = Y;
      o.pl[0][0] = Y.p;
      o.tinv[0] = tinv + P0 * nt;
      o.per = nt;
      o.chi = nu;
      o.koff = off[f];
      oz::half_product(b[tens[f]], ri->oz[tens[f]].planes ? 0 : P0, fs[f], P0, cnt, ri->oz[tens[f]].cscale, coef[f], cs + f * ncp, nc, o,
                       ri->status.p, s);
    }
    oz::Prod p;
    p.a = Y; p.b = cc;
    p.sa = scale + P0 * nt; p.sb = cs + 4 * ncp;
    p.M = cnt * nt; p.N = nc; p.K = 2 * nu;
    p.kchunk = round_up(2 * nu, oz::kBK);
    p.negate_odd = 1;
    p.out = m->B.p + 2 * P0 * nt * nt;
    p.ldo = 2 * nt;
    oz::run_products(&p, 1, ri->status.p, s);
  }
  return true;
}

}  // namespace rr

rr_ri_store::rr_ri_store() {
  auto& l = rr::stores();
  std::lock_guard<std::mutex> lock(l.mu);
  l.all.push_back(this);
}

rr_ri_store::~rr_ri_store() {
  auto& l = rr::stores();
  std::lock_guard<std::mutex> lock(l.mu);
  l.all.erase(std::find(l.all.begin(), l.all.end(), this));
}
