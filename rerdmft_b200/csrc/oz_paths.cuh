// The FP64 paths that run on digit planes (oz_exchange.cu).  Each returns false, with nothing launched, when the
// sizes or the tensor are not for it; the caller then takes the DMMA path.
#pragma once

#include "ri_store.cuh"

namespace rr {

// Smallest AO dimension the digit paths are prepared for.
constexpr int64_t kOzMinDim = 8;

// Whether the nonrelativistic products (a half-transform of `cols` coefficient rows over naux x n x n and what
// follows it) are worth the digit path, which adds three small launches.  Fock build, DMMA path against digit
// path, us: n = 96 (3.2e7) 226 / 241, n = 128 (1.0e8) 263 / 271, n = 128 (2.7e8) 354 / 356, n = 160 (2.6e8)
// 321 / 302, n = 200 (1.6e9) 690 / 492; MO build: n = 64 (6.7e7) 58 / 64, n = 96 (3.4e8) 113 / 108, n = 128
// (1.1e9) 250 / 175.  The relativistic builds take it from kOzMinDim on: one launch for all blocks instead of
// up to 27 products and their reductions (X2C nl = 32: 435 / 249, four components nl = 32: 1069 / 445).
inline bool oz_worth(int64_t naux, int64_t n, int64_t cols) {
  return n >= kOzMinDim && static_cast<double>(naux) * static_cast<double>(n) * static_cast<double>(n) * static_cast<double>(cols) >= 2e8;
}

// The digit data of a store for the time in which a call queues products on it: made on the first use (statistics and planes of
// every tensor; synchronises s), and held against release_idle_planes.  ok: the store's tensors are for the digit path.  Not
// made while s is captured (the call then takes the DMMA path).
class OzUse {
 public:
  OzUse(rr_ri_store* h, cudaStream_t s);
  ~OzUse();
  OzUse(const OzUse&) = delete;
  OzUse& operator=(const OzUse&) = delete;
  bool ok = false;

 private:
  rr_ri_store* h_;
};

// K = sum_P (Ct B^P)^T (Ct B^P); Ct as for exchange_nonrel.  The caller holds an OzUse that is ok.
bool oz_exchange_nonrel(rr_ri_store* h, const double* Ct, int64_t ldct, bool ct_transposed, int64_t nocc, double* K,
                        cudaStream_t s);

// The exchange blocks of the relativistic builds into G (complex ntot x ntot): sgn K, plus J[tens[f]] on the diagonal
// blocks once j_ready has fired (J null: no Coulomb part).
bool oz_exchange_rel(rr_ri_store* h, int nf, const int64_t* off, const int64_t* fs, const int* tens, int64_t ntot,
                     const double* Ct, int64_t r, double* const* J, cudaEvent_t j_ready, double* G, double sgn,
                     cudaStream_t s);

}  // namespace rr

struct rr_mo_store;

namespace rr {
// The FP64 MO transforms of mo.cu: C^T B^P C from the store's tensor, and the four-component transform.
bool oz_mo_build_nonrel(rr_ri_store* ri, const double* Cd, rr_mo_store* m, cudaStream_t s);
bool oz_mo_build_ukb(rr_ri_store* ri, const double* cd, int64_t nt, rr_mo_store* m, cudaStream_t s);
}  // namespace rr
