// One-launch forms of the density step's purification (sp2.cu).
#pragma once

#include <functional>

#include "rr_common.cuh"

namespace rr {

// Largest n the one-launch purification takes.  An iteration of an SCF loop (naux = n / 2), product + step launches / one launch, ms: real n =
// 240 0.96 / 0.63, 400 1.64 / 1.13, 512 2.01 / 1.53, 640 3.30 / 2.84, 800 5.34 / 5.32; complex n = 232 1.10 / 0.83, 320 1.37 / 1.01,
// 400 1.58 / 1.43, 512 2.13 / 1.89, 640 4.41 / 4.62.  The two meet near n = 800 and complex 580, where a step's products fill the GPU by
// themselves; the limits keep clear of that.
constexpr int64_t kSp2MaxReal = 512, kSp2MaxComplex = 400;

// CTAs of the SCF loops' two-stage reductions.
constexpr int kScfRedCtas = 256;

// Doubles of scratch sp2_run needs besides X's second buffer.
int64_t sp2_scratch_doubles();

// SP2 purification of the Hermitian F (n x n): X <- the projector onto its lowest `nocc` eigenvectors, from the spectral
// interval b = [lo, hi] (device; sure: it holds the spectrum for certain); Y: a second n x n buffer; scratch: sp2_scratch_doubles().  outcome (device, 4 doubles): [0]
// = 0 converged, 1 the interval missed part of the spectrum (or max_steps passed), 2 a grid barrier expired; [1], [2] = tr X and
// tr X^2 of the last step; [3] = steps.
void sp2_run(const double* F, int64_t n, double nocc, bool cplx, const double* b, bool sure, int max_steps, double* X,
             double* Y, double* scratch, double* outcome, cudaStream_t s);

// Doubles sp2_projector (scf.cu) reserves for an n x n problem: its reductions and split-K sums, or the one launch's scratch and
// outcome, whose size does not depend on n and is the larger of the two up to n = 8 (complex 6).
int64_t sp2_workspace_doubles(int64_t n, bool cplx);

// The same for complex problems side by side, each on its own group of CTAs with its own barrier (b holds the spectrum,
// at most 120 steps).  put copies a table to the device for launches on s.
struct Sp2Problem {
  const double *F, *b;
  double *X, *Y, *scratch, *outcome;
  double nocc;
  int64_t n;
};
void sp2_run_group(const Sp2Problem* p, int count, const std::function<const void*(const void*, size_t)>& put, cudaStream_t s);

// b = [lo, hi] narrowed to the extreme eigenvalues of T y = theta M y (k x k, k = 32, full Hermitian, M positive
// definite), widened by 10 % of their distance on both sides; unchanged when M is not positive definite.
constexpr int kRitz = 32;
void ritz_interval(const double* T, const double* M, bool cplx, double* b, cudaStream_t s);

}  // namespace rr
