// pf_spectral.cuh -- direct solve of the periodic 7-point pressure equation by
// fast transforms (pf_spectral.cu), used by the mixed forms and by solves
// that ask for it.
#pragma once
#include "pf_sweep.cuh"

namespace pf {

// Longest extent.  A stage's butterflies run in one go, at most 8 values a
// thread, so radix 3, 5 and 7 stages (6, 5 and 7 values) need more threads a line
// than n / 8, and a block (512 threads, at least two line pairs) takes extents
// with a factor 5 up to 1280, else with a factor 3 up to 1536, else with a factor
// 7 up to 1792, all others to 2048 (spectral_applies).
constexpr int kSpectralMaxN = 2048;
constexpr int kSpectralMaxStages = 12;

// The tightest relative residual the direct solve is asked for: its own
// residual is the rounding of an FP64 transform seen through the operator
// (measured max|b - A x| / max|b| of step right-hand sides: 32^3 1e-15,
// 128^3 2.3e-14, 512^3 1.4e-13).  Tighter tolerances go to the iterative solve.
constexpr double kSpectralMinTol = 1e-12;

// One axis' transform: n = product of the radices, run in this order.
struct SpectralAxis {
    int n;
    int stages;
    int radix[kSpectralMaxStages];
    unsigned magic[kSpectralMaxStages];  // ceil(2^32 / product of the earlier radices)
    int odd;                             // n has an odd factor
    int tp;                              // threads per line
    int lines;                           // line pairs per block (8, 4 or 2)
    const double2* tw;                   // exp(-2 pi i k / n), k < n
    const double* lam;                   // eigenvalues of this axis' part of A
};

struct SpectralPlan {
    bool on = false;
    Dims d;
    SpectralAxis ax[3];
    double2* tables = nullptr;
    double vol_d2[3];  // vol / h^2
};

// True when the direct solve takes this grid, tolerance and pointer.
bool spectral_applies(const pf_grid* g, double min_res, const double* DP, const void* tables);
size_t spectral_table_bytes(const pf_grid* g);
// Sets the plan up (no device work); tables: spectral_table_bytes, 16-byte aligned.
cudaError_t spectral_setup(const pf_grid* g, void* tables, SpectralPlan* P);
// Fills the tables (once per plan, or before a solve).
cudaError_t spectral_enqueue_tables(const SpectralPlan& P, cudaStream_t s);
// DP = the zero-mean solution of A DP = c src (c = -vol rho / dt); *nonfin
// becomes 1 where src holds a NaN or Inf (and is left alone otherwise).
cudaError_t spectral_enqueue_solve(const SpectralPlan& P, const double* src, double c, double* DP,
                                   int* nonfin, cudaStream_t s);

}  // namespace pf
