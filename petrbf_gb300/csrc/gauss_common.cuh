// gauss_common.cuh -- what the Gaussian sum kernels of gauss.cu and gauss_fx.cu share.
#pragma once
#include "device.h"

namespace prbf {

constexpr int kTileT = 128;  // targets per work item

constexpr size_t align16(size_t v) { return (v + 15) & ~(size_t)15; }

// Per source a 64-bit word: per axis, bit k (k = 0 .. 2 nb) = the reference's FP64 box test
// |x_j - xc| < trunc_len against the centre of the target cell at offset k - nb from the
// source's cell; its cell's y index in the top 16 bits.
constexpr int kMaskBits = 15;  // 2 nb + 1 <= 15 bits per axis: nb_trunc <= 7
constexpr int kMaskY = kMaskBits, kMaskZ = 2 * kMaskBits, kMaskCellY = 48;

constexpr int kFxSymTile = 64;  // targets per pass of the fixed-point symmetric form

// ---- gauss_fx.cu: the FP64 sums with fixed-point exponents --------------------------------
// Whether the plan's data fit it is plan.fx_ready (set with the point data).
void gauss_fx_sum(const GaussPlan& P, const PointsView& t, const PointsView& s, const double* gv, double* w,
                  unsigned* err, const int* skip, int nv, long long vstride, VecSkip left, cudaStream_t st);
// The symmetric form's sum (2D, one vector; the partial slots are left for k_sym_gather).
void gauss_fx_sym(const GaussPlan& P, const PointsView& s, const double* gv, double* w, unsigned* err,
                  const int* skip, cudaStream_t st);
void gauss_fx_upload_tables(cudaStream_t s);

}  // namespace prbf
