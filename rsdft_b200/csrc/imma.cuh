// FP64 contractions on the INT8 tensor cores (imma.cu).
#pragma once

#include "common.cuh"

namespace rsdft {

// The INT8 slices of a tall FP64 block (imma_slice).
struct ImmaSlices {
    const int8_t* rows = nullptr;  // [slice][K block of 64 grid points][band][64]
    const int8_t* cols = nullptr;  // [slice][K block of 64 bands][grid point][64]
    const int* exps = nullptr;     // per band: |x| < 2^exps
    const int* tail = nullptr;     // per band: set when it decays (imma.cu)
    int* need = nullptr;           // per 128 columns of a rotation, and for all: set when the DMMA form has to make them
    int nb = 0;
    long ml = 0;
};

// Whether Gram products and rotations of nb bands on ml points go to the
// INT8 form (the caller takes dmma.cu otherwise).
bool imma_suits(long ml, int nb);

// Slice A (ml x nb, leading dimension ld) into the workspaces named after ws:
// rows for Gram products, cols for rotations.  *bad (device, cleared by the
// caller) is set when a value is not finite or out of the sliced range, or when a
// band decays so far that its tail would lose digits: the products below then
// leave their results to a DMMA launch conditional on it.
// RSDFT_ENOMEM when the slices do not fit.  All buffers are optional ones
// (workspace_optional): the caller holds them while it uses the slices.
int imma_slice(const double* A, long ld, long ml, int nb, const char* ws, bool need_rows, bool need_cols, int* bad,
               ImmaSlices* out);

// C (nb x nb, ldc) = alpha A^T B, symmetric: only the tiles on and above the
// diagonal are formed, symmetrize averages the 128 x 128 diagonal blocks.
// RSDFT_ENOMEM, and nothing launched, when the partial sums do not fit.
int imma_gram(const ImmaSlices& a, const ImmaSlices& b, double alpha, int symmetrize, const int* bad, double* C,
              long ldc);

// The INT8 slices of a rotation matrix V (nb x nb, leading dimension ldv) and
// its columns' scales.  Sets a.need for the columns that the DMMA form has to make
// (they come out right to 2^-60 of their largest only).  RSDFT_ENOMEM, and nothing
// launched, when they do not fit.
struct ImmaV {
    const int8_t* slices = nullptr;
    const double* scale = nullptr;
};
int imma_slice_v(const ImmaSlices& a, const double* V, int ldv, int* bad, ImmaV* out);

// out (ml x nb, leading dimension ld) = A V.  Reads only A's slices, so out may be
// A itself.
int imma_rotate(const ImmaSlices& a, const ImmaV& v, const int* bad, double* out, long ld);

}  // namespace rsdft
