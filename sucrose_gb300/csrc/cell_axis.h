// Cell of a coordinate along one axis of a periodic box, for the list build and
// for host code.
#pragma once
#include <cmath>

#ifdef __CUDACC__
#define SG_CELL_FN __host__ __device__ __forceinline__
#else
#define SG_CELL_FN inline
#endif

// The cell in [0, nc) of any x, the non-finite ones among them, and x's image
// in the box, consistent with each other: whole boxes are taken off both (in
// FP64 when there are any, so that the image is the position to half an ulp of
// the box). The cell count never leaves floating point before it is known to
// fit: a coordinate of 2^31 cell widths and more has no int, and the build
// indexes memory with what comes out.
SG_CELL_FN int cell_axis(float& x, int nc, float L, float iL, double Ld) {
    const float f = floorf((x + 0.5f * L) * (nc * iL));
    if (f >= 0.f && f < (float)nc) return (int)f;
    const double k = floor((double)f / nc), m = (double)f - k * nc;
    x = (float)((double)x - k * Ld);
    return m > 0.0 ? (m < nc ? (int)m : nc - 1) : 0;   // past 2^53 cells, m is rounded; a NaN: cell 0
}
