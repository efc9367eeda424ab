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
// in the box. Outside the box the image comes first, in FP64, and the cell is the
// image's: an FP32 cell of the coordinate itself is off by 1e-7 of its distance,
// which some tens of boxes out passes what the row search allows for when it
// cuts the cells to the reach of its rows. The cell count never leaves floating
// point before it is known to fit: a coordinate of 2^31 cell widths and more has no
// int, and the build indexes memory with what comes out.
SG_CELL_FN int cell_axis(float& x, int nc, float L, float iL, double Ld) {
    float f = floorf((x + 0.5f * L) * (nc * iL));
    if (f >= 0.f && f < (float)nc) return (int)f;
    x = (float)((double)x - floor((double)x / Ld + 0.5) * Ld);
    f = floorf((x + 0.5f * L) * (nc * iL));
    return f > 0.f ? (f < (float)nc ? (int)f : nc - 1) : 0;   // an image on a face; not finite, or past FP64
}
