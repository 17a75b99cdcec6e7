// The cells a placed disk's bounding box meets on one axis, and how many they
// can be: the placement sizes its cover lists by the bound before the first
// kernel (host and device, place.cu).
#pragma once
#include <cmath>
#include <cuda_runtime.h>

namespace godar {

// Cell index range [a, b] of the interval [lo, hi] on one axis; a periodic
// range longer than the axis becomes the whole axis.
__host__ __device__ inline void cell_span(double lo, double hi, double cw, int nc, int per, int &a, int &b)
{
    a = (int)floor(lo / cw);
    b = (int)floor(hi / cw);
    if (per) {
        if (b - a + 1 >= nc) { a = 0; b = nc - 1; }
    } else {
        a = a < 0 ? 0 : a;
        b = b > nc - 1 ? nc - 1 : b;
    }
}

// The most cells of width cw, nc of them, that a disk of radius r meets
// wherever it lies.  lo and hi and their quotients round: a box a rounding
// error short of a whole number of cells can meet one cell more than its width
// says, so the quotient is taken larger by far more than that error (8,192
// cells: 5e-12) before it is cut.
inline double cells_met(double r, double cw, int nc)
{
    return std::fmin((double)nc, std::floor(2.0 * r / cw + 1e-9) + 2.0);
}

}  // namespace godar
