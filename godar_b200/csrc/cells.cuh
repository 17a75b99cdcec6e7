// The cell grid of a batch's fields: the cell of a position, and the walk over
// the cells around a floe, shared by the neighbour search (build.cu) and bond
// creation (bonds_init.cu).
//
// A cell list is a CSR over cells: coff[c] .. coff[c + 1] are the positions of
// cell c's floes.  Cells are numbered row by row within an instance, so the
// floes of neighbouring cells of one row sit at consecutive positions and a
// stencil row is one range (two where it wraps).
#pragma once
#include "common.cuh"

namespace godar {

GD_DEV void cell_of(const InstParams &P, double x, double y, int &cx, int &cy)
{
    // clamp before the integer conversion so that non-finite or far-away
    // positions land in an edge cell
    double fx = x / P.cw, fy = y / P.ch;
    if (!(fx >= 0.0)) fx = 0.0;
    if (!(fy >= 0.0)) fy = 0.0;
    if (fx > (double)P.ncx) fx = (double)P.ncx;
    if (fy > (double)P.ncy) fy = (double)P.ncy;
    cx = (int)floor(fx);
    cy = (int)floor(fy);
    cx = cx < 0 ? 0 : (cx >= P.ncx ? P.ncx - 1 : cx);
    cy = cy < 0 ? 0 : (cy >= P.ncy ? P.ncy - 1 : cy);
}

GD_DEV uint32_t cell_key(const InstParams &P, double x, double y)
{
    int cx, cy;
    cell_of(P, x, y, cx, cy);
    return (uint32_t)(P.coff + (long long)cy * P.ncx + cx);
}

// Calls f(q) for every position q of the cells within the stencil (kx, ky)
// around (x, y) that falls to lane `sub` of a group of GRP lanes: a group
// reads a range side by side.
template <class F>
GD_DEV void walk_cells(const InstParams &P, double x, double y, const int *coff, int sub, F f)
{
    const bool px = P.boundary & BC_PERIODIC_X, py = P.boundary & BC_PERIODIC_Y;
    int cx, cy;
    cell_of(P, x, y, cx, cy);
    int x0 = cx - P.kx, x1 = cx + P.kx, y0 = cy - P.ky, y1 = cy + P.ky;
    if (px && x1 - x0 + 1 >= P.ncx) { x0 = 0; x1 = P.ncx - 1; }
    if (py && y1 - y0 + 1 >= P.ncy) { y0 = 0; y1 = P.ncy - 1; }
    // the row's cells [a0, a1], and [0, b1] where it wraps
    int a0, a1, b1 = -1;
    if (!px) {
        a0 = x0 < 0 ? 0 : x0;
        a1 = x1 >= P.ncx ? P.ncx - 1 : x1;
    } else {
        a0 = (x0 % P.ncx + P.ncx) % P.ncx;
        a1 = a0 + (x1 - x0);
        if (a1 >= P.ncx) {
            b1 = a1 - P.ncx;
            a1 = P.ncx - 1;
        }
    }
    for (int yy = y0; yy <= y1; yy++) {
        int wy = yy;
        if (py) wy = (yy % P.ncy + P.ncy) % P.ncy;
        else if (yy < 0 || yy >= P.ncy) continue;
        const long long row = P.coff + (long long)wy * P.ncx;
        for (int q = coff[row + a0] + sub, e = coff[row + a1 + 1]; q < e; q += GRP) f(q);
        if (b1 >= 0)
            for (int q = coff[row] + sub, e = coff[row + b1 + 1]; q < e; q += GRP) f(q);
    }
}

// What a group of GRP lanes of a block collects of one floe: at most CAP
// entries in shared memory, in any order.
template <int CAP>
struct GroupBag {
    double d[CAP];
    int t[CAP], id[CAP];
    int n[2];            // entries found (which may exceed CAP): of lower id, of higher id
};

}  // namespace godar
