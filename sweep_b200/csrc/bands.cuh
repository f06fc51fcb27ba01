// bands.cuh -- the boundary bands of the staggered equations: per face a band
// M + 1 wide from M cells outside the physical box over the box's other axes
// (reference boundary/strip.cuh:136-175), each cell once.
//
// Listed as, per axis (z, y, x) and face: the M layers outside the box over
// the box's other axes, then the box's outermost layer without the cells of
// the axes before.  The list is made on the device (`band_table`): marking the
// bands in a grid on the host took 5-20 ms of every call on a 168^3 grid.
#pragma once

#include "common.cuh"

namespace sweep {
namespace bands {

struct Bands {
    int M, z0, z1, y0, y1, x0, x1;  // physical box (2-D: y 0 .. 1)
    int out[3], in[3];              // cells of one face per axis (z, y, x): outside the box, of its outermost layer
    int count;
};

template <int ND>
inline Bands make(int M, int z0, int z1, int y0, int y1, int x0, int x1)
{
    Bands t{};
    t.M = M; t.z0 = z0; t.z1 = z1; t.x0 = x0; t.x1 = x1;
    t.y0 = ND == 3 ? y0 : 0;
    t.y1 = ND == 3 ? y1 : 1;
    const int bz = z1 - z0, by = t.y1 - t.y0, bx = x1 - x0;
    t.out[0] = M * by * bx; t.in[0] = by * bx;
    if (ND == 3) { t.out[1] = M * bz * bx; t.in[1] = (bz - 2) * bx; }
    t.out[2] = M * bz * by; t.in[2] = (bz - 2) * (ND == 3 ? by - 2 : 1);
    for (int a = 0; a < 3; ++a) t.count += 2 * (t.out[a] + t.in[a]);
    return t;
}

// cell e of the list: z, y, x
template <int ND>
__host__ __device__ inline void cell(const Bands& t, int e, int& z, int& y, int& x)
{
    int axis = 0;
    while (axis < 2 && e >= 2 * (t.out[axis] + t.in[axis])) {
        e -= 2 * (t.out[axis] + t.in[axis]);
        ++axis;
    }
    const int face = t.out[axis] + t.in[axis];
    const bool hi = e >= face;
    if (hi) e -= face;
    // layer: 0 the box's outermost, 1 .. M outside it; inner: the cells of that
    // layer leave out the outermost ones of the axes before
    const bool inner = e >= t.out[axis];
    if (inner) e -= t.out[axis];
    const int layer_cells = inner ? t.in[axis] : t.out[axis] / t.M;
    const int layer = inner ? 0 : 1 + e / layer_cells;
    e %= layer_cells;
    const int cut = inner ? 1 : 0, bx = t.x1 - t.x0;
    if (axis == 0) {
        x = t.x0 + e % bx;
        y = t.y0 + e / bx;
        z = hi ? t.z1 - 1 + layer : t.z0 - layer;
    } else if (axis == 1) {
        x = t.x0 + e % bx;
        z = t.z0 + cut + e / bx;
        y = hi ? t.y1 - 1 + layer : t.y0 - layer;
    } else {
        const int rows = ND == 3 ? t.y1 - t.y0 - 2 * cut : 1;
        y = t.y0 + (ND == 3 ? cut : 0) + e % rows;
        z = t.z0 + cut + e / rows;
        x = hi ? t.x1 - 1 + layer : t.x0 - layer;
    }
}

// offsets of the cells in a shot's field of y stride SY and z stride SZ
template <int ND>
__global__ void band_table(const Bands t, int SY, int SZ, int* cells)
{
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < t.count; e += gridDim.x * blockDim.x) {
        int z, y, x;
        cell<ND>(t, e, z, y, x);
        cells[e] = z * SZ + y * SY + x;
    }
}

}  // namespace bands
}  // namespace sweep
