// Row walk shared by the pointwise, reduction, prolongation and table-stencil kernels.
//
// These kernels move 16 to 32 bytes per cell and compute a few operations, so memory bounds them and
// what matters is enough loads in flight with few index instructions. A block is 256 threads: 2^lx
// lanes along x and 256 >> lx rows of y; each thread walks its row with kWalkZ planes at once, issuing
// the planes' loads before the first store. A cell costs one pointer add per field (a flattened walk
// of one cell at a time spends two 64-bit divisions and has one load in flight per cell). Accesses
// stay one element wide: a warp's request is 128 or 256 contiguous bytes whatever the alignment of odd
// or ghosted rows. Measured (B200, 160^3, fields in L2): out = a x + b y, out += k, out *= s, square sum
// and max norm, five calls, 154 -> 92 us.
#pragma once
#include "pb_internal.cuh"

namespace pb {

struct Region {
    int lo[3];
    int n[3];
};
inline Region region_of(const Box3& b)
{
    Region r;
    for (int d = 0; d < 3; d++) { r.lo[d] = b.lo[d]; r.n[d] = (int)bsize(b, d); }
    return r;
}

constexpr int kWalkZ = 4;
constexpr int kWalkThreads = 256;

struct Walk {
    int nx, ny, nz;
    int lx;            // log2 of the lanes along x
};
inline Walk walk_of(const Region& r)
{
    Walk w{r.n[0], r.n[1], r.n[2], 5};
    while (w.lx > 3 && (1 << (w.lx - 1)) >= r.n[0]) w.lx--;   // short rows: more rows per block, fewer idle lanes
    return w;
}
// grid: x over groups of rows, y over groups of kWalkZ planes, z over components
inline dim3 walk_grid(const Walk& w, int ncomp)
{
    const int rows = kWalkThreads >> w.lx;
    const int gx = (w.ny + rows - 1) / rows, gy = (w.nz + kWalkZ - 1) / kWalkZ;
    return dim3(gx, gy < 65535 ? gy : 65535, ncomp < 65535 ? ncomp : 65535);
}

// A field seen from the region's first cell: base address, row and plane pitch.
template <typename T>
struct FieldView {
    T* p;
    long long sy, sz;
};
template <typename T>
inline FieldView<T> view_of(T* base, const Box3& b, const Region& r, const int* shift = nullptr)
{
    FieldView<T> v;
    v.sy = bsize(b, 0);
    v.sz = bsize(b, 0) * bsize(b, 1);
    v.p = base;
    const long long step[3] = {1, v.sy, v.sz};
    for (int d = 0; d < 3; d++) v.p += step[d] * (r.lo[d] + (shift ? shift[d] : 0) - b.lo[d]);
    return v;
}

// body(x, y, z, planes): the cells (x, y, z .. z+planes-1), 1 <= planes <= kWalkZ
template <class F>
__device__ __forceinline__ void walk_rows(const Walk& w, F&& body)
{
    const int lane = threadIdx.x & ((1 << w.lx) - 1), row = threadIdx.x >> w.lx;
    const int y = blockIdx.x * (kWalkThreads >> w.lx) + row;
    if (y >= w.ny) return;
    for (int z = blockIdx.y * kWalkZ; z < w.nz; z += gridDim.y * kWalkZ) {
        const int planes = min(kWalkZ, w.nz - z);
        for (int x = lane; x < w.nx; x += 1 << w.lx) body(x, y, z, planes);
    }
}

} // namespace pb
