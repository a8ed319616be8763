// Row walk shared by the pointwise, reduction, prolongation and table-stencil kernels.
//
// These kernels move 16 to 32 bytes per cell and compute a few operations, so memory bounds them and
// what matters is enough loads in flight with few index instructions. A block is 256 threads: 2^lx
// lanes along x and 256 >> lx rows of y; each thread walks its row with kWalkZ planes at once, issuing
// the planes' loads before the first store. A cell costs one pointer add per field (a flattened walk
// of one cell at a time spends two 64-bit divisions and has one load in flight per cell). Accesses
// stay one element wide: a warp's request is 128 or 256 contiguous bytes whatever the alignment of odd
// or ghosted rows. Measured (B200, 160^3, fields in L2): out = a x + b y, out += k, out *= s, square sum
// and max norm, five calls, 154 -> 87 us; each kernel alone moves its bytes at 6.2 to 6.5 TB/s.
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

int cached_sm_count();

struct Walk {
    int nx, ny, nz;
    int lx;            // log2 of the lanes along x
    int sx;            // blocks that share a row's lane groups
};
inline Walk walk_of(const Region& r)
{
    Walk w{r.n[0], r.n[1], r.n[2], 5, 1};
    while (w.lx > 3 && (1 << (w.lx - 1)) >= r.n[0]) w.lx--;   // short rows: more rows per block, fewer idle lanes
    // a row's lane groups go to several blocks while there are fewer than eight blocks per SM: a small box
    // then has all its loads in flight at once instead of one lane group after another
    const int rows = kWalkThreads >> w.lx, groups = (w.nx + (1 << w.lx) - 1) >> w.lx;
    const long long blocks = ((w.ny + (long long)rows - 1) / rows) * ((w.nz + (long long)kWalkZ - 1) / kWalkZ);
    while (w.sx < groups && blocks * w.sx < 8LL * cached_sm_count()) w.sx++;
    return w;
}
inline Walk walk_cube(int n)
{
    return walk_of(Region{{0, 0, 0}, {n, n, n}});
}
// grid: x over groups of rows and shares of a row, y over groups of kWalkZ planes, z over components
inline dim3 walk_grid(const Walk& w, int ncomp)
{
    const int rows = kWalkThreads >> w.lx;
    const int gx = (w.ny + rows - 1) / rows * w.sx, gy = (w.nz + kWalkZ - 1) / kWalkZ;
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
    const int group = blockIdx.x / w.sx, share = blockIdx.x - group * w.sx;
    const int y = group * (kWalkThreads >> w.lx) + row;
    if (y >= w.ny) return;
    for (int z = blockIdx.y * kWalkZ; z < w.nz; z += gridDim.y * kWalkZ) {
        const int planes = min(kWalkZ, w.nz - z);
        for (int x = lane + (share << w.lx); x < w.nx; x += w.sx << w.lx) body(x, y, z, planes);
    }
}

} // namespace pb
