// Item walk shared by the pointwise, reduction, prolongation and table-stencil kernels.
//
// These kernels move 16 to 32 bytes per cell and compute a few operations, so memory bounds them and
// what matters is enough loads in flight, few index instructions and no idle lanes, for every shape:
// solid boxes, faces, lines. An item is the cells (x, y, z .. z + Z - 1): Z planes of a point, whose loads
// a thread issues before its first store. Items are numbered x fastest, then y, then the groups of Z
// planes, and a thread takes one: a warp covers 32 consecutive items whatever the extents, and the two
// divisions by the extents are multiplications by reciprocals that the host prepared (once for Z cells;
// 64-bit divisions for each cell took longer than the memory). Accesses stay one element wide: a warp's
// request is 128 or 256 contiguous bytes whatever the alignment of odd or ghosted rows.
#pragma once
#include <utility>

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

// Division of any 32-bit number by d >= 1 as a multiplication, an add and two shifts (T. Granlund and P. L.
// Montgomery, "Division by Invariant Integers using Multiplication", 1994, figure 4.1).
struct FastDiv {
    unsigned d, m;
    unsigned char s1, s2;
};
inline FastDiv fast_div(unsigned d)
{
    const unsigned l = d > 1 ? 32 - __builtin_clz(d - 1) : 0;       // 2^l >= d
    return FastDiv{d, (unsigned)(((1ull << 32) * ((1ull << l) - d)) / d + 1), (unsigned char)(l > 0), (unsigned char)(l > 0 ? l - 1 : 0)};
}
__host__ __device__ __forceinline__ unsigned quotient(unsigned n, const FastDiv& f)
{
#ifdef __CUDA_ARCH__
    const unsigned t = __umulhi(n, f.m);
#else
    const unsigned t = (unsigned)(((unsigned long long)n * f.m) >> 32);
#endif
    return (t + ((n - t) >> f.s1)) >> f.s2;
}

int cached_sm_count();

constexpr int kWalkZ = 4;
constexpr int kWalkThreads = 256;

struct Walk {
    int nx, ny, nz;
    int planes;          // of an item
    FastDiv dx, dy;
    long long items;     // above 32 bits the divisions are 64 bits wide
};
inline Walk walk_of(const Region& r, int planes = kWalkZ)
{
    Walk w{r.n[0], r.n[1], r.n[2], planes, {1, 1, 0, 0}, {1, 1, 0, 0}, 0};
    if (w.nx < 1 || w.ny < 1 || w.nz < 1) return w;
    w.dx = fast_div(w.nx);
    w.dy = fast_div(w.ny);
    w.items = (long long)w.nx * w.ny * ((w.nz + (long long)planes - 1) / planes);
    return w;
}
inline Walk walk_cube(int n)
{
    return walk_of(Region{{0, 0, 0}, {n, n, n}});
}
// grid: x over items, z over components
inline dim3 walk_grid(const Walk& w, int ncomp)
{
    return dim3((unsigned)((w.items + kWalkThreads - 1) / kWalkThreads), 1, ncomp < 65535 ? ncomp : 65535);
}

// The same for kernels that take any number of planes up to kWalkZ: single cells while these fit two blocks
// per SM
inline Walk walk_spread(const Region& r)
{
    const bool small = (long long)r.n[0] * r.n[1] * r.n[2] <= 2LL * kWalkThreads * cached_sm_count();
    return walk_of(r, small ? 1 : kWalkZ);
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

// Boxes thin in z walk their y extent in its place, so that the loads in flight have planes to go to.
template <typename... V>
inline bool turn_thin(Region& r, V&... views)
{
    if (r.n[2] >= kWalkZ || r.n[1] <= r.n[2]) return false;
    std::swap(r.n[1], r.n[2]);
    (std::swap(views.sy, views.sz), ...);
    return true;
}

// item i < w.items: its point and its group of planes
__host__ __device__ __forceinline__ void walk_item(const Walk& w, long long i, int& x, int& y, int& group)
{
    if (w.items <= 0xffffffffLL) {
        const unsigned j = (unsigned)i, q = quotient(j, w.dx), g = quotient(q, w.dy);
        x = (int)(j - q * w.dx.d);
        y = (int)(q - g * w.dy.d);
        group = (int)g;
    } else {
        const long long q = i / w.nx;
        x = (int)(i - q * w.nx);
        group = (int)(q / w.ny);
        y = (int)(q - (long long)group * w.ny);
    }
}

// body(x, y, z, planes): the cells (x, y, z .. z+planes-1), 1 <= planes <= w.planes
template <class F>
__device__ __forceinline__ void walk_items(const Walk& w, F&& body)
{
    const long long i = (long long)blockIdx.x * kWalkThreads + threadIdx.x;
    if (i >= w.items) return;
    int x, y, g;
    walk_item(w, i, x, y, g);
    body(x, y, g * w.planes, min(w.planes, w.nz - g * w.planes));
}

} // namespace pb
