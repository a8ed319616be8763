// Stencil objects and Stencil::apply on the device (C ABI: pb_stencil_*).
//
// Replaces the reference's DEVICE branch of Stencil::protoApply
// (include/base/implem/Proto_StencilImplem.H:844-895 in the reference project), whose kernel runs
// one thread per point with coefficients read from global memory. Here:
//   * the seven- and thirteen-point Laplacians (in the exact insertion order the reference's
//     StencilLib produces) run on the TMA-staged z-streaming kernel of pb_star.cuh, or on its
//     one-thread-per-point variant for small or unaligned boxes;
//   * every other stencil (any ratios, destination shift, up to kMaxTerms terms) runs on a
//     table kernel with the coefficients and linearised offsets in kernel parameters.
// All FP64 results equal Stencil::hostApply bit for bit (term order, scale folded into the
// coefficients when scale != 1, no FMA).
#include <cstdio>
#include <cstring>
#include <mutex>
#include <vector>

#include "pb_internal.cuh"
#include "pb_star.cuh"
#include "pb_stencil_impl.cuh"
#include "pb_walk.cuh"

namespace pb {

PB_DEFINE_ERROR_READER(read_error_stencil)

// The bounded wait of the pipelined kernels, made to expire on purpose: one thread waits on an
// mbarrier whose phase never completes (nothing arrives and no copy is in flight), gives up after
// `tries` polls through the same mbar_wait_limited every kernel uses, and records whether the wait
// reported the timeout; the wait also sets the device error flag that pb_device_check reads.
static __device__ int g_wait_expired = 0;
static __global__ void k_wait_expiry(uint32_t tries)
{
    __shared__ uint64_t bar;
    if (threadIdx.x == 0) {
        mbar_init(&bar, 1);
        fence_barrier_init();
    }
    __syncthreads();
    if (threadIdx.x == 0) g_wait_expired = mbar_wait_limited(&bar, 0, tries) ? 0 : 1;
}

static thread_local int t_last_cuda = 0;
void set_cuda_error(cudaError_t e) { t_last_cuda = (int)e; }

// ---- TMA tensor-map encoding through the driver entry point (no -lcuda link needed) ----------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static EncodeTiledFn g_encode = nullptr;
static std::once_flag g_encode_once;

static void load_encode()
{
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
        g_encode = reinterpret_cast<EncodeTiledFn>(fn);
    cudaGetLastError();
}

bool tma_available()
{
    std::call_once(g_encode_once, load_encode);
    return g_encode != nullptr;
}

int encode_tmap_3d(CUtensorMap* map, const void* base, int esize, long long Sx, long long Sy, long long Sz, int boxX,
                   int boxY, int boxZ)
{
    if (!tma_available()) return PB_ERR_UNSUPPORTED;
    if ((reinterpret_cast<uintptr_t>(base) & 15) != 0) return PB_ERR_ALIGN;
    if ((Sx * esize) % 16 != 0) return PB_ERR_ALIGN;
    if (boxX > 256 || boxY > 256 || boxZ > 256 || (boxX * esize) % 16 != 0) return PB_ERR_ALIGN;
    cuuint64_t gdim[3] = {(cuuint64_t)Sx, (cuuint64_t)Sy, (cuuint64_t)Sz};
    cuuint64_t gstr[2] = {(cuuint64_t)(Sx * esize), (cuuint64_t)(Sx * Sy * esize)};
    cuuint32_t box[3] = {(cuuint32_t)boxX, (cuuint32_t)boxY, (cuuint32_t)boxZ};
    cuuint32_t estr[3] = {1, 1, 1};
    CUtensorMapDataType dt = esize == 8 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT64 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32;
    CUresult r = g_encode(map, dt, 3, const_cast<void*>(base), gdim, gstr, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                          CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? PB_OK : PB_ERR_ALIGN;
}

// ---- generic table kernel ---------------------------------------------------------------------
// Any table: acc = sum_j c_j * src[first + off_j], first the term of the span's low corner, so every
// offset is non-negative and, with at most 2^32 source cells, 32 bits wide: a term is then one load
// from a uniform base plus the thread's 32-bit index, one multiply and one add; eight terms' loads are in
// flight. A thread takes one cell: with four planes a thread a small box has a quarter of the warps to
// hide its chain of loads, and a block's source lines outgrow L1 between the two halves of a ratio-2 row.
// Bound by the issue of the terms' loads. Measured (B200, us, one cell a thread / four): 27 points on 33^3
// 3.2 / 7.4, AvgDown to 64^3 3.4 / 4.8, to 160^3 43 / 69, 64 terms on 160^3 56 / 61.
constexpr int kTableTerms = 8;    // unroll of the term loop
template <typename T, typename I, int NMAX>
struct TableKernelArgs {
    T c[NMAX];
    I off[NMAX];
    int n, ncomp, init_zero;
    long long svol, dvol;      // component strides
    long long sx, sy, sz;      // source steps per index-box step
    long long dx, dy, dz;      // destination steps per index-box step
};
template <typename T, typename I, int NMAX>
__global__ void __launch_bounds__(kWalkThreads) k_table(const T* __restrict__ src, T* dst,
                                                        const __grid_constant__ TableKernelArgs<T, I, NMAX> a, Walk w)
{
    for (int c = blockIdx.z; c < a.ncomp; c += gridDim.z) {
        const T* sp = src + c * a.svol;
        T* dp = dst + c * a.dvol;
        walk_items(w, [&](int x, int y, int z, int) {
            T* dq = dp + a.dx * x + a.dy * y + a.dz * z;
            const I at = (I)(a.sx * x + a.sy * y + a.sz * z);
            T acc = a.init_zero ? T(0) : *dq;
#pragma unroll kTableTerms
            for (int j = 0; j < a.n; j++) acc = dadd(acc, dmul(a.c[j], __ldg(sp + a.off[j] + at)));
            *dq = acc;
        });
    }
}

// The 19- and 27-point Laplacians (centre, then the other points of the 3^3 cube, z slowest and x
// fastest; the 19-point table leaves out the corners): a thread walks a column of zd planes, reading each
// plane's nine values once (the table kernel issues 27 loads a cell). In the table's order the terms of
// the plane above come last, so a cell's sum is carried over from the step that completes its lower two
// planes, and only the previous, the current and the next plane (on its way, a whole step early) are in
// registers. Bound by FP64 issue (27 multiplies and 27 adds, each rounded: 12 us at 3.95 M cells) and
// load latency. Measured (B200, two components of 193 x 161 x 127 FP64 cells): 68 us a component one cell
// per thread, 43 with the three planes held, 33 with the next plane loaded a step early, 28 with four more
// asked into L2. Below kCubeMin cells the columns are too few to fill the GPU (16^3: 2.88 us, table 2.84;
// 24^3 2.84 / 3.15; 33^3 2.95 / 3.23), and boxes thin along an axis leave its threads idle (share of steps
// that give a cell: 256 x 256 x 2 0.5, 3.1 / 4.1; 2048 x 2048 x 1 0.33, 78 / 57; 2 x 1024 x 1024 0.25, 45 / 30).
constexpr long long kCubeMin = 1 << 15;
constexpr double kCubeShare = 0.4;
constexpr int kCubeThreads = 128, kCubePerSm = 5;
constexpr int kCubePrefetch = 4;   // planes past the next one whose lines are asked into L2
template <typename T>
struct CubeArgs {
    T c[27];                    // by cube position (z+1)*9 + (y+1)*3 + (x+1)
    int ncomp, init_zero, zd, chunks;
    int nx, ny, nz, lx;         // lx: log2 of the lanes along x
    long long svol, dvol;
};
template <typename T, bool CORNERS>
__global__ void __launch_bounds__(kCubeThreads, kCubePerSm) k_cube(FieldView<const T> s, FieldView<T> d,
                                                                   const __grid_constant__ CubeArgs<T> a)
{
    const int lane = threadIdx.x & ((1 << a.lx) - 1), row = threadIdx.x >> a.lx;
    const int x = blockIdx.x * (1 << a.lx) + lane, y = blockIdx.y * (kCubeThreads >> a.lx) + row;
    if (x >= a.nx || y >= a.ny) return;
    for (int u = blockIdx.z; u < a.chunks * a.ncomp; u += gridDim.z) {
        const int comp = u / a.chunks, z0 = (u - comp * a.chunks) * a.zd, z1 = min(z0 + a.zd, a.nz);
        const T* q = s.p + comp * a.svol + x + s.sy * y + s.sz * (z0 - 1);   // the next plane to load
        T* o = d.p + comp * a.dvol + x + d.sy * y + d.sz * z0;               // the next cell to start
        auto load = [&](T* p) {
#pragma unroll
            for (int k = 0; k < 9; k++) p[k] = __ldg(q + (k % 3 - 1) + s.sy * (k / 3 - 1));
            q += s.sz;
        };
        auto term = [&](T& acc, int k, T v) {
            const int dist = (k / 9 != 1) + ((k / 3) % 3 != 1) + (k % 3 != 1);
            if (dist != 0 && (CORNERS || dist != 3)) acc = dadd(acc, dmul(a.c[k], v));
        };
        T acc = T(0);
        // plane z of the chunk in cur, z - 1 in prev, z + 1 on its way into next: completes cell z - 1
        // (its upper plane), then starts cell z
        auto step = [&](const T* prev, const T* cur, T* next, int z) {
            if (z < z1) load(next);               // moves q to plane z + 2
            if (z + 1 + kCubePrefetch <= z1) prefetch_l2(q + (kCubePrefetch - 1) * s.sz);
            if (z > z0) {
#pragma unroll
                for (int k = 18; k < 27; k++) term(acc, k, cur[k - 18]);
                *(o - d.sz) = acc;
            }
            if (z < z1) {
                acc = a.init_zero ? T(0) : *o;
                acc = dadd(acc, dmul(a.c[13], cur[4]));
#pragma unroll
                for (int k = 0; k < 9; k++) term(acc, k, prev[k]);
#pragma unroll
                for (int k = 9; k < 18; k++) term(acc, k, cur[k - 9]);
                o += d.sz;
            }
        };
        T p0[9], p1[9], p2[9];
#pragma unroll
        for (int k = 0; k <= kCubePrefetch; k++)
            if (z0 + k <= z1) prefetch_l2(q + (k + 1) * s.sz);
        load(p0);
        load(p1);
        for (int z = z0; z <= z1; z += 3) {
            step(p0, p1, p2, z);
            if (z + 1 > z1) break;
            step(p1, p2, p0, z + 1);
            if (z + 2 > z1) break;
            step(p2, p0, p1, z + 2);
        }
    }
}

// ---- host-side stencil object -----------------------------------------------------------------
} // namespace pb

struct pb_stencil {
    std::vector<double> coefs;
    std::vector<int> offs;   // n x 3
    int sr[3], dr[3], ds[3];
    int spanLo[3], spanHi[3];
    int shape;               // 0 table, 1 Lap7, 2 Lap13
    int cube = 0;            // shape 0 on the 3^3 cube in StencilLib's order: 19 or 27 points (0: neither)
};

namespace pb {

template <class S>
static bool matches_shape(const pb_stencil* s)
{
    if ((int)s->coefs.size() != S::NT) return false;
    for (int d = 0; d < 3; d++)
        if (s->sr[d] != 1 || s->dr[d] != 1 || s->ds[d] != 0) return false;
    for (int j = 0; j < S::NT; j++)
        for (int d = 0; d < 3; d++)
            if (s->offs[3 * j + d] != S::off(j, d)) return false;
    return true;
}

// 27 (or 19) when the table is StencilLib's 27-point (19-point) one: the centre, then the cube's other
// points (without its corners) with z slowest and x fastest, ratios 1 and no shift; 0 otherwise
static int matches_cube(const pb_stencil* s)
{
    const int n = (int)s->coefs.size();
    if (n != 27 && n != 19) return 0;
    for (int d = 0; d < 3; d++)
        if (s->sr[d] != 1 || s->dr[d] != 1 || s->ds[d] != 0 || s->offs[d] != 0) return 0;
    int j = 1;
    for (int k = 0; k < 27; k++) {
        const int o[3] = {k % 3 - 1, (k / 3) % 3 - 1, k / 9 - 1};
        const int dist = (o[0] != 0) + (o[1] != 0) + (o[2] != 0);
        if (dist == 0 || (n == 19 && dist == 3)) continue;
        for (int d = 0; d < 3; d++)
            if (s->offs[3 * j + d] != o[d]) return 0;
        j++;
    }
    return n;
}

// scale folded into the coefficients as Stencil::hostApply does (Proto_StencilImplem.H:771-779)
template <typename T>
static inline T fold(double c, T scale)
{
    return scale != T(1) ? (T)c * scale : (T)c;
}

int cached_sm_count()
{
    static int sms = 0;
    if (sms == 0) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (sms <= 0) sms = 148;
    }
    return sms;
}

int grid_for(long long total, int threads)
{
    long long b = (total + threads - 1) / threads;
    long long cap = (long long)cached_sm_count() * 16;
    if (b > cap) b = cap;
    if (b < 1) b = 1;
    return (int)b;
}

int stencil_coefs(const pb_stencil* s, double* c, int cap)
{
    int n = (int)s->coefs.size();
    for (int j = 0; j < n && j < cap; j++) c[j] = s->coefs[j];
    return n;
}

static StarTune g_default_tune;
StarTune& default_star_tune() { return g_default_tune; }

} // namespace pb

// Launch-shape knobs of the star kernels (used by the autotuner and by profiling sweeps):
// mode 0 auto / 1 TMA only / 2 simple only; zc z-chunk (0 heuristic); (ty, yb, xv) CTA tile height,
// rows per consumer thread and adjacent x points per consumer thread (xv 0: one point per thread
// for Stencil::apply, two for the multigrid sweeps).
extern "C" int pb_star_tune_set(int mode, int zc, int ty, int yb, int xv, long long min_tma_points)
{
    const bool shape_ok = (ty == 8 && yb == 1 && xv == 1) || (ty == 8 && yb == 2 && xv >= 0 && xv <= 2) ||
                          (ty == 4 && yb == 2 && xv == 2);
    if (mode < 0 || mode > 2 || zc < 0 || !shape_ok) return PB_ERR_ARG;
    pb::StarTune& t = pb::default_star_tune();
    t.mode = mode;
    t.zc = zc;
    t.ty = ty;
    t.yb = yb;
    t.xv = xv;
    if (min_tma_points >= 0) t.min_tma_points = min_tma_points;
    return PB_OK;
}

extern "C" int pb_star_tune_ring(int nst, int aux_smem)
{
    if (nst != 0 && (nst < 3 || nst > 16)) return PB_ERR_ARG;
    if (aux_smem != 0 && aux_smem != 1) return PB_ERR_ARG;
    pb::StarTune& t = pb::default_star_tune();
    t.nst = nst;
    t.aux_smem = aux_smem;
    return PB_OK;
}

namespace pb {

// ---- apply dispatch ---------------------------------------------------------------------------
static inline OutMap out_map(const Box3& ib, const Box3& db)
{
    OutMap m;
    m.dx = ib.lo[0] - db.lo[0];
    m.dy = ib.lo[1] - db.lo[1];
    m.dz = ib.lo[2] - db.lo[2];
    m.Dx = bsize(db, 0);
    m.Dxy = bsize(db, 0) * bsize(db, 1);
    return m;
}

// Validate / infer the index box; returns PB_OK or an error status.
static int resolve_box(const pb_stencil* s, const Box3& sb, const Box3& db, pb_box box, Box3* out)
{
    Box3 ib = to_box(box);
    if (bempty(ib)) {
        // indexDomain(dst) & indexRange(src) (Proto_StencilImplem.H:324-346)
        Box3 r, d;
        for (int k = 0; k < 3; k++) {
            r.lo[k] = sb.lo[k] - s->spanLo[k];
            r.hi[k] = sb.hi[k] - s->spanHi[k];
            d.lo[k] = db.lo[k] - s->ds[k];
            d.hi[k] = db.hi[k] - s->ds[k];
        }
        ib = intersect(taper_coarsen(r, s->sr), taper_coarsen(d, s->dr));
    }
    // the source must hold every point the terms read
    if (!bempty(ib)) {
        Box3 need;
        for (int k = 0; k < 3; k++) {
            need.lo[k] = ib.lo[k] * s->sr[k] + s->spanLo[k];
            need.hi[k] = ib.hi[k] * s->sr[k] + s->spanHi[k];
        }
        if (!contains_box(sb, need)) return PB_ERR_GHOST;
    }
    *out = ib;
    return PB_OK;
}

// the index-box points whose destination lies in the destination box
static Box3 clip_to_dst(const pb_stencil* s, Box3 ib, const Box3& db)
{
    for (int k = 0; k < 3; k++) {
        const int lo = ceil_div(db.lo[k] - s->ds[k], s->dr[k]), hi = floor_div(db.hi[k] - s->ds[k], s->dr[k]);
        if (ib.lo[k] < lo) ib.lo[k] = lo;
        if (ib.hi[k] > hi) ib.hi[k] = hi;
    }
    return ib;
}

template <typename T, typename I, int NMAX>
static int launch_table(const pb_stencil* s, const T* src, const Box3& sb, T* dst, const Box3& db, const Box3& ib,
                        int ncomp, int init_to_zero, T scale, int n, cudaStream_t st)
{
    const Region rg = region_of(ib);
    const Walk w = walk_of(rg, 1);
    const long long sS[3] = {1, bsize(sb, 0), bsize(sb, 0) * bsize(sb, 1)};
    const long long dS[3] = {1, bsize(db, 0), bsize(db, 0) * bsize(db, 1)};
    TableKernelArgs<T, I, NMAX> a;
    a.n = n;
    a.ncomp = ncomp;
    a.init_zero = init_to_zero ? 1 : 0;
    a.svol = bvol(sb);
    a.dvol = bvol(db);
    a.sx = sS[0] * s->sr[0];
    a.sy = sS[1] * s->sr[1];
    a.sz = sS[2] * s->sr[2];
    a.dx = dS[0] * s->dr[0];
    a.dy = dS[1] * s->dr[1];
    a.dz = dS[2] * s->dr[2];
    // first: the span's low corner at the first point (inside the source box when a term is read)
    for (int d = 0; d < 3; d++) {
        if (n > 0) src += sS[d] * ((long long)ib.lo[d] * s->sr[d] + s->spanLo[d] - sb.lo[d]);
        dst += dS[d] * ((long long)ib.lo[d] * s->dr[d] + s->ds[d] - db.lo[d]);
    }
    for (int j = 0; j < n; j++) {
        a.c[j] = fold<T>(s->coefs[j], scale);
        long long o = 0;
        for (int d = 0; d < 3; d++) o += sS[d] * (s->offs[3 * j + d] - s->spanLo[d]);
        a.off[j] = (I)o;
    }
    k_table<T, I, NMAX><<<walk_grid(w, ncomp), kWalkThreads, 0, st>>>(src, dst, a, w);
    PB_LAUNCH_CHECK();
    return PB_OK;
}

// log2 of the column kernel's lanes along x: short rows take more rows per block, with fewer idle lanes
static int cube_lanes(long long nx)
{
    int lx = 5;
    while (lx > 3 && (1 << (lx - 1)) >= nx) lx--;
    return lx;
}
// share of the column kernel's thread steps that give a cell (a column starts with two planes of loads)
static double cube_share(const Box3& b)
{
    const long long n[3] = {bsize(b, 0), bsize(b, 1), bsize(b, 2)};
    const int lx = cube_lanes(n[0]), lanes = 1 << lx, rows = kCubeThreads >> lx;
    auto full = [](long long v, int m) { return (double)v / (double)((v + m - 1) / m * m); };
    return full(n[0], lanes) * full(n[1], rows) * n[2] / (n[2] + 2.0);
}

template <typename T>
static int launch_cube(const pb_stencil* s, const T* src, const Box3& sb, T* dst, const Box3& db, const Box3& ib,
                       int ncomp, int init_to_zero, T scale, cudaStream_t st)
{
    const Region rg = region_of(ib);
    CubeArgs<T> a{};
    a.ncomp = ncomp;
    a.init_zero = init_to_zero ? 1 : 0;
    a.svol = bvol(sb);
    a.dvol = bvol(db);
    for (int j = 0; j < (int)s->coefs.size(); j++)
        a.c[(s->offs[3 * j + 2] + 1) * 9 + (s->offs[3 * j + 1] + 1) * 3 + s->offs[3 * j] + 1] = fold<T>(s->coefs[j], scale);
    a.nx = rg.n[0];
    a.ny = rg.n[1];
    a.nz = rg.n[2];
    a.lx = cube_lanes(a.nx);
    const int rows = kCubeThreads >> a.lx, gx = (a.nx + (1 << a.lx) - 1) >> a.lx, gy = (a.ny + rows - 1) / rows;
    // the z chunk that makes waves of resident blocks x (planes + 2) smallest: a chunk starts with two
    // planes of loads beyond its own
    const long long slots = (long long)kCubePerSm * cached_sm_count();
    long long best = -1;
    for (int zd = 4; zd < a.nz + 4; zd += zd < 64 ? 4 : 16) {
        const long long blocks = (long long)gx * gy * ((a.nz + zd - 1) / zd) * ncomp;
        const long long cost = (blocks + slots - 1) / slots * (zd + 2);
        if (best < 0 || cost < best) {
            best = cost;
            a.zd = zd;
        }
    }
    a.chunks = (a.nz + a.zd - 1) / a.zd;
    const long long gz = (long long)a.chunks * ncomp;
    const dim3 grid(gx, gy, (unsigned)(gz < 65535 ? gz : 65535));
    const FieldView<const T> sv = view_of(src, sb, rg);
    const FieldView<T> dv = view_of(dst, db, rg);
    if (s->cube == 27) k_cube<T, true><<<grid, kCubeThreads, 0, st>>>(sv, dv, a);
    else k_cube<T, false><<<grid, kCubeThreads, 0, st>>>(sv, dv, a);
    PB_LAUNCH_CHECK();
    return PB_OK;
}

template <typename T>
static int apply_impl(const pb_stencil* s, const T* src, pb_box src_box, T* dst, pb_box dst_box, pb_box box,
                      int ncomp, int init_to_zero, T scale, cudaStream_t st)
{
    if (!s || !src || !dst || ncomp < 1) return PB_ERR_ARG;
    Box3 sb = to_box(src_box), db = to_box(dst_box), ib;
    if (bempty(sb) || bempty(db)) return PB_ERR_BOX;
    int e = resolve_box(s, sb, db, box, &ib);
    if (e != PB_OK) return e;
    if (bempty(ib) || s->coefs.empty()) return PB_OK;
    if (scale == T(0)) {
        // the reference zeroes the destination for "|=" and does nothing else
        if (!init_to_zero) return PB_OK;
        ib = clip_to_dst(s, ib, db);
        if (bempty(ib)) return PB_OK;
        return launch_table<T, unsigned, 32>(s, src, sb, dst, db, ib, ncomp, 1, scale, 0, st);
    }
    const long long svol = bvol(sb), dvol = bvol(db);
    if (s->shape == 1 || s->shape == 2) {
        // star kernels: destination ratio 1, no shift -> clip to the destination box
        Box3 cib = intersect(ib, db);
        if (bempty(cib)) return PB_OK;
        Coefs<T> cf;
        for (int j = 0; j < (int)s->coefs.size(); j++) cf.c[j] = fold<T>(s->coefs[j], scale);
        for (int c = 0; c < ncomp; c++) {
            EpiStore<T> epi;
            epi.dst = dst + c * dvol;
            epi.m = out_map(cib, db);
            epi.accumulate = !init_to_zero;
            int r = (s->shape == 1) ? launch_star<ShapeLap7>(src + c * svol, sb, cib, cf, epi, st, default_star_tune())
                                    : launch_star<ShapeLap13>(src + c * svol, sb, cib, cf, epi, st, default_star_tune());
            if (r != PB_OK) return r;
        }
        return PB_OK;
    }
    const int n = (int)s->coefs.size();
    if (n > kMaxTerms) return PB_ERR_UNSUPPORTED;
    ib = clip_to_dst(s, ib, db);
    if (bempty(ib)) return PB_OK;
    if (s->cube && bvol(ib) >= kCubeMin && cube_share(ib) >= kCubeShare && (bsize(ib, 1) + 3) / 4 <= 65535)
        return launch_cube<T>(s, src, sb, dst, db, ib, ncomp, init_to_zero, scale, st);
    if (svol > 0xffffffffLL) return launch_table<T, long long, kMaxTerms>(s, src, sb, dst, db, ib, ncomp, init_to_zero, scale, n, st);
    if (n <= 32) return launch_table<T, unsigned, 32>(s, src, sb, dst, db, ib, ncomp, init_to_zero, scale, n, st);
    return launch_table<T, unsigned, kMaxTerms>(s, src, sb, dst, db, ib, ncomp, init_to_zero, scale, n, st);
}

} // namespace pb

using namespace pb;

extern "C" {

const char* pb_status_string(int s)
{
    switch (s) {
        case PB_OK: return "ok";
        case PB_ERR_ARG: return "invalid argument";
        case PB_ERR_BOX: return "invalid box";
        case PB_ERR_CUDA: return "CUDA runtime error";
        case PB_ERR_ALIGN: return "alignment requirement not met";
        case PB_ERR_NOMEM: return "out of memory";
        case PB_ERR_UNSUPPORTED: return "unsupported request";
        case PB_ERR_BUDGET: return "memory budget exceeded";
        case PB_ERR_DEVICE: return "device-side error flagged";
        case PB_ERR_GHOST: return "source box does not cover the stencil footprint";
    }
    return "unknown status";
}

int pb_last_cuda_error(void) { return t_last_cuda; }

const char* pb_version(void) { return "proto_b200 1.0 sm_100a"; }

int pb_debug_wait_expiry(unsigned int tries, int* expired, void* stream)
{
    if (!expired || tries == 0 || tries > kMaxWaitTries) return PB_ERR_ARG;
    cudaStream_t st = (cudaStream_t)stream;
    k_wait_expiry<<<1, 32, 0, st>>>(tries);
    PB_LAUNCH_CHECK();
    PB_CUDA(cudaStreamSynchronize(st));
    PB_CUDA(cudaMemcpyFromSymbol(expired, g_wait_expired, sizeof(int)));
    return PB_OK;
}

int pb_device_check(void* stream)
{
    cudaStream_t st = (cudaStream_t)stream;
    PB_CUDA(cudaStreamSynchronize(st));
    int a = read_error_stencil(), b = read_error_mg(), c = read_error_serve();
    if (a < 0 || b < 0 || c < 0) return PB_ERR_CUDA;
    return (a || b || c) ? PB_ERR_DEVICE : PB_OK;
}

int pb_stencil_create(const double* coefs, const int* offsets, int nterms, const int src_ratio[3],
                      const int dst_ratio[3], const int dst_shift[3], pb_stencil** out)
{
    if (!out || nterms < 0 || (nterms > 0 && (!coefs || !offsets))) return PB_ERR_ARG;
    pb_stencil* s = new (std::nothrow) pb_stencil;
    if (!s) return PB_ERR_NOMEM;
    s->coefs.assign(coefs, coefs + nterms);
    s->offs.assign(offsets, offsets + 3 * nterms);
    for (int d = 0; d < 3; d++) {
        s->sr[d] = src_ratio ? src_ratio[d] : 1;
        s->dr[d] = dst_ratio ? dst_ratio[d] : 1;
        s->ds[d] = dst_shift ? dst_shift[d] : 0;
        if (s->sr[d] <= 0 || s->dr[d] <= 0) { delete s; return PB_ERR_ARG; }
        s->spanLo[d] = 0;
        s->spanHi[d] = 0;
    }
    // span: Stencil::addCoef grows it with every offset (Proto_StencilImplem.H:238-276)
    for (int j = 0; j < nterms; j++)
        for (int d = 0; d < 3; d++) {
            int v = offsets[3 * j + d];
            if (j == 0 || v < s->spanLo[d]) s->spanLo[d] = v;
            if (j == 0 || v > s->spanHi[d]) s->spanHi[d] = v;
        }
    s->shape = matches_shape<ShapeLap7>(s) ? 1 : matches_shape<ShapeLap13>(s) ? 2 : 0;
    s->cube = matches_cube(s);
    *out = s;
    return PB_OK;
}

int pb_stencil_destroy(pb_stencil* s)
{
    delete s;
    return PB_OK;
}

int pb_stencil_info(const pb_stencil* s, int* nterms, pb_box* span, int* shape)
{
    if (!s) return PB_ERR_ARG;
    if (nterms) *nterms = (int)s->coefs.size();
    if (span)
        for (int d = 0; d < 3; d++) { span->lo[d] = s->spanLo[d]; span->hi[d] = s->spanHi[d]; }
    if (shape) *shape = s->shape;
    return PB_OK;
}

int pb_stencil_apply_f64(const pb_stencil* s, const double* src, pb_box src_box, double* dst, pb_box dst_box,
                         pb_box box, int ncomp, int init_to_zero, double scale, void* stream)
{
    return apply_impl<double>(s, src, src_box, dst, dst_box, box, ncomp, init_to_zero, scale, (cudaStream_t)stream);
}

int pb_stencil_apply_f32(const pb_stencil* s, const float* src, pb_box src_box, float* dst, pb_box dst_box,
                         pb_box box, int ncomp, int init_to_zero, float scale, void* stream)
{
    return apply_impl<float>(s, src, src_box, dst, dst_box, box, ncomp, init_to_zero, scale, (cudaStream_t)stream);
}

int pb_stencil_apply_fused_f64(const pb_stencil* s, int epilogue, const double* u, pb_box u_box, double* out,
                               pb_box out_box, pb_box box, double scale, double a, double b, void* stream)
{
    if (!s || !u || !out) return PB_ERR_ARG;
    if (epilogue != PB_EPI_AXPBY && epilogue != PB_EPI_EULER) return PB_ERR_ARG;
    if (s->shape != 1 && s->shape != 2) return PB_ERR_UNSUPPORTED;
    Box3 sb = to_box(u_box), db = to_box(out_box), ib;
    if (bempty(sb) || bempty(db)) return PB_ERR_BOX;
    int e = resolve_box(s, sb, db, box, &ib);
    if (e != PB_OK) return e;
    ib = intersect(ib, db);
    if (bempty(ib)) return PB_OK;
    Coefs<double> cf;
    for (int j = 0; j < (int)s->coefs.size(); j++) cf.c[j] = fold<double>(s->coefs[j], scale);
    EpiAxpby<double> epi;
    epi.dst = out;
    epi.m = out_map(ib, db);
    epi.a = a;
    epi.b = b;
    epi.euler = (epilogue == PB_EPI_EULER);
    cudaStream_t st = (cudaStream_t)stream;
    return (s->shape == 1) ? launch_star<ShapeLap7>(u, sb, ib, cf, epi, st, default_star_tune())
                           : launch_star<ShapeLap13>(u, sb, ib, cf, epi, st, default_star_tune());
}

} // extern "C"
