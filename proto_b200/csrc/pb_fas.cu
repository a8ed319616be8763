// FAS multigrid with the 4th-order flux-form Laplacian (C ABI: pb_fas_*).
//
// Reference counterparts (paths within the reference project):
//   LevelMultigridSolver::solve / resnorm ....... include/utils/implem/Proto_LevelMultigridSolverImplem.H:85-159
//   MGLevel::relax / coarseForce / fineCorrect / vCycle ..................... same file :261-433
//   BoxOp::operator() (flux divergence, fluxScale) include/base/implem/Proto_BoxOpImplem.H:125-172
//   BoxOp_Laplace::flux (DiffCellToFace(d, Lo, 4)) examples/_common/BoxOp_Laplace.H:22-27
//   averageDown .................................. include/base/implem/Proto_LevelBoxDataImplem.H:993-1038
// The reference evaluates the operator patch by patch through four temporaries (three face-flux
// BoxData and a divergence) after an exchange; here every level is one periodic box and one kernel per
// step evaluates, per cell, the same operations in the same order (face gradients with |=, the divergence
// with +=, the sum, the flux scale -1), so the residual history and the solution are bitwise the
// reference's. A level keeps two ghost columns in x and two ghost rows in y, no ghost planes (the kernels
// wrap z) and no valid edges or corners between them (no tap reads those): a writer then has at most one
// image per axis to store beside its cell. With all ghost layers the images cost a sweep of a 128^3 level
// more than its stencil; with none, resolving every neighbour's wrapped address did.
#include <cmath>
#include <cstring>
#include <vector>

#include "pb_internal.cuh"
#include "pb_lap4.cuh"
#include "pb_stencil_impl.cuh"
#include "pb_walk.cuh"

namespace pb {

constexpr int kFasGhost = 2;      // reach of the operator

// index of cell (x, y, z) of a plain n^3 field, and of a level's state (x and y may be ghosts)
__host__ __device__ __forceinline__ long long fas_index(int n, int x, int y, int z)
{
    return x + (long long)n * (y + (long long)n * z);
}
__host__ __device__ __forceinline__ long long fas_state(int n, int x, int y, int z)
{
    const int S = n + 2 * kFasGhost;
    return (x + kFasGhost) + (long long)S * ((y + kFasGhost) + (long long)S * z);
}

// distance of coordinate c's image on a periodic axis of n >= 4 cells (0: none)
__device__ __forceinline__ int fas_image(int c, int n) { return c < kFasGhost ? n : (c >= n - kFasGhost ? -n : 0); }

// the ghost cells that are images of the valid cell at q, edges below 4 (several images per axis)
__device__ __noinline__ void fas_images_small(double* q, int n, int x, int y, double v)
{
    const int S = n + 2 * kFasGhost;
    for (int k = -2; k <= 2; k++) {
        if (k == 0) continue;
        if (x + k * n >= -kFasGhost && x + k * n < n + kFasGhost) q[k * n] = v;
        if (y + k * n >= -kFasGhost && y + k * n < n + kFasGhost) q[k * n * S] = v;
    }
}

// v to the valid cell at q and to its ghost images in x and y (SMALL: edges below 4)
template <bool SMALL>
__device__ __forceinline__ void fas_store(double* q, int n, int x, int y, double v)
{
    *q = v;
    if constexpr (SMALL) {
        fas_images_small(q, n, x, y, v);
        return;
    }
    const int ix = fas_image(x, n), iy = fas_image(y, n) * (n + 2 * kFasGhost);
    if (ix) q[ix] = v;
    if (iy) q[iy] = v;
}

// ---- the level passes: epilogues of the march (pb_lap4.cuh); op(u) = -t -------------------------------
// Jacobi sweep: out = u + (-lambda) * (op(u) + f). FIRST: the level has just
// been averaged into and f holds only AvgDown(op(u) + f) of the finer level; the coarse force is that
// minus op of this level's state, which is the op this sweep evaluates anyway, so the sweep completes
// and stores it (one launch and one pass less per level). Measured (B200, FP64, data in L2): a 128^3 sweep
// 22.5 -> 17.6 us, 64^3 7.8 -> 5.7.
// SMALL: edges below 4, where a cell has several images per axis. NORM: also max |op(u) + f| of the state
// the sweep starts from, into result (Reduction<Abs>: NaN ignored): the solver's test of a cycle rides on
// the next cycle's first sweep, which writes the other buffer, so the state measured stays intact.
template <bool FIRST, bool SMALL, bool NORM = false>
struct EpiFasRelax {
    double* out;
    double* f;
    int n;
    double neg_lambda;
    double* result = nullptr;
    double m = 0.0;
    struct Cursor {
        double* o;           // (x, y, plane z) of the output state
        double* f;           // of the force
        int x, y;
        int ix, iy0, iy1;    // offsets of the cells' images in x and, row by row, in y (edges >= 4)
        bool a0, a1;
    };
    __device__ __forceinline__ Cursor cursor(int x, int y, int z0, bool a0, bool a1) const
    {
        const int S = n + 2 * kFasGhost;
        return Cursor{out + fas_state(n, x, y, z0), f + fas_index(n, x, y, z0), x, y,
                      fas_image(x, n), fas_image(y, n) * S, fas_image(y + 1, n) * S, a0, a1};
    }
    __device__ __forceinline__ void pre(const Cursor& c, int ahead, double& p0, double& p1) const
    {
        const double* q = c.f + (ahead ? n * n : 0);
        if (c.a0) p0 = q[0];
        if (c.a1) p1 = q[n];
    }
    __device__ __forceinline__ void cells(Cursor& c, int, double t0, double t1, double c0, double c1, double p0, double p1)
    {
        const int S = n + 2 * kFasGhost;
        if (NORM) {
            if (c.a0) m = upd_abs(m, dsub(p0, t0));
            if (c.a1) m = upd_abs(m, dsub(p1, t1));
        }
        if (FIRST) {
            p0 = dadd(p0, t0);
            p1 = dadd(p1, t1);
            if (c.a0) c.f[0] = p0;
            if (c.a1) c.f[n] = p1;
        }
        const double v0 = dadd(c0, dmul(neg_lambda, dsub(p0, t0))), v1 = dadd(c1, dmul(neg_lambda, dsub(p1, t1)));
        double* const o1 = c.o + S;
        if (c.a0) c.o[0] = v0;
        if (c.a1) o1[0] = v1;
        if constexpr (SMALL) {
            if (c.a0) fas_images_small(c.o, n, c.x, c.y, v0);
            if (c.a1) fas_images_small(o1, n, c.x, c.y + 1, v1);
        } else {
            if (c.a0 && c.ix) c.o[c.ix] = v0;
            if (c.a0 && c.iy0) c.o[c.iy0] = v0;
            if (c.a1 && c.ix) o1[c.ix] = v1;
            if (c.a1 && c.iy1) o1[c.iy1] = v1;
        }
        c.o += S * S;
        c.f += n * n;
    }
    __device__ __forceinline__ void end() const
    {
        if (NORM) block_max_atomic(m, result);
    }
};

// To the coarser level, in one pass over the finer: coarse state = AvgDown(u) and its copy
// c0, and AvgDown(op(u) + f), the first part of the coarse force. A thread's two rows of an even and an
// odd plane and its x neighbour's (a shuffle away) are a coarse cell's eight children, added in their
// order; the even lanes keep the sums.
template <bool SMALL>   // the coarse edge is below 4
struct EpiFasRestrict {
    const double* f;
    int n;
    double* uc;
    double* c0;
    double* fc;
    double ar, au;
    struct Cursor {
        const double* f;
        int x, y;
        bool a0;
    };
    __device__ __forceinline__ Cursor cursor(int x, int y, int z0, bool a0, bool) const
    {
        return Cursor{f + x + (long long)n * (y + (long long)n * z0), x, y, a0};
    }
    __device__ __forceinline__ void pre(const Cursor& c, int ahead, double& p0, double& p1) const
    {
        const double* q = c.f + (ahead ? n * n : 0);
        p0 = __ldg(q);           // idle threads follow a cell of the level, whose edge is even
        p1 = c.y + 1 < n ? __ldg(q + n) : 0.0;
    }
    __device__ __forceinline__ static void add4(double& acc, double v0, double v1)
    {
        const double w0 = __shfl_down_sync(0xffffffffu, v0, 1), w1 = __shfl_down_sync(0xffffffffu, v1, 1);
        acc = dadd(acc, dmul(0.125, v0));
        acc = dadd(acc, dmul(0.125, w0));
        acc = dadd(acc, dmul(0.125, v1));
        acc = dadd(acc, dmul(0.125, w1));
    }
    __device__ __forceinline__ void cells(Cursor& c, int z, double t0, double t1, double u0, double u1, double p0, double p1)
    {
        if ((z & 1) == 0) ar = au = 0.0;
        add4(ar, dsub(p0, t0), dsub(p1, t1));
        add4(au, u0, u1);
        if ((z & 1) && c.a0 && (c.x & 1) == 0) {
            const long long i = fas_index(n / 2, c.x / 2, c.y / 2, z / 2);
            fc[i] = ar;
            c0[i] = au;
            fas_store<SMALL>(uc + fas_state(n / 2, c.x / 2, c.y / 2, z / 2), n / 2, c.x / 2, c.y / 2, au);
        }
        c.f += n * n;
    }
    __device__ __forceinline__ void end() const {}
};

// fine correction: u += -(c0 - uc) of the cell's coarse cell (c0: the coarse state as it was averaged,
// uc: as the coarse cycle left it). An item walk with four planes' loads in flight.
template <bool SMALL>
__global__ void __launch_bounds__(kWalkThreads) k_fas_correct(double* u, const double* __restrict__ c0,
                                                              const double* __restrict__ uc, int nf, Walk w)
{
    const int nc = nf / 2, S = nf + 2 * kFasGhost, Sc = nc + 2 * kFasGhost;
    const long long nf2 = (long long)S * S, nc2 = (long long)nc * nc, sc2 = (long long)Sc * Sc;
    walk_items(w, [&](int x, int y, int z, int planes) {          // z is even: planes z, z+1 share a coarse one
        double* q = u + fas_state(nf, x, y, z);
        const double* a = c0 + fas_index(nc, x / 2, y / 2, z / 2);
        const double* b = uc + fas_state(nc, x / 2, y / 2, z / 2);
        double v[kWalkZ], d[kWalkZ / 2];
#pragma unroll
        for (int k = 0; k < kWalkZ; k++)
            if (k < planes) v[k] = q[k * nf2];
#pragma unroll
        for (int k = 0; k < kWalkZ / 2; k++)
            if (2 * k < planes) d[k] = dsub(__ldg(a + k * nc2), __ldg(b + k * sc2));
#pragma unroll
        for (int k = 0; k < kWalkZ; k++)
            if (k < planes) fas_store<SMALL>(q + k * nf2, nf, x, y, dsub(v[k], d[k / 2]));
    });
}

// n^3 <-> state, x and y ghosts included
__global__ void __launch_bounds__(kWalkThreads) k_fas_pack(const double* __restrict__ src, double* u, int n, Walk w)
{
    const long long S = n + 2 * kFasGhost;
    walk_items(w, [&](int x, int y, int z, int planes) {          // x, y of the grown plane
        const double* q = src + lap4_wrap(x - kFasGhost, n) + (long long)n * (lap4_wrap(y - kFasGhost, n) + (long long)n * z);
        double* o = u + x + S * (y + S * z);
        double v[kWalkZ];
#pragma unroll
        for (int k = 0; k < kWalkZ; k++)
            if (k < planes) v[k] = __ldg(q + (long long)n * n * k);
#pragma unroll
        for (int k = 0; k < kWalkZ; k++)
            if (k < planes) o[S * S * k] = v[k];
    });
}
__global__ void __launch_bounds__(kWalkThreads) k_fas_unpack(const double* __restrict__ u, double* dst, int n, Walk w)
{
    const long long S = n + 2 * kFasGhost;
    walk_items(w, [&](int x, int y, int z, int planes) {
        double v[kWalkZ];
#pragma unroll
        for (int k = 0; k < kWalkZ; k++)
            if (k < planes) v[k] = __ldg(u + fas_state(n, x, y, z) + S * S * k);
#pragma unroll
        for (int k = 0; k < kWalkZ; k++)
            if (k < planes) dst[fas_index(n, x, y, z + k)] = v[k];
    });
}

// ---- the levels of edge <= kFasCoarseEdge in one CTA ------------------------------------------
// The same per-cell operations as the passes above, in the same order (sweeps, averaging, coarse
// force, recursion, correction), with every level's state (two buffers), force and averaged copy in
// shared memory, a cell per thread whose neighbours' indices stay in registers. One launch replaces about
// thirty launch-bound ones: 18 us (46 with the levels in L2 and their images stored). A 16^3 level keeps
// its own launches: its sweep is more FP64 work than one SM does in a launch's time (with it: 139 us).
constexpr int kFasCoarseEdge = 8, kFasCoarseMax = 8, kFasCoarseThreads = 512;

struct FasCoarseLevel {
    int n;
    FasCoef k;
    double neg_lambda;
    int u[2], f, c0;         // offsets in shared memory (doubles)
};
struct FasCoarseArgs {
    FasCoarseLevel lv[kFasCoarseMax];   // 0 = coarsest
    int top;                            // index of the entry level
    int num_pre, num_post, num_bottom;
    double* u;                          // entry level: state (in and out) and force without its op part
    const double* f;
};

#define FAS_BLOCK_LOOP(total) for (int i = threadIdx.x; i < (total); i += blockDim.x)

// A level has at most one cell per thread (8^3 = 512): the thread's cell and its neighbours' indices
static_assert(kFasCoarseEdge * kFasCoarseEdge * kFasCoarseEdge <= kFasCoarseThreads, "a thread per cell");
struct FasCell {
    int nb[3][4];            // per axis the cells at -2, -1, +1, +2
    bool in;
    __device__ __forceinline__ FasCell(int n)
    {
        const int i = threadIdx.x, step[3] = {1, n, n * n}, p[3] = {i % n, i / n % n, i / (n * n)};
        in = i < n * n * n;
#pragma unroll
        for (int d = 0; d < 3; d++)
#pragma unroll
            for (int o = 0; o < 4; o++)
                nb[d][o] = in ? i + (lap4_wrap(p[d] + (o < 2 ? o - 2 : o - 1), n) - p[d]) * step[d] : 0;
    }
    // t as in the march
    __device__ __forceinline__ double value(const double* u, double c, const FasCoef& k) const
    {
        double v[3][4];
#pragma unroll
        for (int d = 0; d < 3; d++)
#pragma unroll
            for (int o = 0; o < 4; o++) v[d][o] = u[nb[d][o]];
        return lap4_cell(v, c, k);
    }
};

// sweeps from buffer `from`; first: the first sweep completes the force (EpiFasRelax)
__device__ void fas_blk_relax(const FasCoarseLevel& L, double* sm, int from, int sweeps, bool first)
{
    const FasCell cell(L.n);
    const int i = threadIdx.x;
    const FasCoef k = L.k;
    double fv = cell.in ? sm[L.f + i] : 0.0;
    int c = from;
    for (int s = 0; s < sweeps; s++) {
        if (cell.in) {
            const double* u = sm + L.u[c];
            const double centre = u[i], t = cell.value(u, centre, k);
            if (first && s == 0) sm[L.f + i] = fv = dadd(fv, t);
            sm[L.u[1 - c] + i] = dadd(centre, dmul(L.neg_lambda, dsub(fv, t)));
        }
        __syncthreads();
        c = 1 - c;
    }
}

__global__ void __launch_bounds__(kFasCoarseThreads) k_fas_coarse_cycle(const __grid_constant__ FasCoarseArgs a)
{
    extern __shared__ __align__(16) double fas_sm[];
    double* sm = fas_sm;
    {
        const FasCoarseLevel& T = a.lv[a.top];
        FAS_BLOCK_LOOP(T.n * T.n * T.n)
        {
            sm[T.u[0] + i] = a.u[fas_state(T.n, i % T.n, i / T.n % T.n, i / (T.n * T.n))];
            sm[T.f + i] = a.f[i];
        }
    }
    __syncthreads();
    // Every level is entered with its state in buffer 0, so the buffer holding a level's state is
    // fixed by the sweep counts: after the pre-sweeps (and through the correction) pre & 1; at the end,
    // post-sweeps included, (pre + post) & 1; the coarsest level's after its sweeps, bottom & 1.
    const int c_pre = a.num_pre & 1, c_end = (a.num_pre + a.num_post) & 1, c_bot = a.num_bottom & 1;
    // down: pre-sweeps, coarse state and force
    for (int l = a.top; l >= 1; l--) {
        const FasCoarseLevel& L = a.lv[l];
        const FasCoarseLevel& C = a.lv[l - 1];
        fas_blk_relax(L, sm, 0, a.num_pre, true);
        const int nf = L.n, nc = C.n;
        const double* u = sm + L.u[c_pre];
        double* res = sm + L.u[1 - c_pre];       // op(u) + f of the fine cells (n^3), until the next sweep
        {
            const FasCell cell(nf);
            const int i = threadIdx.x;
            if (cell.in) res[i] = dsub(sm[L.f + i], cell.value(u, u[i], L.k));
        }
        __syncthreads();
        FAS_BLOCK_LOOP(nc * nc * nc)
        {
            const int x = i % nc, y = i / nc % nc, z = i / (nc * nc);
            double ar = 0.0, au = 0.0;
#pragma unroll
            for (int c = 0; c < 8; c++) {
                const int q = 2 * x + (c & 1) + nf * (2 * y + ((c >> 1) & 1) + nf * (2 * z + (c >> 2)));
                ar = dadd(ar, dmul(0.125, res[q]));
                au = dadd(au, dmul(0.125, u[q]));
            }
            sm[C.f + i] = ar;
            sm[C.c0 + i] = au;
            sm[C.u[0] + i] = au;
        }
        __syncthreads();
    }
    fas_blk_relax(a.lv[0], sm, 0, a.num_bottom, true);
    // up: correction from the level below, post-sweeps
    for (int l = 1; l <= a.top; l++) {
        const FasCoarseLevel& L = a.lv[l];
        const FasCoarseLevel& C = a.lv[l - 1];
        const int nf = L.n, nc = C.n;
        const double* uc = sm + C.u[l - 1 == 0 ? c_bot : c_end];
        const double* c0 = sm + C.c0;
        double* u = sm + L.u[c_pre];
        FAS_BLOCK_LOOP(nf * nf * nf)
        {
            const int x = i % nf, y = i / nf % nf, z = i / (nf * nf);
            const int q = x / 2 + nc * (y / 2 + nc * (z / 2));
            u[i] = dsub(u[i], dsub(c0[q], uc[q]));
        }
        __syncthreads();
        fas_blk_relax(L, sm, c_pre, a.num_post, false);
    }
    {
        const FasCoarseLevel& T = a.lv[a.top];
        const double* u = sm + T.u[a.top == 0 ? c_bot : c_end];
        FAS_BLOCK_LOOP(T.n * T.n * T.n) a.u[fas_state(T.n, i % T.n, i / T.n % T.n, i / (T.n * T.n))] = u[i];
    }
}

struct FasLevel {
    int n;
    double dx;
    FasCoef k;
    double neg_lambda;
    double* u[2] = {nullptr, nullptr};   // ping-pong state (fas_state)
    int cur = 0;
    double* f = nullptr;                  // n^3
    double* c0 = nullptr;                 // n^3: copy of the averaged-down state (coarse levels)
};

static FasCoef fas_coefs(double dx)
{
    static const double base[4] = {1.0, -15.0, 15.0, -1.0};
    const double s = 1.0 / dx;
    FasCoef k;
    for (int t = 0; t < 4; t++) {
        const double c = base[t] * (1.0 / 12.0);
        k.g[t] = (s != 1.0) ? c * s : c;
    }
    k.cp = (s != 1.0) ? 1.0 * s : 1.0;
    return k;
}

// BoxOp<BoxOp_Laplace>::operator() on a box: out = ((0 + div) * flux_scale) [* scale], the march of
// pb_lap4.cuh with the field's own strides. Measured (B200, 160^3): 39.5 -> 26.6 us against one cell per
// thread.
struct EpiBoxOp {
    double* out;             // cell (0, 0, 0) of the range
    long long sy, sz;
    double flux_scale, scale;
    int apply_scale;
    struct Cursor {
        double* o;
        bool a0, a1;
    };
    __device__ __forceinline__ Cursor cursor(int x, int y, int z0, bool a0, bool a1) const
    {
        return Cursor{out + x + sy * y + sz * z0, a0, a1};
    }
    __device__ __forceinline__ void pre(const Cursor&, int, double&, double&) const {}
    __device__ __forceinline__ double value(double t) const
    {
        const double v = dmul(t, flux_scale);
        return apply_scale ? dmul(v, scale) : v;
    }
    __device__ __forceinline__ void cells(Cursor& c, int, double t0, double t1, double, double, double, double) const
    {
        if (c.a0) c.o[0] = value(t0);
        if (c.a1) c.o[sy] = value(t1);
        c.o += sz;
    }
    __device__ __forceinline__ void end() const {}
};

// The same for boxes that would leave most of the march's threads idle: a cell per thread.
__global__ void __launch_bounds__(kWalkThreads) k_boxop_cells(FieldView<const double> u, EpiBoxOp epi, FasCoef k, Walk w)
{
    walk_items(w, [&](int x, int y, int z, int) {
        const double* q = u.p + x + u.sy * y + u.sz * z;
        const long long step[3] = {1, u.sy, u.sz};
        double v[3][4];
#pragma unroll
        for (int d = 0; d < 3; d++)
#pragma unroll
            for (int o = 0; o < 4; o++) v[d][o] = __ldg(q + (o < 2 ? o - 2 : o - 1) * step[d]);
        epi.out[x + epi.sy * y + epi.sz * z] = epi.value(lap4_cell(v, __ldg(q), k));
    });
}

// Share of the march's thread steps that give a cell: rows of 32 lanes, pairs of rows in blocks of 8 or 4
// rows, and a chunk's start. Measured (B200, us, march / cells): 160^3 (share 0.99) 19.1 / 26.1, 512 x 512 x 4
// (0.73) 7.0 / 8.0, 100^3 (0.69) 7.5 / 7.7, 65 x 129 x 200 (0.60) 13.0 / 11.6, 48 x 50 x 52 (0.57) 3.1 / 2.5,
// 33^3 (0.34) 2.4 / 2.2, 1 x 2048 x 2048 (0.03) 489 / 45.
constexpr double kBoxOpMarch = 0.65;
static double boxop_march_share(const Region& r)
{
    const double gx = (r.n[0] + 31) / 32 * 32.0, gy = r.n[1] > 8 ? (r.n[1] + 15) / 16 * 16.0 : 8.0;
    return r.n[0] / gx * (r.n[1] / gy) * (r.n[2] / (r.n[2] + 1.5));
}

} // namespace pb

struct pb_fas {
    std::vector<pb::FasLevel> lv;   // 0 = coarsest
    double* d_res = nullptr;
    double* h_res = nullptr;
    int num_pre = 6, num_post = 6, num_bottom = 10;
    // the V-cycle plus the residual norm, captured once per parity of the finest level's buffer
    cudaGraphExec_t graph[2] = {nullptr, nullptr};
    int graph_cur[2] = {0, 0};           // the finest level's buffer after the captured cycle
    cudaStream_t graph_stream = nullptr;
};

using namespace pb;

static Lap4Geom fas_geom(const FasLevel& L)
{
    const long long S = L.n + 2 * kFasGhost;
    return Lap4Geom{L.u[L.cur] + fas_state(L.n, 0, 0, 0), S, S * S, L.n, L.n, L.n, 0, 0};
}

// first: the level's force still lacks its op part (every level below the finest, on the way down)
static int fas_relax(pb_fas* m, int l, int sweeps, bool first, cudaStream_t st)
{
    FasLevel& L = m->lv[l];
    for (int s = 0; s < sweeps; s++) {
        const Lap4Geom g = fas_geom(L);
        double* out = L.u[1 - L.cur];
        const int sms = cached_sm_count();
        const bool fs = first && s == 0;
        int e;
        if (L.n < 4)
            e = fs ? launch_lap4<true>(g, L.k, EpiFasRelax<true, true>{out, L.f, L.n, L.neg_lambda}, sms, st)
                   : launch_lap4<true>(g, L.k, EpiFasRelax<false, true>{out, L.f, L.n, L.neg_lambda}, sms, st);
        else
            e = fs ? launch_lap4<true>(g, L.k, EpiFasRelax<true, false>{out, L.f, L.n, L.neg_lambda}, sms, st)
                   : launch_lap4<true>(g, L.k, EpiFasRelax<false, false>{out, L.f, L.n, L.neg_lambda}, sms, st);
        if (e != PB_OK) return e;
        L.cur = 1 - L.cur;
    }
    return PB_OK;
}

// every level of edge <= kFasCoarseEdge (l and below) in one single-CTA launch; level l's state comes
// and goes in buffer 0 (its parent has just averaged into it)
static int fas_coarse(pb_fas* m, int l, cudaStream_t st)
{
    FasCoarseArgs a;
    memset(&a, 0, sizeof(a));
    int off = 0;
    for (int q = 0; q <= l; q++) {
        const FasLevel& L = m->lv[q];
        const int c = L.n * L.n * L.n;
        a.lv[q] = FasCoarseLevel{L.n, L.k, L.neg_lambda, {off, off + c}, off + 2 * c, off + 3 * c};
        off += (q < l ? 4 : 3) * c;                      // the entry level's averaged copy stays with its parent
    }
    a.top = l;
    a.num_pre = m->num_pre;
    a.num_post = m->num_post;
    a.num_bottom = m->num_bottom;
    FasLevel& T = m->lv[l];
    a.u = T.u[0];
    a.f = T.f;
    const size_t smem = sizeof(double) * (size_t)off;   // 15 KB at most (edge 8)
    k_fas_coarse_cycle<<<1, kFasCoarseThreads, smem, st>>>(a);
    PB_LAUNCH_CHECK();
    T.cur = 0;
    return PB_OK;
}

// The finest level's first sweep has been done by the norm pass that measured its state.
static int fas_vcycle(pb_fas* m, int l, cudaStream_t st)
{
    const bool top = l == (int)m->lv.size() - 1;
    const int done = top ? 1 : 0;
    if (m->lv[l].n <= kFasCoarseEdge && l < kFasCoarseMax && !top) return fas_coarse(m, l, st);
    if (l == 0) return fas_relax(m, l, m->num_bottom - done, !top, st);
    FasLevel& L = m->lv[l];
    FasLevel& C = m->lv[l - 1];
    int e;
    if ((e = fas_relax(m, l, m->num_pre - done, !top, st)) != PB_OK) return e;
    C.cur = 0;
    e = C.n < 4 ? launch_lap4<true>(fas_geom(L), L.k, EpiFasRestrict<true>{L.f, L.n, C.u[0], C.c0, C.f, 0.0, 0.0}, cached_sm_count(), st)
                : launch_lap4<true>(fas_geom(L), L.k, EpiFasRestrict<false>{L.f, L.n, C.u[0], C.c0, C.f, 0.0, 0.0}, cached_sm_count(), st);
    if (e != PB_OK) return e;
    if ((e = fas_vcycle(m, l - 1, st)) != PB_OK) return e;
    const Walk w = walk_cube(L.n);
    if (L.n < 4) k_fas_correct<true><<<walk_grid(w, 1), kWalkThreads, 0, st>>>(L.u[L.cur], C.c0, C.u[C.cur], L.n, w);
    else k_fas_correct<false><<<walk_grid(w, 1), kWalkThreads, 0, st>>>(L.u[L.cur], C.c0, C.u[C.cur], L.n, w);
    PB_LAUNCH_CHECK();
    return fas_relax(m, l, m->num_post, false, st);
}

// max |op(u) + f| on the finest level into the pinned host word (stream ordered, no wait), fused with the
// next cycle's first sweep into the other buffer; T.cur stays on the state measured
static int fas_enqueue_resnorm(pb_fas* m, cudaStream_t st)
{
    FasLevel& T = m->lv.back();
    PB_CUDA(cudaMemsetAsync(m->d_res, 0, sizeof(double), st));
    double* out = T.u[1 - T.cur];
    const int sms = cached_sm_count();
    const int e = T.n < 4 ? launch_lap4<true>(fas_geom(T), T.k, EpiFasRelax<false, true, true>{out, T.f, T.n, T.neg_lambda, m->d_res}, sms, st)
                          : launch_lap4<true>(fas_geom(T), T.k, EpiFasRelax<false, false, true>{out, T.f, T.n, T.neg_lambda, m->d_res}, sms, st);
    if (e != PB_OK) return e;
    PB_CUDA(cudaMemcpyAsync(m->h_res, m->d_res, sizeof(double), cudaMemcpyDeviceToHost, st));
    return PB_OK;
}

static int fas_resnorm(pb_fas* m, cudaStream_t st, double* out)
{
    const int e = fas_enqueue_resnorm(m, st);
    if (e != PB_OK) return e;
    PB_CUDA(cudaStreamSynchronize(st));
    *out = *m->h_res;
    return PB_OK;
}

static int fas_cycle_and_norm(pb_fas* m, cudaStream_t st)
{
    m->lv.back().cur = 1 - m->lv.back().cur;   // on from the sweep that the last norm pass did
    const int e = fas_vcycle(m, (int)m->lv.size() - 1, st);
    return e != PB_OK ? e : fas_enqueue_resnorm(m, st);
}

static void fas_free(pb_fas* m)
{
    for (auto& L : m->lv) {
        cudaFree(L.u[0]);
        cudaFree(L.u[1]);
        cudaFree(L.f);
        cudaFree(L.c0);
    }
    cudaFree(m->d_res);
    cudaFreeHost(m->h_res);
    for (int p = 0; p < 2; p++)
        if (m->graph[p]) cudaGraphExecDestroy(m->graph[p]);
    if (m->graph_stream) cudaStreamDestroy(m->graph_stream);
    delete m;
}

extern "C" {

int pb_boxop_laplace_f64(const double* state, pb_box state_box, double* out, pb_box out_box, pb_box range, double dx,
                         double flux_scale, double scale, void* stream)
{
    if (!state || !out || !(dx > 0)) return PB_ERR_ARG;
    const Box3 sb = to_box(state_box), ob = to_box(out_box);
    Box3 rb = to_box(range);
    if (bempty(sb) || bempty(ob)) return PB_ERR_BOX;
    if (bempty(rb)) rb = ob;
    if (!contains_box(ob, rb)) return PB_ERR_BOX;
    Box3 need = rb;
    for (int d = 0; d < 3; d++) {
        need.lo[d] -= kFasGhost;      // the face fluxes reach two cells down and two up
        need.hi[d] += kFasGhost;
    }
    if (!contains_box(sb, need)) return PB_ERR_GHOST;
    const Region rg = region_of(rb);
    const FieldView<const double> uv = view_of(state, sb, rg);
    const FieldView<double> ov = view_of(out, ob, rg);
    const EpiBoxOp epi{ov.p, ov.sy, ov.sz, flux_scale, scale, scale != 1.0};
    if (boxop_march_share(rg) < kBoxOpMarch) {
        const Walk w = walk_of(rg, 1);
        k_boxop_cells<<<walk_grid(w, 1), kWalkThreads, 0, (cudaStream_t)stream>>>(uv, epi, fas_coefs(dx), w);
        PB_LAUNCH_CHECK();
        return PB_OK;
    }
    const Lap4Geom g{uv.p, uv.sy, uv.sz, rg.n[0], rg.n[1], rg.n[2], 0, 0};
    return launch_lap4<false>(g, fas_coefs(dx), epi, cached_sm_count(), (cudaStream_t)stream);
}

int pb_fas_create(int n, int num_levels, pb_fas** out)
{
    if (!out || n < 1 || num_levels < 1 || num_levels > 20) return PB_ERR_ARG;
    if ((n >> (num_levels - 1)) < 1 || ((n >> (num_levels - 1)) << (num_levels - 1)) != n) return PB_ERR_ARG;
    pb_fas* m = new (std::nothrow) pb_fas;
    if (!m) return PB_ERR_NOMEM;
    m->lv.resize(num_levels);
    bool ok = true;
    for (int l = 0; l < num_levels && ok; l++) {
        FasLevel& L = m->lv[l];
        L.n = n >> (num_levels - 1 - l);
        L.dx = (double)(1 << (num_levels - 1 - l)) / (double)n;
        L.k = fas_coefs(L.dx);
        // lambda = 0.5 / spectralRadius, spectralRadius = (2*DIM) / dx^2
        L.neg_lambda = -(0.5 / ((2.0 * 3) / std::pow(L.dx, 2)));
        const size_t c = sizeof(double) * (size_t)L.n * L.n * L.n;
        const size_t g = sizeof(double) * (size_t)(L.n + 2 * kFasGhost) * (L.n + 2 * kFasGhost) * L.n;
        ok = cudaMalloc(&L.u[0], g) == cudaSuccess && cudaMalloc(&L.u[1], g) == cudaSuccess &&
             cudaMalloc(&L.f, c) == cudaSuccess && cudaMalloc(&L.c0, c) == cudaSuccess &&
             cudaMemset(L.u[0], 0, g) == cudaSuccess && cudaMemset(L.u[1], 0, g) == cudaSuccess;
    }
    if (ok) ok = cudaMalloc(&m->d_res, sizeof(double)) == cudaSuccess && cudaMallocHost(&m->h_res, sizeof(double)) == cudaSuccess;
    if (!ok) {
        cudaGetLastError();
        fas_free(m);
        return PB_ERR_NOMEM;
    }
    *out = m;
    return PB_OK;
}

int pb_fas_destroy(pb_fas* m)
{
    if (m) fas_free(m);
    return PB_OK;
}

int pb_fas_solve(pb_fas* m, const double* force, double* phi, int max_iter, double tol, int* iters, double* hist,
                 void* stream)
{
    if (!m || !force || !phi || max_iter < 0) return PB_ERR_ARG;
    cudaStream_t st = (cudaStream_t)stream;
    FasLevel& T = m->lv.back();
    const long long n3 = (long long)T.n * T.n * T.n;
    T.cur = 0;
    PB_CUDA(cudaMemcpyAsync(T.f, force, sizeof(double) * n3, cudaMemcpyDeviceToDevice, st));
    const int S = T.n + 2 * kFasGhost;
    const Walk wg = walk_of(Region{{0, 0, 0}, {S, S, T.n}}), wv = walk_cube(T.n);
    k_fas_pack<<<walk_grid(wg, 1), kWalkThreads, 0, st>>>(phi, T.u[0], T.n, wg);
    PB_LAUNCH_CHECK();
    double r0, r;
    int e;
    if ((e = fas_resnorm(m, st, &r0)) != PB_OK) return e;
    if (hist) hist[0] = r0;
    int it = 0;
    while (it < max_iter) {
        const int par = T.cur;
        if (!m->graph[par]) {
            if (!m->graph_stream) PB_CUDA(cudaStreamCreateWithFlags(&m->graph_stream, cudaStreamNonBlocking));
            cudaGraph_t g;
            PB_CUDA(cudaStreamBeginCapture(m->graph_stream, cudaStreamCaptureModeThreadLocal));
            e = fas_cycle_and_norm(m, m->graph_stream);
            cudaError_t ce = cudaStreamEndCapture(m->graph_stream, &g);
            if (e != PB_OK) {
                if (ce == cudaSuccess) cudaGraphDestroy(g);
                return e;
            }
            if (ce != cudaSuccess) { set_cuda_error(ce); return PB_ERR_CUDA; }
            ce = cudaGraphInstantiate(&m->graph[par], g, 0);
            cudaGraphDestroy(g);
            if (ce != cudaSuccess) { m->graph[par] = nullptr; set_cuda_error(ce); return PB_ERR_CUDA; }
            m->graph_cur[par] = T.cur;   // capture recorded the buffer flips without running them
            T.cur = par;
        }
        PB_CUDA(cudaGraphLaunch(m->graph[par], st));
        T.cur = m->graph_cur[par];
        PB_CUDA(cudaStreamSynchronize(st));
        r = *m->h_res;
        ++it;
        if (hist) hist[it] = r;
        if (r < tol * r0) break;
    }
    k_fas_unpack<<<walk_grid(wv, 1), kWalkThreads, 0, st>>>(T.u[T.cur], phi, T.n, wv);
    PB_LAUNCH_CHECK();
    PB_CUDA(cudaStreamSynchronize(st));
    if (iters) *iters = it;
    return PB_OK;
}

} // extern "C"
