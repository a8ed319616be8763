// BoxData algebra, copyTo, pointwise (forall) kernels, reductions and constant prolongation.
//
// Reference counterparts (paths within the reference project):
//   BoxData::operatorT / scalar ops ... include/base/implem/Proto_BoxDataImplem.H:860-985, 1086-1110
//   BoxData::copyTo (general) ......... include/base/implem/Proto_BoxDataImplem.H:493-640
//   forall / forallInPlace ............ include/base/implem/Proto_ForallImplem.H:178-389
//   Reduction<T,OP,DEVICE> ............ include/base/Proto_Reduction.H:113-185,
//                                       include/base/implem/Proto_ReductionImplem.H:108-192
//   InterpStencil::Constant ........... include/base/implem/Proto_InterpStencilDefs.H:1-15
// The reference launches one kernel per call with blocks of one x-row each; these kernels walk rows
// with several planes' loads in flight.
#include <cfloat>
#include <cstring>
#include <mutex>
#include <new>

#include "pb_internal.cuh"
#include "pb_stencil_impl.cuh"
#include "pb_walk.cuh"

namespace pb {

template <int OP>
__device__ __forceinline__ double apply_op(double d, double s)
{
    if (OP == PB_OP_ADD) return dadd(d, s);
    if (OP == PB_OP_SUB) return dsub(d, s);
    if (OP == PB_OP_MUL) return dmul(d, s);
    if (OP == PB_OP_DIV) return ddiv(d, s);
    return s;
}

// ---- dst op= src on a region (both fields addressed through their own boxes) -----------------
template <int OP>
__global__ void __launch_bounds__(kWalkThreads) k_binop(FieldView<double> d, long long dvol, FieldView<const double> s,
                                                        long long svol, Walk w, int ncomp)
{
    for (int c = blockIdx.z; c < ncomp; c += gridDim.z) {
        double* dp = d.p + c * dvol;
        const double* sp = s.p + c * svol;
        walk_rows(w, [&](int x, int y, int z, int planes) {
            double* dq = dp + x + d.sy * y + d.sz * z;
            const double* sq = sp + x + s.sy * y + s.sz * z;
            double sv[kWalkZ], dv[kWalkZ];
#pragma unroll
            for (int k = 0; k < kWalkZ; k++)
                if (k < planes) {
                    sv[k] = sq[k * s.sz];
                    if (OP != PB_OP_ASSIGN) dv[k] = dq[k * d.sz];
                }
#pragma unroll
            for (int k = 0; k < kWalkZ; k++)
                if (k < planes) dq[k * d.sz] = apply_op<OP>(OP != PB_OP_ASSIGN ? dv[k] : 0.0, sv[k]);
        });
    }
}

template <int OP>
__global__ void __launch_bounds__(kWalkThreads) k_scalar(FieldView<double> d, long long dvol, Walk w, double v, int ncomp)
{
    for (int c = blockIdx.z; c < ncomp; c += gridDim.z) {
        double* dp = d.p + c * dvol;
        walk_rows(w, [&](int x, int y, int z, int planes) {
            double* dq = dp + x + d.sy * y + d.sz * z;
            double dv[kWalkZ];
#pragma unroll
            for (int k = 0; k < kWalkZ; k++)
                if (OP != PB_OP_ASSIGN && k < planes) dv[k] = dq[k * d.sz];
#pragma unroll
            for (int k = 0; k < kWalkZ; k++)
                if (k < planes) dq[k * d.sz] = apply_op<OP>(OP != PB_OP_ASSIGN ? dv[k] : 0.0, v);
        });
    }
}

// forall body "out = a*x + b*y" (config: out = a*L(u) + b*u when Lu is materialised)
__global__ void __launch_bounds__(kWalkThreads) k_axpby(FieldView<double> o, FieldView<const double> xs,
                                                        FieldView<const double> ys, Walk w, double a, double b)
{
    walk_rows(w, [&](int x, int y, int z, int planes) {
        double* oq = o.p + x + o.sy * y + o.sz * z;
        const double* xq = xs.p + x + xs.sy * y + xs.sz * z;
        const double* yq = ys.p + x + ys.sy * y + ys.sz * z;
        double xv[kWalkZ], yv[kWalkZ];
#pragma unroll
        for (int k = 0; k < kWalkZ; k++)
            if (k < planes) {
                xv[k] = xq[k * xs.sz];
                yv[k] = yq[k * ys.sz];
            }
#pragma unroll
        for (int k = 0; k < kWalkZ; k++)
            if (k < planes) oq[k * o.sz] = dadd(dmul(a, xv[k]), dmul(b, yv[k]));
    });
}

// ---- reductions ---------------------------------------------------------------------------------
// Pass 1: every block folds its share; pass 2 (the last block to finish, found through an atomic
// ticket) folds the per-block partials in block order, so sums are deterministic. A share is a fixed
// set of tiles (a block's rows x kRedZ planes), walked like the pointwise kernels: each thread keeps kRedZ
// loads in flight, one accumulator per plane of the tile. (Sharing a row between blocks, as those kernels
// do, was slower: 11.0 -> 13.5 us at 160^3; the last block has more partial results to fold.)
constexpr int kRedBlocks = 1024;
constexpr int kRedThreads = 256;
constexpr int kRedZ = 8;

__device__ __forceinline__ double red_init(int op)
{
    return op == 0 ? DBL_MIN : op == 1 ? DBL_MAX : 0.0;
}
__device__ __forceinline__ double red_upd(int op, double v1, double v2)
{
    switch (op) {
        case 0: return (v1 < v2) ? v2 : v1;                 // std::max
        case 1: return (v2 < v1) ? v2 : v1;                 // std::min
        case 2: return upd_abs(v1, v2);
        case 3: return dadd(v1, v2);
        case 4: return dadd(v1, v2 > 0 ? v2 : -v2);
        default: return dadd(v1, dmul(v2, v2));
    }
}
// combining two partial results (for Abs/SumAbs/SumSquare the partials are already folded)
__device__ __forceinline__ double red_comb(int op, double a, double b)
{
    switch (op) {
        case 0: return (a < b) ? b : a;
        case 1: return (b < a) ? b : a;
        case 2: return (a < b) ? b : a;
        default: return dadd(a, b);
    }
}

__device__ double block_reduce(int op, double v)
{
    __shared__ double sh[32];
    int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    for (int o = 16; o > 0; o >>= 1) v = red_comb(op, v, __shfl_down_sync(0xffffffffu, v, o));
    if (lane == 0) sh[wid] = v;
    __syncthreads();
    v = (threadIdx.x < (blockDim.x >> 5)) ? sh[lane] : red_init(op == 2 ? 2 : op);
    if (wid == 0)
        for (int o = 16; o > 0; o >>= 1) v = red_comb(op, v, __shfl_down_sync(0xffffffffu, v, o));
    __syncthreads();
    return v;
}

// OP is a template argument so that the fold is one instruction or two, not a switch per cell.
template <int op>
__global__ void __launch_bounds__(kRedThreads) k_reduce(FieldView<const double> f, Walk w, double* partials,
                                                        unsigned int* ticket, double* result)
{
    double acc[kRedZ];
#pragma unroll
    for (int k = 0; k < kRedZ; k++) acc[k] = red_init(op);
    const int rows = kRedThreads >> w.lx;
    const int lane = threadIdx.x & ((1 << w.lx) - 1), row = threadIdx.x >> w.lx;
    const int ty = (w.ny + rows - 1) / rows, tz = (w.nz + kRedZ - 1) / kRedZ;
    const long long tiles = (long long)ty * tz;
    for (long long t = blockIdx.x; t < tiles; t += gridDim.x) {
        const int y = (int)(t % ty) * rows + row, z = (int)(t / ty) * kRedZ;
        if (y >= w.ny) continue;
        const double* q = f.p + f.sy * y + f.sz * z;
        const int planes = min(kRedZ, w.nz - z);
        for (int x = lane; x < w.nx; x += 1 << w.lx) {
            double v[kRedZ];
#pragma unroll
            for (int k = 0; k < kRedZ; k++)
                if (k < planes) v[k] = __ldg(q + x + k * f.sz);
#pragma unroll
            for (int k = 0; k < kRedZ; k++)
                if (k < planes) acc[k] = red_upd(op, acc[k], v[k]);
        }
    }
    double v = acc[0];
#pragma unroll
    for (int k = 1; k < kRedZ; k++) v = red_comb(op, v, acc[k]);
    v = block_reduce(op, v);
    __shared__ bool last;
    if (threadIdx.x == 0) {
        partials[blockIdx.x] = v;
        __threadfence();
        unsigned int t = atomicAdd(ticket, 1u);
        last = (t == gridDim.x - 1);
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    double folded = red_init(op);
    // fixed order over the partials: thread k folds partials k, k+256, ... then the block tree
    for (int k = threadIdx.x; k < gridDim.x; k += blockDim.x) {
        double p = ((volatile double*)partials)[k];
        folded = (k == threadIdx.x) ? p : red_comb(op, folded, p);
    }
    if (threadIdx.x >= gridDim.x) folded = red_init(op);
    folded = block_reduce(op, folded);
    if (threadIdx.x == 0) {
        *result = folded;
        *ticket = 0;
    }
}

// ---- piecewise-constant prolongation ----------------------------------------------------------
// Fine cell p takes coarse cell floor(p / ratio). LR is log2(ratio) where that is a power of two (an
// arithmetic shift floors like floor_div); -1 divides. Walked like the pointwise kernels; the four
// planes' coarse and fine loads go out together. Measured (B200): AvgDown from 192^3, a copy of a 192^3
// field and the prolongation added to it, 107 -> 67 us together with pb_stencil.cu's table kernel.
template <int LR>
__device__ __forceinline__ int coarse_of(int p, int ratio) { return LR >= 0 ? p >> (LR < 0 ? 0 : LR) : floor_div(p, ratio); }

template <int LR>
__global__ void __launch_bounds__(kWalkThreads) k_interp_const(int ratio, const double* __restrict__ src, Box3 sb,
                                                               FieldView<double> d, Region r, Walk w, int overwrite,
                                                               double scale)
{
    const long long Sx = bsize(sb, 0), Sxy = Sx * bsize(sb, 1);
    walk_rows(w, [&](int x, int y, int z, int planes) {
        const double* sq = src + (coarse_of<LR>(r.lo[0] + x, ratio) - sb.lo[0]) + Sx * (coarse_of<LR>(r.lo[1] + y, ratio) - sb.lo[1]);
        double* dq = d.p + x + d.sy * y + d.sz * z;
        double v[kWalkZ], acc[kWalkZ];
#pragma unroll
        for (int k = 0; k < kWalkZ; k++)
            if (k < planes) {
                v[k] = __ldg(sq + Sxy * (coarse_of<LR>(r.lo[2] + z + k, ratio) - sb.lo[2]));
                acc[k] = overwrite ? 0.0 : dq[k * d.sz];
            }
#pragma unroll
        for (int k = 0; k < kWalkZ; k++)
            if (k < planes) dq[k * d.sz] = dadd(acc[k], dmul(scale, v[k]));
    });
}

// ---- reduction scratch ------------------------------------------------------------------------
// A slot is what one reduction needs while it is in flight: partial results, a ticket and, for calls
// that wait, a page-locked result word (written by the kernel: no copy to fetch it). Calls come from
// several threads and on several streams, so no two reductions in flight share a slot:
//   * a call that waits takes an idle slot and gives it back after its synchronise;
//   * an asynchronous call uses its stream's slot, and its kernel waits (on the device) for the event that
//     the slot's last kernel recorded: nothing to wait for on the same stream, and right when a stream's
//     handle comes back or streams beyond kRedStreams take over a slot;
//   * a captured call's slot belongs to the graph, which may run at any time beside other reductions,
//     and becomes idle when the graph and its executables are gone.
struct RedSlot {
    double* partials = nullptr;    // kRedBlocks
    unsigned int* ticket = nullptr;
    double* result = nullptr;      // allocated when a call that waits first takes the slot
    cudaEvent_t done = nullptr;    // after the last kernel (slots of streams)
    RedSlot* next = nullptr;       // idle list
    int device = 0;
};
constexpr int kRedDevices = 16, kRedStreams = 32, kRedIdleMax = 64;
struct RedPool {
    std::mutex mutex;
    RedSlot* idle = nullptr;
    int nidle = 0;
    cudaStream_t stream[kRedStreams];
    RedSlot* of_stream[kRedStreams] = {};
    unsigned evict = 0;
};
// not destroyed: a graph may give its slot back while the process exits
static RedPool* red_pools()
{
    static RedPool* p = new (std::nothrow) RedPool[kRedDevices];
    return p;
}

// Allocating and freeing are forbidden while this thread (or, in the global mode, any thread) captures,
// unless the thread says that it is not part of the capture.
struct RelaxedCapture {
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
    ~RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
};

static void red_free(RedSlot* s)
{
    if (!s) return;
    RelaxedCapture relaxed;
    cudaFree(s->partials);
    if (s->result) cudaFreeHost(s->result);
    if (s->done) cudaEventDestroy(s->done);
    delete s;
}

static cudaError_t red_alloc(RedSlot* s)
{
    RelaxedCapture relaxed;
    cudaStream_t st;
    const size_t bytes = kRedBlocks * sizeof(double) + 256;
    cudaError_t e = cudaMalloc(&s->partials, bytes);
    if (e != cudaSuccess) return e;
    s->ticket = reinterpret_cast<unsigned int*>(s->partials + kRedBlocks);
    // cleared on a stream of its own: the caller's may be capturing
    if ((e = cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking)) != cudaSuccess) return e;
    e = cudaMemsetAsync(s->partials, 0, bytes, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    cudaStreamDestroy(st);
    return e;
}

static int red_new(int dev, RedSlot** out)
{
    RedSlot* s = new (std::nothrow) RedSlot;
    if (!s) return PB_ERR_NOMEM;
    s->device = dev;
    const cudaError_t e = red_alloc(s);
    if (e != cudaSuccess) {
        red_free(s);
        set_cuda_error(e);
        return PB_ERR_CUDA;
    }
    *out = s;
    return PB_OK;
}

static int red_pool(int* dev, RedPool** out)
{
    PB_CUDA(cudaGetDevice(dev));
    if (*dev < 0 || *dev >= kRedDevices) return PB_ERR_UNSUPPORTED;
    RedPool* p = red_pools();
    if (!p) return PB_ERR_NOMEM;
    *out = p + *dev;
    return PB_OK;
}

// an idle slot of the current device, or a new one
static int red_take(RedSlot** out)
{
    int dev;
    RedPool* p;
    const int e = red_pool(&dev, &p);
    if (e != PB_OK) return e;
    {
        std::lock_guard<std::mutex> lock(p->mutex);
        if (p->idle) {
            *out = p->idle;
            p->idle = p->idle->next;
            p->nidle--;
            return PB_OK;
        }
    }
    return red_new(dev, out);
}

static void red_idle(RedSlot* s)
{
    RedPool* p = red_pools() + s->device;
    std::lock_guard<std::mutex> lock(p->mutex);
    s->next = p->idle;
    p->idle = s;
    p->nidle++;
}

// back from a call that waited; idle slots above the limit are freed here (a graph's destructor may not)
static void red_give(RedSlot* s)
{
    red_idle(s);
    RedPool* p = red_pools() + s->device;
    RedSlot* extra = nullptr;
    {
        std::lock_guard<std::mutex> lock(p->mutex);
        if (p->nidle > kRedIdleMax) {
            extra = p->idle;
            p->idle = extra->next;
            p->nidle--;
        }
    }
    red_free(extra);
}
static void CUDART_CB red_graph_gone(void* s) { red_idle(static_cast<RedSlot*>(s)); }

// The fold itself, with the scratch of slot s.
static int launch_reduce(int op, const double* data, const Box3& b, const Box3& r, RedSlot* s, double* result, cudaStream_t st)
{
    Region rg;                           // an empty intersection folds nothing: the operation's initial value
    if (bempty(r)) { rg.lo[0] = b.lo[0]; rg.lo[1] = b.lo[1]; rg.lo[2] = b.lo[2]; rg.n[0] = rg.n[1] = rg.n[2] = 0; }
    else rg = region_of(r);
    const Walk w = walk_of(rg);
    const int rows = kRedThreads >> w.lx;
    const long long tiles = (long long)((w.ny + rows - 1) / rows) * ((w.nz + kRedZ - 1) / kRedZ);
    int grid = tiles < kRedBlocks ? (int)tiles : kRedBlocks;
    if (grid < 1) grid = 1;
    const FieldView<const double> f = view_of(data, b, rg);
    switch (op) {
        case 0: k_reduce<0><<<grid, kRedThreads, 0, st>>>(f, w, s->partials, s->ticket, result); break;
        case 1: k_reduce<1><<<grid, kRedThreads, 0, st>>>(f, w, s->partials, s->ticket, result); break;
        case 2: k_reduce<2><<<grid, kRedThreads, 0, st>>>(f, w, s->partials, s->ticket, result); break;
        case 3: k_reduce<3><<<grid, kRedThreads, 0, st>>>(f, w, s->partials, s->ticket, result); break;
        case 4: k_reduce<4><<<grid, kRedThreads, 0, st>>>(f, w, s->partials, s->ticket, result); break;
        default: k_reduce<5><<<grid, kRedThreads, 0, st>>>(f, w, s->partials, s->ticket, result); break;
    }
    PB_LAUNCH_CHECK();
    return PB_OK;
}

// on the capturing stream: the graph keeps the slot
static int reduce_captured(int op, const double* data, const Box3& b, const Box3& r, double* result, cudaGraph_t graph,
                           cudaStream_t st)
{
    RedSlot* s;
    int e = red_take(&s);
    if (e != PB_OK) return e;
    cudaUserObject_t keep;
    cudaError_t ce = cudaUserObjectCreate(&keep, s, red_graph_gone, 1, cudaUserObjectNoDestructorSync);
    if (ce != cudaSuccess) {
        red_idle(s);
        set_cuda_error(ce);
        return PB_ERR_CUDA;
    }
    ce = cudaGraphRetainUserObject(graph, keep, 1, cudaGraphUserObjectMove);
    if (ce != cudaSuccess) {
        cudaUserObjectRelease(keep, 1);      // gives the slot back
        set_cuda_error(ce);
        return PB_ERR_CUDA;
    }
    return launch_reduce(op, data, b, r, s, result, st);
}

static int reduce_on_stream(int op, const double* data, const Box3& b, const Box3& r, double* result, cudaStream_t st)
{
    int dev;
    RedPool* p;
    int e = red_pool(&dev, &p);
    if (e != PB_OK) return e;
    std::lock_guard<std::mutex> lock(p->mutex);
    int k = 0;
    while (k < kRedStreams && p->of_stream[k] && p->stream[k] != st) k++;
    if (k == kRedStreams) k = p->evict++ % kRedStreams;
    RedSlot*& s = p->of_stream[k];
    p->stream[k] = st;
    if (!s) {
        RedSlot* fresh;
        if ((e = red_new(dev, &fresh)) != PB_OK) return e;
        const cudaError_t ce = cudaEventCreateWithFlags(&fresh->done, cudaEventDisableTiming);
        if (ce != cudaSuccess) {
            red_free(fresh);
            set_cuda_error(ce);
            return PB_ERR_CUDA;
        }
        s = fresh;
    }
    PB_CUDA(cudaStreamWaitEvent(st, s->done, 0));
    if ((e = launch_reduce(op, data, b, r, s, result, st)) != PB_OK) return e;
    PB_CUDA(cudaEventRecord(s->done, st));
    return PB_OK;
}

} // namespace pb

using namespace pb;

extern "C" {

int pb_boxdata_op_f64(int op, double* dst, pb_box dst_box, const double* src, pb_box src_box, int ncomp, void* stream)
{
    if (!dst || !src || ncomp < 1 || op < 0 || op > PB_OP_ASSIGN) return PB_ERR_ARG;
    Box3 db = to_box(dst_box), sb = to_box(src_box);
    Box3 r = intersect(db, sb);
    if (bempty(r)) return PB_OK;
    const Region rg = region_of(r);
    const Walk w = walk_of(rg);
    const dim3 grid = walk_grid(w, ncomp);
    const FieldView<double> d = view_of(dst, db, rg);
    const FieldView<const double> sv = view_of(src, sb, rg);
    cudaStream_t st = (cudaStream_t)stream;
    switch (op) {
        case PB_OP_ADD: k_binop<PB_OP_ADD><<<grid, kWalkThreads, 0, st>>>(d, bvol(db), sv, bvol(sb), w, ncomp); break;
        case PB_OP_SUB: k_binop<PB_OP_SUB><<<grid, kWalkThreads, 0, st>>>(d, bvol(db), sv, bvol(sb), w, ncomp); break;
        case PB_OP_MUL: k_binop<PB_OP_MUL><<<grid, kWalkThreads, 0, st>>>(d, bvol(db), sv, bvol(sb), w, ncomp); break;
        case PB_OP_DIV: k_binop<PB_OP_DIV><<<grid, kWalkThreads, 0, st>>>(d, bvol(db), sv, bvol(sb), w, ncomp); break;
        default: k_binop<PB_OP_ASSIGN><<<grid, kWalkThreads, 0, st>>>(d, bvol(db), sv, bvol(sb), w, ncomp); break;
    }
    PB_LAUNCH_CHECK();
    return PB_OK;
}

int pb_boxdata_scalar_f64(int op, double* dst, pb_box dst_box, pb_box region, double scalar, int ncomp, void* stream)
{
    if (!dst || ncomp < 1 || op < 0 || op > PB_OP_ASSIGN) return PB_ERR_ARG;
    Box3 db = to_box(dst_box), r = to_box(region);
    if (bempty(db)) return PB_ERR_BOX;
    r = bempty(r) ? db : intersect(r, db);
    if (bempty(r)) return PB_OK;
    const Region rg = region_of(r);
    const Walk w = walk_of(rg);
    const dim3 grid = walk_grid(w, ncomp);
    const FieldView<double> d = view_of(dst, db, rg);
    cudaStream_t st = (cudaStream_t)stream;
    switch (op) {
        case PB_OP_ADD: k_scalar<PB_OP_ADD><<<grid, kWalkThreads, 0, st>>>(d, bvol(db), w, scalar, ncomp); break;
        case PB_OP_SUB: k_scalar<PB_OP_SUB><<<grid, kWalkThreads, 0, st>>>(d, bvol(db), w, scalar, ncomp); break;
        case PB_OP_MUL: k_scalar<PB_OP_MUL><<<grid, kWalkThreads, 0, st>>>(d, bvol(db), w, scalar, ncomp); break;
        case PB_OP_DIV: k_scalar<PB_OP_DIV><<<grid, kWalkThreads, 0, st>>>(d, bvol(db), w, scalar, ncomp); break;
        default: k_scalar<PB_OP_ASSIGN><<<grid, kWalkThreads, 0, st>>>(d, bvol(db), w, scalar, ncomp); break;
    }
    PB_LAUNCH_CHECK();
    return PB_OK;
}

int pb_boxdata_copy_f64(const double* src, pb_box src_box, double* dst, pb_box dst_box, pb_box src_region,
                        const int shift[3], int ncomp, void* stream)
{
    if (!dst || !src || ncomp < 1) return PB_ERR_ARG;
    Box3 sb = to_box(src_box), db = to_box(dst_box), r = to_box(src_region);
    int sh[3] = {shift ? shift[0] : 0, shift ? shift[1] : 0, shift ? shift[2] : 0};
    r = bempty(r) ? sb : intersect(r, sb);
    Box3 dshift;
    for (int d = 0; d < 3; d++) { dshift.lo[d] = db.lo[d] - sh[d]; dshift.hi[d] = db.hi[d] - sh[d]; }
    r = intersect(r, dshift);
    if (bempty(r)) return PB_OK;
    const Region rg = region_of(r);      // source points; their destinations are shifted
    const Walk w = walk_of(rg);
    k_binop<PB_OP_ASSIGN><<<walk_grid(w, ncomp), kWalkThreads, 0, (cudaStream_t)stream>>>(
        view_of(dst, db, rg, sh), bvol(db), view_of(src, sb, rg), bvol(sb), w, ncomp);
    PB_LAUNCH_CHECK();
    return PB_OK;
}

int pb_forall_axpby_f64(double* out, pb_box out_box, const double* x, pb_box x_box, const double* y, pb_box y_box,
                        double a, double b, void* stream)
{
    if (!out || !x || !y) return PB_ERR_ARG;
    Box3 ob = to_box(out_box), xb = to_box(x_box), yb = to_box(y_box);
    Box3 r = intersect(intersect(ob, xb), yb);
    if (bempty(r)) return PB_OK;
    const Region rg = region_of(r);
    const Walk w = walk_of(rg);
    k_axpby<<<walk_grid(w, 1), kWalkThreads, 0, (cudaStream_t)stream>>>(view_of(out, ob, rg), view_of(x, xb, rg),
                                                                        view_of(y, yb, rg), w, a, b);
    PB_LAUNCH_CHECK();
    return PB_OK;
}

int pb_reduce_async_f64(int op, const double* data, pb_box box, pb_box region, double* result_dev, void* stream)
{
    if (!data || !result_dev || op < 0 || op > 5) return PB_ERR_ARG;
    Box3 b = to_box(box), r = to_box(region);
    if (bempty(b)) return PB_ERR_BOX;
    r = bempty(r) ? b : intersect(r, b);
    cudaStream_t st = (cudaStream_t)stream;
    cudaStreamCaptureStatus cs;
    cudaGraph_t graph = nullptr;
    PB_CUDA(cudaStreamGetCaptureInfo_v2(st, &cs, nullptr, &graph, nullptr, nullptr));
    return cs == cudaStreamCaptureStatusActive ? reduce_captured(op, data, b, r, result_dev, graph, st)
                                               : reduce_on_stream(op, data, b, r, result_dev, st);
}

int pb_reduce_f64(int op, const double* data, pb_box box, pb_box region, double* result, void* stream)
{
    if (!data || !result || op < 0 || op > 5) return PB_ERR_ARG;
    Box3 b = to_box(box), r = to_box(region);
    if (bempty(b)) return PB_ERR_BOX;
    r = bempty(r) ? b : intersect(r, b);
    RedSlot* s;
    int e = red_take(&s);
    if (e != PB_OK) return e;
    if (!s->result) {
        RelaxedCapture relaxed;
        const cudaError_t ce = cudaHostAlloc(&s->result, sizeof(double), cudaHostAllocMapped | cudaHostAllocPortable);
        if (ce != cudaSuccess) {
            s->result = nullptr;
            red_idle(s);
            set_cuda_error(ce);
            return PB_ERR_CUDA;
        }
    }
    e = launch_reduce(op, data, b, r, s, s->result, (cudaStream_t)stream);
    if (e == PB_OK) {
        const cudaError_t ce = cudaStreamSynchronize((cudaStream_t)stream);
        if (ce != cudaSuccess) {       // the kernel may still run (or was captured): the slot is not given back
            set_cuda_error(ce);
            return PB_ERR_CUDA;
        }
        *result = *(volatile double*)s->result;
    }
    red_give(s);
    return e;
}

int pb_interp_constant_f64(int ratio, const double* src, pb_box src_box, double* dst, pb_box dst_box, int overwrite,
                           double scale, void* stream)
{
    if (!src || !dst || ratio < 1) return PB_ERR_ARG;
    Box3 sb = to_box(src_box), db = to_box(dst_box);
    if (bempty(sb) || bempty(db)) return PB_ERR_BOX;
    Box3 rb;
    for (int d = 0; d < 3; d++) { rb.lo[d] = sb.lo[d] * ratio; rb.hi[d] = sb.hi[d] * ratio + ratio - 1; }
    rb = intersect(rb, db);
    if (bempty(rb)) return PB_OK;
    // InterpStencil::apply's final stage is "S = scale*Shift::Zeros()", folded like hostApply
    const Region rg = region_of(rb);
    const Walk w = walk_of(rg);
    const dim3 grid = walk_grid(w, 1);
    const FieldView<double> d = view_of(dst, db, rg);
    cudaStream_t st = (cudaStream_t)stream;
    if (ratio == 2) k_interp_const<1><<<grid, kWalkThreads, 0, st>>>(ratio, src, sb, d, rg, w, overwrite, scale);
    else if (ratio == 4) k_interp_const<2><<<grid, kWalkThreads, 0, st>>>(ratio, src, sb, d, rg, w, overwrite, scale);
    else k_interp_const<-1><<<grid, kWalkThreads, 0, st>>>(ratio, src, sb, d, rg, w, overwrite, scale);
    PB_LAUNCH_CHECK();
    return PB_OK;
}

} // extern "C"
