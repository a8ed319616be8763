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
#include <type_traits>
#include <utility>

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
        walk_items(w, [&](int x, int y, int z, int planes) {
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
        walk_items(w, [&](int x, int y, int z, int planes) {
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
    walk_items(w, [&](int x, int y, int z, int planes) {
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
// ticket) folds the per-block partials in block order, so sums are deterministic. A share is a run of
// consecutive items of kRedZ planes (pb_walk.cuh): a thread has the loads of two items in flight and one
// accumulator per plane. Two blocks per SM: more partial results cost the last block more than the extra
// warps give (160^3: 592 blocks 8.5 us, 296 7.8). The number is fixed, so a result does not depend on the GPU.
// Boxes thin in z fold along y, and lines take kRedZ single cells a thread. Measured (B200, us): square
// sum of 160^3 7.9, 256^3 33; maximum norm of a line of 2^20 cells 6.2, of 2048 x 2048 x 1 8.2, each the
// same along any axis.
constexpr int kRedBlocks = 296;
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
        case 4: return dadd(v1, fabs(v2));
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

// OP is a template argument so that the fold is one instruction or two, not a switch per cell. chunk: items
// of a block. LINE: items are single cells.
template <int op, bool LINE>
__global__ void __launch_bounds__(kRedThreads) k_reduce(FieldView<const double> f, Walk w, long long chunk, double* partials,
                                                        unsigned int* ticket, double* result)
{
    double acc[kRedZ];
#pragma unroll
    for (int k = 0; k < kRedZ; k++) acc[k] = red_init(op);
    auto fold = [&](auto first, auto step, auto end) {       // 32- or 64-bit item numbers
        if constexpr (LINE) {
            for (auto i = first; i < end; i += kRedZ * step) {
                double v[kRedZ];
#pragma unroll
                for (int k = 0; k < kRedZ; k++) {
                    const auto j = i + k * step;
                    int x, y, z;
                    if (j < end) {
                        walk_item(w, j, x, y, z);
                        v[k] = __ldg(f.p + x + f.sy * y + f.sz * z);
                    }
                }
#pragma unroll
                for (int k = 0; k < kRedZ; k++)
                    if (i + k * step < end) acc[k] = red_upd(op, acc[k], v[k]);
            }
        } else {
#pragma unroll 2
            for (auto i = first; i < end; i += step) {
                int x, y, g;
                walk_item(w, i, x, y, g);
                const double* q = f.p + x + f.sy * y + f.sz * (g * kRedZ);
                const int planes = min(kRedZ, w.nz - g * kRedZ);
                double v[kRedZ];
#pragma unroll
                for (int k = 0; k < kRedZ; k++)
                    if (k < planes) v[k] = __ldg(q + k * f.sz);
#pragma unroll
                for (int k = 0; k < kRedZ; k++)
                    if (k < planes) acc[k] = red_upd(op, acc[k], v[k]);
            }
        }
    };
    // the largest item number of a thread's last round stays below 2^31 in the narrow form
    const long long begin = blockIdx.x * chunk, end = begin + chunk < w.items ? begin + chunk : w.items;
    if (w.items < (1LL << 30)) fold((unsigned)begin + threadIdx.x, (unsigned)kRedThreads, (unsigned)end);
    else fold(begin + threadIdx.x, (long long)kRedThreads, end);
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
// Fine cell p takes coarse cell floor(p / ratio); a shift where the ratio is a power of two. The planes'
// coarse and fine loads go out together. Measured (B200, us): 160^3, ratio 2 8.5, ratio 3 9.6.
struct CoarseMap {
    FastDiv ratio;
    int shift;
    int off[3], first[3];    // region coordinate p lies in source cell (p + off) / ratio + first
};

template <bool POW2>
__global__ void __launch_bounds__(kWalkThreads) k_interp_const(FieldView<const double> s, CoarseMap m, FieldView<double> d, Walk w, int overwrite,
                                                               double scale)
{
    walk_items(w, [&](int x, int y, int z, int planes) {
        auto coarse = [&](int p, int a) {
            const unsigned q = (unsigned)p + (unsigned)m.off[a];
            return (int)(POW2 ? q >> m.shift : quotient(q, m.ratio)) + m.first[a];
        };
        const double* sq = s.p + coarse(x, 0) + s.sy * coarse(y, 1);
        double* dq = d.p + x + d.sy * y + d.sz * z;
        double v[kWalkZ], acc[kWalkZ];
#pragma unroll
        for (int k = 0; k < kWalkZ; k++)
            if (k < planes) {
                v[k] = __ldg(sq + s.sz * coarse(z + k, 2));
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
    double* partials = nullptr;    // kRedBlocks, then the ticket
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
    FieldView<const double> f = view_of(data, b, rg);
    if (rg.n[2] < kRedZ && rg.n[1] > rg.n[2]) {      // thin in z: the loads in flight go along y
        std::swap(rg.n[1], rg.n[2]);
        std::swap(f.sy, f.sz);
    }
    const bool line = rg.n[2] < kRedZ;               // thin in y as well: a thread takes kRedZ single cells
    const Walk w = walk_of(rg, line ? 1 : kRedZ);
    const long long blocks = (w.items + kRedThreads - 1) / kRedThreads;
    const long long chunk = (blocks + kRedBlocks - 1) / kRedBlocks * kRedThreads;      // items of a block
    const int grid = blocks < 1 ? 1 : (int)((w.items + chunk - 1) / chunk);
    auto launch = [&](auto opc) {
        constexpr int OP = decltype(opc)::value;
        if (line) k_reduce<OP, true><<<grid, kRedThreads, 0, st>>>(f, w, chunk, s->partials, s->ticket, result);
        else k_reduce<OP, false><<<grid, kRedThreads, 0, st>>>(f, w, chunk, s->partials, s->ticket, result);
    };
    switch (op) {
        case 0: launch(std::integral_constant<int, 0>{}); break;
        case 1: launch(std::integral_constant<int, 1>{}); break;
        case 2: launch(std::integral_constant<int, 2>{}); break;
        case 3: launch(std::integral_constant<int, 3>{}); break;
        case 4: launch(std::integral_constant<int, 4>{}); break;
        default: launch(std::integral_constant<int, 5>{}); break;
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
    Region rg = region_of(r);
    FieldView<double> d = view_of(dst, db, rg);
    FieldView<const double> sv = view_of(src, sb, rg);
    turn_thin(rg, d, sv);
    const Walk w = walk_spread(rg);
    const dim3 grid = walk_grid(w, ncomp);
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
    Region rg = region_of(r);
    FieldView<double> d = view_of(dst, db, rg);
    turn_thin(rg, d);
    const Walk w = walk_spread(rg);
    const dim3 grid = walk_grid(w, ncomp);
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
    Region rg = region_of(r);            // source points; their destinations are shifted
    FieldView<double> d = view_of(dst, db, rg, sh);
    FieldView<const double> sv = view_of(src, sb, rg);
    turn_thin(rg, d, sv);
    const Walk w = walk_spread(rg);
    k_binop<PB_OP_ASSIGN><<<walk_grid(w, ncomp), kWalkThreads, 0, (cudaStream_t)stream>>>(d, bvol(db), sv, bvol(sb), w, ncomp);
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
    Region rg = region_of(r);
    FieldView<double> ov = view_of(out, ob, rg);
    FieldView<const double> xv = view_of(x, xb, rg), yv = view_of(y, yb, rg);
    turn_thin(rg, ov, xv, yv);
    const Walk w = walk_spread(rg);
    k_axpby<<<walk_grid(w, 1), kWalkThreads, 0, (cudaStream_t)stream>>>(ov, xv, yv, w, a, b);
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
    Region rg = region_of(rb);
    FieldView<double> d = view_of(dst, db, rg);
    CoarseMap m;
    m.ratio = fast_div(ratio);
    m.shift = 31 - __builtin_clz((unsigned)ratio);
    for (int k = 0; k < 3; k++) {
        const int c = floor_div(rb.lo[k], ratio);
        m.off[k] = rb.lo[k] - c * ratio;
        m.first[k] = c - sb.lo[k];
    }
    FieldView<const double> sv{src, bsize(sb, 0), bsize(sb, 0) * bsize(sb, 1)};
    if (turn_thin(rg, d, sv)) {
        std::swap(m.off[1], m.off[2]);
        std::swap(m.first[1], m.first[2]);
    }
    const Walk w = walk_spread(rg);
    cudaStream_t st = (cudaStream_t)stream;
    if (ratio & (ratio - 1)) k_interp_const<false><<<walk_grid(w, 1), kWalkThreads, 0, st>>>(sv, m, d, w, overwrite, scale);
    else k_interp_const<true><<<walk_grid(w, 1), kWalkThreads, 0, st>>>(sv, m, d, w, overwrite, scale);
    PB_LAUNCH_CHECK();
    return PB_OK;
}

} // extern "C"
