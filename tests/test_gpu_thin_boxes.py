"""Lines, faces and slabs: the pointwise, reduction, prolongation and stencil kernels give the right values
there, and a thin box costs what a solid one of as many cells does."""
import ctypes
import math

import numpy as np
import pytest

from tests.util import table

pytestmark = pytest.mark.gpu

LINE = 4099
THIN = [(LINE, 1, 1), (1, LINE, 1), (1, 1, LINE), (LINE, 3, 1), (2, LINE, 1), (3, 1, LINE), (301, 150, 1), (301, 1, 150),
        (1, 301, 150), (2, 150, 301), (150, 2, 301), (150, 301, 2), (5, 5, 2000), (75777, 1, 1)]


def _dev(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _box(pb, n, g=0):
    return pb.Box((-g,) * 3, tuple(v - 1 + g for v in n))


def _shape(n, g=0):
    return tuple(v + 2 * g for v in reversed(n))


@pytest.mark.parametrize("n", THIN)
def test_pointwise_and_reductions(pb, n):
    rng = np.random.default_rng(sum(n))
    x, y = rng.uniform(1, 2, _shape(n, 1)), rng.uniform(1, 2, _shape(n))
    inner = x[1:-1, 1:-1, 1:-1]
    b, gb = _box(pb, n), _box(pb, n, 1)
    dx, dy, out = _dev(x), _dev(y), _dev(np.zeros(_shape(n)))
    pb.forall_axpby(out, b, dx, gb, dy, b, 0.5, -2.0)
    assert np.array_equal(out.cpu().numpy(), 0.5 * inner + (-2.0) * y)
    pb.boxdata_op(pb.OP_MUL, dy, b, dx, gb)
    pb.boxdata_scalar(pb.OP_SUB, dy, b, 0.3)
    assert np.array_equal(dy.cpu().numpy(), y * inner - 0.3)
    # a face or line of a larger field moved into it
    pb.boxdata_copy(dy, b, dx, gb, shift=(1, 0, -1))
    want = x.copy()
    want[0:-2, 1:-1, 2:] = y * inner - 0.3
    assert np.array_equal(dx.cpu().numpy(), want)
    v = (x - 1.5)
    d = _dev(v)
    w = v[1:-1, 1:-1, 1:-1].reshape(-1)
    assert pb.reduce(pb.RED_MAX, d, gb, b) == max(w.max(), np.finfo(np.float64).tiny)
    assert pb.reduce(pb.RED_MIN, d, gb, b) == w.min()
    assert pb.reduce(pb.RED_ABS, d, gb, b) == np.abs(w).max()
    # any order of the additions: |error| <= N u sum |w|
    for op, t in ((pb.RED_SUM, w), (pb.RED_SUMABS, np.abs(w)), (pb.RED_SUMSQ, w * w)):
        assert abs(pb.reduce(op, d, gb, b) - math.fsum(t)) <= len(t) * 2.0 ** -53 * math.fsum(np.abs(t))


@pytest.mark.parametrize("ratio", [2, 3])
@pytest.mark.parametrize("n", THIN)
def test_constant_prolongation(pb, n, ratio):
    rng = np.random.default_rng(sum(n) + ratio)
    lo = (-1, 3, -5)
    clo = [v // ratio for v in lo]
    chi = [(lo[d] + n[d] - 1) // ratio for d in range(3)]
    src = rng.uniform(-1, 1, tuple(chi[d] - clo[d] + 1 for d in (2, 1, 0)))
    dst = rng.uniform(-1, 1, _shape(n))
    dd = _dev(dst)
    pb.interp_constant(ratio, _dev(src), pb.Box(clo, chi), dd, pb.Box(lo, [lo[d] + n[d] - 1 for d in range(3)]), scale=0.75)
    at = [(np.arange(n[d]) + lo[d]) // ratio - clo[d] for d in (2, 1, 0)]
    assert np.array_equal(dd.cpu().numpy(), dst + 0.75 * src[np.ix_(*at)])


def _boxop(pb, src, sb, dst, db):
    import torch
    status = pb.lib().pb_boxop_laplace_f64(ctypes.c_void_p(src.data_ptr()), sb.c(), ctypes.c_void_p(dst.data_ptr()), db.c(),
                                           db.c(), ctypes.c_double(0.125), ctypes.c_double(-1.0), ctypes.c_double(1.0),
                                           ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert status == 0


@pytest.mark.parametrize("n", THIN + [(33, 33, 33), (65, 40, 9)])
@pytest.mark.parametrize("name", ["laplacian27", "laplacian19", "corners2cells4", "boxop"])
def test_stencils(golden, pb, name, n):
    """Thin boxes against the same cells inside a solid one, which other tests pin."""
    import torch
    g = 3
    solid = tuple(max(v, 40) for v in n) if max(n) <= 301 else tuple(max(v, 8) for v in n)
    rng = np.random.default_rng(sum(n))
    src = _dev(rng.uniform(-1, 1, _shape(solid, g)))
    sb, b, whole = _box(pb, solid, g), _box(pb, n), _box(pb, solid)
    out, ref = _dev(np.zeros(_shape(n))), _dev(np.zeros(_shape(solid)))
    if name == "boxop":
        _boxop(pb, src, sb, out, b)
        _boxop(pb, src, sb, ref, whole)
    else:
        c, o, _ = table(golden[1], name)
        S = pb.Stencil(c, o)
        S.apply(src, sb, out, b, b)
        S.apply(src, sb, ref, whole, whole)
    assert torch.equal(out, ref[:n[2], :n[1], :n[0]])


def _us(f, calls=10):
    """Device time of one call, launches aside."""
    import torch
    st = torch.cuda.Stream()
    with torch.cuda.stream(st):
        f()
        st.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=st):
            for _ in range(calls):
                f()
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        best = math.inf
        for _ in range(5):
            a.record(st)
            graph.replay()
            b.record(st)
            st.synchronize()
            best = min(best, a.elapsed_time(b) * 1e3 / calls)
    return best


@pytest.mark.parametrize("name", ["add", "copy", "interp3", "reduce", "laplacian27", "boxop"])
def test_a_line_costs_what_a_solid_box_does(golden, pb, name):
    """The same 2^18 cells as a 64^3 box and as lines along each axis. The bound is loose: a line reads up to 25
    times the source of a solid box's stencil. A kernel that leaves lanes or blocks idle on lines takes 20
    to 1000 times as long."""
    import torch
    g = {"laplacian27": 1, "boxop": 2}.get(name, 0)
    times = []
    for n in [(64, 64, 64), (1 << 18, 1, 1), (1, 1 << 18, 1), (1, 1, 1 << 18)]:
        src = torch.rand(int(np.prod(_shape(n, g))), dtype=torch.float64, device="cuda")
        dst = torch.zeros(int(np.prod(n)), dtype=torch.float64, device="cuda")
        sb, b = _box(pb, n, g), _box(pb, n)
        res = torch.zeros(1, dtype=torch.float64, device="cuda")
        S = pb.Stencil(*table(golden[1], "laplacian27")[:2])
        times.append(_us({"add": lambda: pb.boxdata_op(pb.OP_ADD, dst, b, src, sb),
                          "copy": lambda: pb.boxdata_copy(src, sb, dst, b),
                          "interp3": lambda: pb.interp_constant(3, src, sb, dst, b),
                          "reduce": lambda: pb.reduce_async(pb.RED_ABS, src, sb, res),
                          "laplacian27": lambda: S.apply(src, sb, dst, b, b),
                          "boxop": lambda: _boxop(pb, src, sb, dst, b)}[name]))
    assert max(times[1:]) <= 8 * times[0], times
