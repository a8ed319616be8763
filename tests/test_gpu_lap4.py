"""The 4th-order flux-form Laplacian's march (BoxOp_Laplace on boxes, the FAS solver's passes) at the edges
of its lane, row-pair and plane groups, and the FAS levels that share one CTA."""
import numpy as np
import pytest

from proto_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(1, 1, 1), (2, 3, 5), (31, 2, 4), (32, 16, 8), (33, 17, 9), (65, 15, 3), (40, 33, 34), (96, 7, 70)])
@pytest.mark.parametrize("scale", [1.0, -0.5])
def test_boxop_sizes(pb, port, n, scale):
    import ctypes
    import torch
    rng = np.random.default_rng(sum(n))
    lo = (3, -2, 1)
    # the state reaches three cells out in x, two elsewhere; the range leaves a border of the output alone
    sb = (tuple(lo[d] - (3 if d == 0 else 2) for d in range(3)), tuple(lo[d] + n[d] + 1 for d in range(3)))
    ob = (tuple(v - 1 for v in lo), tuple(lo[d] + n[d] for d in range(3)))
    rb = (lo, tuple(lo[d] + n[d] - 1 for d in range(3)))
    shape = lambda b: tuple(b[1][d] - b[0][d] + 1 for d in (2, 1, 0))
    u, want = rng.uniform(-1, 1, shape(sb)), rng.uniform(-1, 1, shape(ob))
    u[0, 0, 0] = -0.0
    du, do = torch.from_numpy(u).cuda(), torch.from_numpy(want.copy()).cuda()
    box = lambda b: pb.Box(*b).c()
    dbl = ctypes.c_double
    st = pb.lib().pb_boxop_laplace_f64(ctypes.c_void_p(du.data_ptr()), box(sb), ctypes.c_void_p(do.data_ptr()), box(ob),
                                       box(rb), dbl(1.0 / 16), dbl(-1.0), dbl(scale), None)
    assert st == 0
    torch.cuda.synchronize()
    port.boxop_laplace(u, sb, want, ob, rb, 1.0 / 16, -1.0, scale)
    assert np.array_equal(do.cpu().numpy(), want)


# (edge, levels): tops above and below the shared-memory levels, odd coarsest grids, edges below the ghost
# width, coarsest grids that keep their own launches, and a single level
@pytest.mark.parametrize("n,levels,cycles", [(16, 1, 2), (3, 1, 2), (8, 4, 3), (32, 6, 3), (20, 3, 3), (24, 4, 3), (28, 3, 2),
                                             (36, 2, 2), (40, 2, 2), (44, 3, 2), (34, 2, 2), (96, 6, 2)])
def test_fas_level_shapes(pb, port, n, levels, cycles):
    import torch
    force = -W.poisson_rho(n, seed=n).reshape(-1).copy()
    mg = pb.FAS(n, levels)
    phi = torch.zeros(n ** 3, dtype=torch.float64, device="cuda")
    for _ in range(2):                       # the captured cycle, then its replay
        phi.zero_()
        it, hist = mg.solve(torch.from_numpy(force).cuda(), phi, max_iter=cycles, tol=1e-14)
    pb.device_check()
    want = np.zeros(n ** 3)
    n2, h2 = port.mg_fas(n, levels, cycles, 1e-14, force, want)
    assert it == n2 and hist == list(h2)
    assert np.array_equal(phi.cpu().numpy(), want)


def test_fas_solve_waits_for_its_own_stream_only(pb):
    """A solve on a stream of its own ends while the default stream is still busy."""
    import torch
    m, side = pb.FAS(32, 3), torch.cuda.Stream()
    f = torch.from_numpy(np.random.default_rng(2).uniform(-1, 1, 32 ** 3)).cuda()
    phi = torch.zeros_like(f)
    torch.cuda.synchronize()
    want = m.solve(f, phi, max_iter=3, tol=0.0, stream=side.cuda_stream)     # captures its graphs
    phi.zero_()
    torch.cuda.synchronize()
    busy = torch.cuda.Event()
    torch.cuda._sleep(1 << 30)                                               # about half a second
    busy.record()
    assert m.solve(f, phi, max_iter=3, tol=0.0, stream=side.cuda_stream) == want
    assert not busy.query()
    torch.cuda.synchronize()
