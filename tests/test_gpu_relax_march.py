"""Sweeps of levels below 128 around the lines between the marching and the star kernels, odd edges (a last
row without a partner, a last chunk of one plane) among them."""
import numpy as np
import pytest

from proto_b200 import workloads as W
from tests.test_gpu_mg import _gpu_solve

pytestmark = pytest.mark.gpu


def _problem(n, form):
    if form == "poisson":
        return None, W.poisson_rho(n, seed=1)
    return W.helmholtz_alpha(n, seed=3), -W.poisson_rho(n, seed=1)


# FP64 levels that march: 41 to 64 but 48 and 56, and 81 to 96. 126 -> 63 and 180 -> 90 sweep it as a coarse level
@pytest.mark.parametrize("n,levels", [(40, 0), (41, 0), (52, 0), (56, 0), (57, 0), (63, 0), (64, 0), (65, 0), (80, 0), (81, 0), (95, 0), (96, 0), (97, 0),
                                      (126, 1), (122, 1), (180, 1)])
@pytest.mark.parametrize("form", ["poisson", "helmholtz"])
def test_fp64_edges_bitwise(pb, port, n, levels, form):
    alpha, rhs = _problem(n, form)
    it, hist, phi = _gpu_solve(pb, n, levels, pb.MG_FP64, max_iter=2, alpha=alpha, rhs=rhs)
    p2 = np.zeros(n ** 3)
    n2, h2 = port.mg_cs(n, levels, 4, 4, 10, 2.0 / 3.0, 1.0, None if alpha is None else alpha.reshape(-1).copy(), 2, 1e-10,
                        rhs.reshape(-1).copy(), p2)
    assert it == n2 and hist == list(h2)
    assert np.array_equal(phi, p2)


# FP32 levels that march: below 48 the edges that are no multiple of 8, 48 to 64, and 72 to 127
@pytest.mark.parametrize("n,levels", [(18, 1), (22, 1), (30, 1), (36, 2), (44, 2), (50, 1), (58, 1), (66, 1), (70, 1), (72, 1), (94, 1),
                                      (122, 1), (126, 1)])
@pytest.mark.parametrize("form", ["poisson", "helmholtz"])
def test_fp32_edges_follow_fp64(pb, n, levels, form):
    """The residual history of mixed precision against FP64's. A cycle's correction goes through about 20 sweeps,
    each rounding its 8 terms to 2^-24; the residual takes 12 times that: 20 * 8 * 12 * 2^-24 = 1.2e-4 of the
    first residual. One wrong row is a change of a hundredth."""
    alpha, rhs = _problem(n, form)
    _, h64, _ = _gpu_solve(pb, n, levels, pb.MG_FP64, max_iter=3, alpha=alpha, rhs=rhs)
    _, hmx, _ = _gpu_solve(pb, n, levels, pb.MG_MIXED, max_iter=3, alpha=alpha, rhs=rhs)
    assert hmx[0] == h64[0] and len(hmx) == len(h64)
    assert np.max(np.abs(np.array(hmx) - np.array(h64))) <= 1.2e-4 * h64[0]
