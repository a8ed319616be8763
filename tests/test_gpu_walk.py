"""The row-walking kernels (pointwise, copy, reductions, constant prolongation, table stencils) at the
edges of their lane, row and plane groups."""
import math

import numpy as np
import pytest

from tests.util import table

pytestmark = pytest.mark.gpu

# x: below, at and above a lane group; y: rows of a block; z: the four- and eight-plane groups
SIZES = [(1, 1, 1), (7, 33, 4), (8, 31, 5), (9, 9, 3), (16, 17, 8), (17, 8, 9), (32, 1, 13), (33, 7, 16), (70, 12, 7)]


def _dev(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _cube(n, lo=(0, 0, 0), g=0):
    return tuple(l - g for l in lo), tuple(l + k - 1 + g for l, k in zip(lo, n))


def _inner(a, g):
    return a[..., g:a.shape[-3] - g, g:a.shape[-2] - g, g:a.shape[-1] - g] if g else a


@pytest.mark.parametrize("n", SIZES)
def test_pointwise_and_copy(pb, n):
    rng = np.random.default_rng(sum(n))
    nx, ny, nz = n
    lo = (-3, 5, -1)
    vb, gb = pb.Box(*_cube(n, lo)), pb.Box(*_cube(n, lo, 1))
    x = rng.uniform(1, 2, (2, nz + 2, ny + 2, nx + 2))
    y = rng.uniform(1, 2, (2, nz, ny, nx))
    dy, dx = _dev(y), _dev(x)
    pb.boxdata_op(pb.OP_DIV, dy, vb, dx, gb, ncomp=2)
    pb.boxdata_scalar(pb.OP_SUB, dy, vb, 0.3, ncomp=2)
    want = y / _inner(x, 1) - 0.3
    assert np.array_equal(dy.cpu().numpy(), want)
    out = _dev(np.zeros((nz, ny, nx)))
    pb.forall_axpby(out, vb, dx, gb, dy, vb, 0.5, -2.0)
    assert np.array_equal(out.cpu().numpy(), 0.5 * _inner(x, 1)[0] + (-2.0) * want[0])
    moved = _dev(np.zeros((2, nz, ny, nx)))
    pb.boxdata_copy(dx, gb, moved, pb.Box(*_cube(n, (0, 0, 0))), shift=(4, -4, 2), ncomp=2)
    full = np.zeros((2, nz, ny, nx))
    # source point p goes to p + shift: destination (i, j, k) holds source (i-4, j+4, k-2)
    for k in range(nz):
        for j in range(ny):
            for i in range(nx):
                sx, sy, sz = i - 4 - (lo[0] - 1), j + 4 - (lo[1] - 1), k - 2 - (lo[2] - 1)
                if 0 <= sx < nx + 2 and 0 <= sy < ny + 2 and 0 <= sz < nz + 2:
                    full[:, k, j, i] = x[:, sz, sy, sx]
    assert np.array_equal(moved.cpu().numpy(), full)


@pytest.mark.parametrize("n", SIZES + [(64, 64, 70), (5, 300, 41)])
def test_reductions(pb, n):
    rng = np.random.default_rng(sum(n) + 1)
    nx, ny, nz = n
    a = rng.uniform(-1, 1, (nz + 2, ny + 2, nx + 2))
    d, gb, vb = _dev(a), pb.Box(*_cube(n, g=1)), pb.Box(*_cube(n))
    v = _inner(a, 1).reshape(-1)
    assert pb.reduce(pb.RED_MAX, d, gb, vb) == max(v.max(), np.finfo(np.float64).tiny)
    assert pb.reduce(pb.RED_MIN, d, gb, vb) == v.min()
    assert pb.reduce(pb.RED_ABS, d, gb, vb) == np.abs(v).max()
    # any order of the additions: |error| <= (N - 1) u sum |v|
    for op, w in ((pb.RED_SUM, v), (pb.RED_SUMABS, np.abs(v)), (pb.RED_SUMSQ, v * v)):
        assert abs(pb.reduce(op, d, gb, vb) - math.fsum(w)) <= len(w) * 2.0 ** -53 * math.fsum(np.abs(w))


def test_reductions_nan_and_empty(pb):
    a = np.array([np.nan, -3.0, 2.0, np.nan] * 9)
    d, b = _dev(a), pb.Box((0, 0, 0), (35, 0, 0))
    assert pb.reduce(pb.RED_ABS, d, b) == 3.0 and pb.reduce(pb.RED_MIN, d, b) == -3.0 and pb.reduce(pb.RED_MAX, d, b) == 2.0
    assert math.isnan(pb.reduce(pb.RED_SUM, d, b))
    away = pb.Box((100, 0, 0), (101, 0, 0))
    assert pb.reduce(pb.RED_SUM, d, b, away) == 0.0 and pb.reduce(pb.RED_MIN, d, b, away) == np.finfo(np.float64).max


@pytest.mark.parametrize("ratio", [1, 2, 3, 4])
@pytest.mark.parametrize("overwrite", [False, True])
def test_constant_prolongation(pb, port, ratio, overwrite):
    rng = np.random.default_rng(ratio)
    sb = ((-3, -2, 1), (5, 3, 4))
    db = ((-3 * ratio - 1, -2 * ratio + 1, ratio - 2), (5 * ratio, 3 * ratio + 4, 4 * ratio + ratio - 1))
    shape = lambda b: tuple(b[1][d] - b[0][d] + 1 for d in (2, 1, 0))
    src, dst = rng.uniform(-1, 1, shape(sb)), rng.uniform(-1, 1, shape(db))
    dd = _dev(dst)
    pb.interp_constant(ratio, _dev(src), pb.Box(*sb), dd, pb.Box(*db), overwrite=overwrite, scale=0.75)
    port.interp_constant(ratio, src, sb, dst, db, overwrite, 0.75)
    assert np.array_equal(dd.cpu().numpy(), dst)


def _apply_both(pb, port, c, o, meta, n, dtype, ncomp=2, init=True, scale=1.0, ghost=2):
    """The device's and the oracle's (FP32: numpy's, term by term) result on the same inputs."""
    rng = np.random.default_rng(len(c) + sum(n))
    o = np.asarray(o).reshape(-1, 3)
    sr, dr, ds = [tuple(int(v) for v in meta[k:k + 3]) for k in (0, 3, 6)]
    sb = tuple(-ghost + 2 for _ in range(3)), tuple(2 + sr[d] * n[d] + ghost for d in range(3))
    db = tuple(ds[d] - 1 for d in range(3)), tuple(ds[d] + dr[d] * n[d] for d in range(3))
    shape = lambda b: (ncomp,) + tuple(b[1][d] - b[0][d] + 1 for d in (2, 1, 0))
    src, dst = rng.uniform(-1, 1, shape(sb)).astype(dtype), rng.uniform(-1, 1, shape(db)).astype(dtype)
    dd = _dev(dst)
    S = pb.Stencil(c, o, sr, dr, ds)
    S.apply(_dev(src), pb.Box(*sb), dd, pb.Box(*db), init_to_zero=init, scale=scale, ncomp=ncomp)
    ib = port.infer_box(o.reshape(-1), meta, sb, db)
    if dtype == np.float64:
        port.stencil_apply(c, o.reshape(-1), meta, src, sb, dst, db, ib, init, scale, ncomp)
        return dd.cpu().numpy(), dst
    lo, hi = [list(int(v) for v in p) for p in ib]
    src_at = lambda off: tuple(slice(lo[d] * sr[d] + off[d] - sb[0][d], hi[d] * sr[d] + off[d] - sb[0][d] + 1, sr[d]) for d in (2, 1, 0))
    dst_at = (slice(None),) + tuple(slice(lo[d] * dr[d] + ds[d] - db[0][d], hi[d] * dr[d] + ds[d] - db[0][d] + 1, dr[d]) for d in (2, 1, 0))
    acc = np.zeros_like(dst[dst_at]) if init else dst[dst_at].copy()
    for k, off in enumerate(o):
        w = np.float32(c[k]) * np.float32(scale) if scale != 1.0 else np.float32(c[k])
        acc = acc + w * src[(slice(None),) + src_at([int(v) for v in off])]
    dst[dst_at] = acc
    return dd.cpu().numpy(), dst


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("name", ["avgdown2", "laplacian27", "corners2cells4", "deriv_2_1_4"])
def test_table_stencils(golden, pb, port, name, dtype, n):
    c, o, meta = table(golden[1], name)
    got, want = _apply_both(pb, port, c, o, meta, n, dtype, init=sum(n) % 2 == 0, scale=0.5 if n[0] > 8 else 1.0)
    assert np.array_equal(got, want)


@pytest.mark.parametrize("sr,dr,ds", [((2, 1, 3), (1, 1, 1), (0, 0, 0)), ((1, 1, 1), (2, 3, 1), (1, -1, 2))])
def test_table_ratios_and_far_offsets(pb, port, sr, dr, ds):
    """Ratios, a destination shift, and a span that does not hold the origin."""
    o = np.array([(2, 1, 2), (1, 2, 2), (2, 2, 1)])
    got, want = _apply_both(pb, port, np.array([0.5, -1.25, 2.0]), o, np.array(sr + dr + ds), (9, 7, 6), np.float64, ghost=3)
    assert np.array_equal(got, want)


@pytest.mark.parametrize("n", [(193, 33, 24), (33, 70, 61), (64, 64, 32), (8, 257, 70)])   # above the column kernel's floor
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("name", ["laplacian19", "laplacian27"])
def test_cube_stencils(golden, pb, port, name, dtype, n):
    c, o, meta = table(golden[1], name)
    for init, scale in ((True, 3.0), (False, 1.0)):
        got, want = _apply_both(pb, port, c, o, meta, n, dtype, init=init, scale=scale, ghost=1)
        assert np.array_equal(got, want)
