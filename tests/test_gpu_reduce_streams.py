"""Reductions from several threads and streams at once: no call uses another's scratch or result word."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROUNDS = 150


def _fields(pb, count):
    """Fields of different sizes with their exact maximum norms, sums (of whole numbers) and boxes."""
    import torch
    out = []
    for k in range(count):
        n = (40 + 13 * k, 31 + k, 29)
        rng = np.random.default_rng(k)
        a = rng.integers(-1000, 1000, n[0] * n[1] * n[2]).astype(np.float64)
        a[k] = 2000.0 + k
        out.append((torch.from_numpy(a).cuda(), pb.Box((0, 0, 0), tuple(v - 1 for v in n)), np.abs(a).max(), a.sum()))
    torch.cuda.synchronize()
    return out


def _run(jobs):
    errors = []

    def body(job):
        try:
            job()
        except Exception as e:      # reported by the main thread
            errors.append(e)

    threads = [threading.Thread(target=body, args=(j,)) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[0]


@pytest.mark.parametrize("shared_stream", [False, True])
def test_threads_get_their_own_results(pb, shared_stream):
    import torch
    streams = [torch.cuda.Stream() for _ in range(4)]

    def job(k, field):
        d, b, absmax, total = field
        st = streams[0 if shared_stream else k].cuda_stream
        res = torch.zeros(ROUNDS, dtype=torch.float64, device="cuda")
        torch.cuda.current_stream().synchronize()
        for i in range(ROUNDS):
            pb.reduce_async(pb.RED_SUM, d, b, res[i:], stream=st)
            assert pb.reduce(pb.RED_ABS, d, b, stream=st) == absmax
        assert (res.cpu().numpy() == total).all()

    _run([lambda k=k, f=f: job(k, f) for k, f in enumerate(_fields(pb, 4))])


def test_more_streams_than_slots(pb):
    """Asynchronous calls from 64 streams, unordered between them."""
    import torch
    fields = _fields(pb, 5)
    streams = [torch.cuda.Stream() for _ in range(32)] + [torch.cuda.Stream(priority=-1) for _ in range(32)]
    res = torch.zeros((3, len(streams)), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    for i in range(3):
        for k, st in enumerate(streams):
            d, b, _, _ = fields[k % 5]
            pb.reduce_async(pb.RED_SUM, d, b, res[i, k:], stream=st.cuda_stream)
    torch.cuda.synchronize()
    want = np.array([fields[k % 5][3] for k in range(len(streams))])
    assert (res.cpu().numpy() == want).all()


def test_captured_reductions_run_beside_others(pb):
    """A replayed graph of reductions (captured on a stream that never reduced before) and calls on other
    streams; graphs come and go, their slots are used again."""
    import torch
    fields = _fields(pb, 3)
    st, other = torch.cuda.Stream(), torch.cuda.Stream()
    res, spare = torch.zeros(3, dtype=torch.float64, device="cuda"), torch.zeros(1, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    for _ in range(3):
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=st):
            for k, (d, b, _, _) in enumerate(fields):
                pb.reduce_async(pb.RED_SUM, d, b, res[k:], stream=st.cuda_stream)
        for _ in range(40):
            with torch.cuda.stream(st):
                res.zero_()
                g.replay()
            d, b, absmax, _ = fields[1]
            assert pb.reduce(pb.RED_ABS, d, b, stream=other.cuda_stream) == absmax
            pb.reduce_async(pb.RED_ABS, d, b, spare, stream=other.cuda_stream)
            st.synchronize()
            assert (res.cpu().numpy() == [f[3] for f in fields]).all()
        other.synchronize()
        del g
