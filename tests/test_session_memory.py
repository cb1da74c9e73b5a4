"""Sessions that come and go through the memory pool: results do not depend on
what the memory held before, a view still being read outlives its session, and
sessions of several threads keep apart."""
import threading

import numpy as np
import pytest

from gpumap_gb300.datasets import gaussian_mixture

pytestmark = pytest.mark.gpu


def build(native, X, precision, k=10, overlap=0):
    n, d = X.shape
    s = native.Session(native.default_params(n_instances=n, n_features=d, n_neighbors=k, max_epoch=20, device=0,
                                             precision=precision, overlap=overlap))
    for c in range(0, n, 300):
        s.append_host(X[c : c + 300])
        s.run(300, 300, 300)
    return s


def tables(s):
    return [s.copy(b, t) for b, t in (("pub_idx", np.uint32), ("pub_dist", np.float32), ("sigma", np.float32),
                                      ("sched_eps", np.float32), ("bloom", np.uint32))]


@pytest.mark.parametrize("precision,overlap", [(0, 0), (1, 0), (1, 1)])
def test_reused_memory(native, precision, overlap):
    A, _ = gaussian_mixture(1500, 20, seed=1)
    B, _ = gaussian_mixture(1100, 37, seed=2)
    first = tables(build(native, A, precision, overlap=overlap))
    for _ in range(3):  # other contents and other sizes in the same memory
        build(native, B, 1 - precision, k=17)
        again = tables(build(native, A, precision, overlap=overlap))
        for x, y in zip(first, again):
            assert np.array_equal(x, y)


def test_view_read_while_its_session_goes(native):
    import gpumap_gb300 as gm
    import torch
    from gpumap_gb300.data_loader import ArrayDataLoader

    X, _ = gaussian_mixture(20_000, 8, seed=3)
    p = gm.GPUMAPParams()
    p.n_instances, p.n_features, p.precision = 20_000, 8, 1
    big = torch.randn(8192, 8192, device="cuda")
    m = gm.GPUMAP(ArrayDataLoader(X), p)
    m.run_with_n_ops(20_000, 0, 0)
    want = m.get_neighbor_dists().cpu()
    view = m.get_neighbor_dists()
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        for _ in range(20):  # keeps the copy waiting
            big = torch.tanh(big @ big * 1e-4)
        got = view.clone()
    del view, m
    build(native, X[:3000], 1)  # may take the same memory
    side.synchronize()
    assert torch.equal(got.cpu(), want)


def test_threads(native):
    data = [gaussian_mixture(900, 10 + i, seed=i)[0] for i in range(4)]
    alone = [tables(build(native, X, i % 2)) for i, X in enumerate(data)]
    got = [None] * 4

    def work(i):
        for _ in range(3):
            got[i] = tables(build(native, data[i], i % 2))

    ts = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    for a, g in zip(alone, got):
        for x, y in zip(a, g):
            assert np.array_equal(x, y)
