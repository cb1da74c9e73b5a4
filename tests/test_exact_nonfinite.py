"""Rows with NaN or infinite features among others, precision 1: such a row has no
neighbours and is nobody's, and every other row's list is that of the data
without it, bit for bit against the oracle."""
import numpy as np
import pytest

from gpumap_gb300.datasets import gaussian_mixture

pytestmark = pytest.mark.gpu

SENTINEL = 0x7FFFFFFF


@pytest.mark.parametrize("metric", [0, 1])
@pytest.mark.parametrize("n,cap", [(900, None), (3000, None), (3000, 0), (3000, 1), (9600, None)])
def test_other_rows_lists(native, oracle_mod, n, cap, metric):
    # column tiles: 4 (no seed), 12 (seed and store; heaps; overflow), 38
    d = 24
    X, _ = gaussian_mixture(n, d, seed=n + metric)
    rng = np.random.default_rng(n)
    bad = np.unique(np.concatenate([rng.integers(0, n, 25), [0, n // 2, n - 1]]))
    X[bad[::3], 3] = np.nan
    X[bad[1::3], d - 1] = np.inf
    X[bad[2::3]] = -np.inf
    X[5] = 0.0  # (its bound factor is 0)
    bad = bad[bad != 5]
    good = np.setdiff1d(np.arange(n), bad)
    s = native.Session(native.default_params(n_instances=n, n_features=d, n_neighbors=15, metric=metric, device=0,
                                             precision=1))
    if cap is not None:
        s.pre_capacity(cap)
    o = oracle_mod.OracleSession(good.size, d, k=15, metric=metric, precision=1)
    for c0, c1 in ((0, n // 2), (n // 2, n - 70), (n - 70, n)):
        s.append_host(X[c0:c1])
        s.run(c1 - c0, 0, 0)
        part = good[(good >= c0) & (good < c1)]
        o.append(X[part])
        o.run(part.size, 0, 0)
    ids, dists = s.copy("graph_ids", np.int32).reshape(n, 32), s.copy("graph_dists", np.float32).reshape(n, 32)
    want = o.copy("graph_ids", np.int32).reshape(good.size, 32)
    assert (ids[bad] == SENTINEL).all()
    assert np.array_equal(ids[good], good[want])
    assert np.array_equal(dists[good], o.copy("graph_dists", np.float32).reshape(good.size, 32))
