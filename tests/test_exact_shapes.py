"""Exact insertion (precision 1) where its screen's kernels can go wrong: rows
whose stored entries exceed the shared-memory stage (data far from the origin,
so that the pair bound admits a tenth of the columns), the column tile counts
around the seeded screen's threshold, and blocks of one row.  Lists bit for bit
against the oracle's brute force."""
import numpy as np
import pytest

from gpumap_gb300.datasets import gaussian_mixture
from test_gpu_parity import same_result, same_state

pytestmark = pytest.mark.gpu


def build(native, oracle_mod, X, steps, k=15, metric=0):
    n, d = X.shape
    s = native.Session(native.default_params(n_instances=n, n_features=d, n_neighbors=k, metric=metric, max_epoch=5,
                                             device=0, precision=1))
    o = oracle_mod.OracleSession(n, d, k=k, metric=metric, max_epoch=5, precision=1)
    s.set_stats(True)
    c0 = 0
    for rows in steps:
        s.append_host(X[c0 : c0 + rows])
        o.append(X[c0 : c0 + rows])
        c0 += rows
        same_result(s.run(rows, 0, 0), o.run(rows, 0, 0))
        same_state(s, o, tag=f"rows {c0}")
    assert c0 == n
    return s


@pytest.mark.parametrize("offset", [20.0, 26.0, 32.0, 42.0, 120.0])
def test_wide_bounds(native, oracle_mod, offset):
    # from a few hundred stored entries a row to more than the segments hold
    X = (np.random.default_rng(1).normal(size=(9600, 8)) + offset).astype(np.float32)
    s = build(native, oracle_mod, X, [9000, 599, 1])
    print("offset", offset, "overflowed blocks", s.stats().exact_overflow_blocks)


@pytest.mark.parametrize("steps", [[1, 1, 254, 1], [1023, 1, 1, 256], [1279, 1, 1, 300], [4096, 63, 129], [8191, 1, 1]])
def test_tile_edges(native, oracle_mod, steps):
    X, _ = gaussian_mixture(sum(steps), 40, seed=len(steps) + steps[0])
    build(native, oracle_mod, X, steps)
