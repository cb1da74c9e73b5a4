"""Exact insertion of rows that come ordered by cluster: a row's neighbours lie
side by side, so the seed (chunk minima of all columns) admits whole tiles.  Up to
32 column tiles the segments of stored columns hold them all.  Lists bit for bit
against the oracle, and the path is asserted."""
import numpy as np
import pytest

from gpumap_gb300.datasets import gaussian_mixture
from test_exact_shapes import build

pytestmark = pytest.mark.gpu


def ordered(n, d, clusters, seed, spread=4.0):
    rng = np.random.default_rng(seed)
    c = spread * rng.normal(size=(clusters, d))
    z = np.sort(rng.integers(0, clusters, n))
    return (c[z] + rng.normal(size=(n, d))).astype(np.float32)


@pytest.mark.parametrize("n,d,clusters,cycle,metric", [
    (4999, 131, 10, 333, 0),   # five to twenty tiles, ragged blocks
    (4999, 131, 10, 333, 1),
    (8000, 16, 20, 1024, 0),   # 32 tiles, blocks of eight row tiles
    (8192, 16, 8, 700, 0),     # the last column of the last of them
])
def test_no_block_overflows(native, oracle_mod, n, d, clusters, cycle, metric):
    X = ordered(n, d, clusters, seed=n + d)
    steps = [min(cycle, n - c) for c in range(0, n, cycle)]
    s = build(native, oracle_mod, X, steps, metric=metric)
    assert s.stats().exact_overflow_blocks == 0


@pytest.mark.parametrize("n,offset,overflows,wide", [
    (9600, 20.0, False, False),  # 38 tiles: common path
    (9600, 120.0, True, False),  # segments too short: every block takes the heap and candidate passes
    (8000, 20.0, False, False),  # 32 tiles: room for every column
    (8000, 120.0, False, True),  # and more stored than the selection stages
])
def test_path_of_wide_bounds(native, oracle_mod, n, offset, overflows, wide):
    from test_exact_wide_rows import wide_rows

    X = (np.random.default_rng(1).normal(size=(n, 8)) + offset).astype(np.float32)
    s = build(native, oracle_mod, X, [n - 600, 599, 1])
    assert (s.stats().exact_overflow_blocks > 0) == overflows
    assert (wide_rows(native, s) > 0) == wide
