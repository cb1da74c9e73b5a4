"""NN-Descent insertion (precision 0) at the sizes where its kernels can go
wrong: list widths around the 256-candidate rule, feature counts around the
32-feature chunk, fewer rows than list slots, ragged batches, and rows that are
appended but not yet inserted.  Bit for bit against the oracle."""
import numpy as np
import pytest

from gpumap_gb300.datasets import gaussian_mixture
from test_gpu_parity import pair, same_result, same_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,d,k,metric,append,insert", [
    (37, 3, 1, 0, 5, 5),            # one neighbour; fewer rows than list slots
    (700, 31, 15, 0, 233, 233),     # below the 256-candidate rule, chunk - 1 features
    (900, 33, 16, 0, 450, 450),     # exactly 256 positions, chunk + 1 features
    (900, 64, 17, 1, 300, 100),     # rows queued behind the inserted ones, cosine
    (1500, 129, 32, 0, 750, 333),   # the widest list, five chunks, ragged batches
    (600, 24, 30, 1, 600, 600),     # one batch, no existing rows
])
def test_insertion_bitexact(native, oracle_mod, n, d, k, metric, append, insert):
    X, _ = gaussian_mixture(n, d, seed=n + d + k)
    s, o = pair(native, oracle_mod, n, d, k=k, metric=metric, max_epoch=5)
    for c in range(0, n, append):
        chunk = X[c : c + append]
        s.append_host(chunk)
        o.append(chunk)
        for _ in range(max(1, append // insert)):
            same_result(s.run(insert, 0, 0), o.run(insert, 0, 0))
            same_state(s, o, tag=f"rows {c}")
    same_result(s.run(n, 2 * n, 0), o.run(n, 2 * n, 0))
    same_state(s, o, tag="update")
    assert np.isfinite(s.copy("embedding", np.float32)).all()
