"""Update rounds (NN-Descent local join) at the sizes where their kernels can
go wrong: small and large join nodes (32 members is the line), the widest and the
narrowest lists, feature counts around the 32-feature chunk, and rounds whose
node blocks take several passes over the join pool.  Bit for bit against the
oracle."""
import pytest

from gpumap_gb300.datasets import gaussian_mixture
from test_gpu_parity import pair, same_result, same_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,d,k,metric,words", [
    (40, 3, 1, 0, None),       # one neighbour
    (150, 31, 5, 0, None),     # small nodes only
    (700, 33, 16, 1, None),    # both kinds
    (900, 100, 32, 0, None),   # the widest lists, large nodes of up to 128 members
    (900, 64, 32, 0, 20_000),  # several passes
    (300, 8, 15, 0, 2),        # a pass for every block or two
])
def test_update_bitexact(native, oracle_mod, n, d, k, metric, words):
    X, _ = gaussian_mixture(n, d, seed=n + d + k)
    s, o = pair(native, oracle_mod, n, d, k=k, metric=metric, max_epoch=5)
    if words is not None:
        s.join_words(words)
    half = n // 2
    for c0, rows in ((0, half), (half, n - half)):
        chunk = X[c0 : c0 + rows]
        s.append_host(chunk)
        o.append(chunk)
        for upd in (rows // 3, rows, 3 * n):  # part of the queue, the queue and more, every row twice over
            same_result(s.run(rows, upd, 0), o.run(rows, upd, 0))
            same_state(s, o, tag=f"rows {c0}+{rows}, {upd} updates")
