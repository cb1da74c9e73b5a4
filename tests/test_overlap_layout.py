"""The layout of an overlapped build against the same build with the phases in
order, at a small learning rate, where repeats of one build differ only by the
SGD's concurrent updates (about 1e-5 of the layout's norm).  Every kernel reads
what it would read in order, so the two modes' layouts may differ by little more
than repeats do; a kernel that read positions or lists before their turn moves
whole rows (1e-3 and more)."""
import numpy as np
import pytest

from gpumap_gb300.datasets import gaussian_mixture

pytestmark = pytest.mark.gpu

REPEATS = 6


def layouts(native, X, overlap, precision, chunk=500, emb=700, upd=0):
    n, d = X.shape
    out = []
    for _ in range(REPEATS):
        s = native.Session(native.default_params(n_instances=n, n_features=d, n_neighbors=15, max_epoch=50, device=0, alpha=1e-4,
                                                 a=1.577, b=0.895, precision=precision, overlap=overlap))
        for c in range(0, n, chunk):
            s.append_host(X[c : c + chunk])
            s.run(chunk, upd, emb)
        out.append(s.copy("embedding", np.float32).astype(np.float64))
    return out


def distance(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(a)


@pytest.mark.parametrize("precision,upd", [(1, 0), (0, 0), (1, 500)])
def test_overlapped_layout(native, precision, upd):
    X, _ = gaussian_mixture(5000, 24, seed=9)
    plain, over = (layouts(native, X, o, precision, upd=upd) for o in (0, 1))
    own = [np.median([distance(a, b) for i, a in enumerate(x) for b in x[:i]]) for x in (plain, over)]
    across = np.median([distance(a, b) for a in plain for b in over])
    print("repeats", own, "across", across)
    assert max(own) < 1e-4  # (else the comparison says nothing)
    assert across < 10 * max(own)
