"""A device error (the word a bounded wait sets, here written by a hook) is
reported by the next run, also when its insertion and update have nothing to do,
and the queues stay as the phases left them."""
import numpy as np
import pytest

from gpumap_gb300.datasets import gaussian_mixture

pytestmark = pytest.mark.gpu


def session(native, X, **kw):
    n, d = X.shape
    return native.Session(native.default_params(n_instances=n, n_features=d, max_epoch=5, device=0, **kw))


@pytest.mark.parametrize("ops", [(0, 0, 50), (100, 0, 50), (0, 0, 0), (0, 40, 0), (100, 40, 50)])
def test_reported_by_the_next_run(native, ops):
    X, _ = gaussian_mixture(1000, 8, seed=1)
    s = session(native, X, precision=1, overlap=1)
    s.append_host(X[:500])
    s.run(500, 0, 200)
    native.check(native.load().gm_debug_raise(s.handle, 2))
    with pytest.raises(native.GMError, match="wait ran out"):
        s.run(*ops)
    # reported once; the session goes on
    s.append_host(X[500:])
    assert s.run(500, 0, 200).n_insertion_ops == 500


@pytest.mark.parametrize("precision,ops", [(0, (300, 0, 0)), (1, (300, 0, 0)), (0, (300, 1500, 0))])
def test_queues_after_an_error(native, precision, ops):
    X, _ = gaussian_mixture(1000, 8, seed=2)
    left = []
    for fail in (False, True):
        s = session(native, X, precision=precision)
        s.append_host(X)
        s.run(600, 0, 0)
        if fail:
            native.check(native.load().gm_debug_raise(s.handle, 2))
            with pytest.raises(native.GMError, match="wait ran out"):
                s.run(ops[0], 0, 0)
            if ops[1]:
                native.check(native.load().gm_debug_raise(s.handle, 2))
                with pytest.raises(native.GMError, match="wait ran out"):
                    s.run(0, ops[1], 0)
        else:
            s.run(ops[0], 0, 0)
            if ops[1]:
                s.run(0, ops[1], 0)
        left.append((s.update_queue(), s.copy("knn_ids", np.int32), s.scalars()))
    assert np.array_equal(left[0][0], left[1][0]) and np.array_equal(left[0][1], left[1][1])
    assert left[0][2] == left[1][2]
