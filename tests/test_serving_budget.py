"""Admission with an update in the request: the update's join pool takes what the
budget leaves it, in more passes, and does not refuse the request."""
import numpy as np
import pytest

from gpumap_gb300.datasets import gaussian_mixture
from test_gpu_parity import pair, same_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("room", [100 << 10, 1 << 20, 1 << 30])
def test_update_within_the_budget(native, oracle_mod, room):
    from gpumap_gb300.serving import Server

    n, d, k = 3000, 16, 15
    X, _ = gaussian_mixture(n, d, seed=8)
    _, o = pair(native, oracle_mod, n, d, k=k, max_epoch=5)
    p = native.default_params(n_instances=n, n_features=d, n_neighbors=k, max_epoch=5, device=0)
    with Server(slots=1, hbm_budget=10**12) as srv:  # what the session holds once its rows are in
        sid = srv.open_session(p)
        assert srv.wait(srv.submit(sid, X, 0, 0)).status == 0
        held = srv.stats().bytes_in_use
    with Server(slots=1, hbm_budget=held + room) as srv:
        sid = srv.open_session(p)
        assert srv.wait(srv.submit(sid, X, 0, 0)).status == 0
        o.append(X)
        o.run(n, 0, 0)
        none = np.zeros((0, d), np.float32)
        for upd in (n, 700):  # every row; a part
            assert srv.wait(srv.submit(sid, none, upd, 0)).status == 0
            assert srv.stats().bytes_in_use <= held + room
            o.run(0, upd, 0)
        same_state(srv.session(sid), o, tag=f"{room} bytes for the pool")
