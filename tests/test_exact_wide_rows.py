"""The exact screen's selection of a row's threshold and candidates where the
row has more stored columns than the shared-memory stage: data far from the
origin, whose pair bounds admit most columns, in a session with room for them.
Bit for bit against the oracle, and the path is asserted."""
import ctypes as C

import numpy as np
import pytest

from test_gpu_parity import same_result, same_state

pytestmark = pytest.mark.gpu


def wide_rows(native, s):
    out = (C.c_int64 * 12)()
    native.check(native.load().gm_debug_scalars(s.handle, out, 12))
    return out[11]


@pytest.mark.parametrize("offset,wide", [(20.0, False), (70.0, True), (120.0, True)])
def test_more_than_the_stage(native, oracle_mod, offset, wide):
    steps, room = [9000, 599, 1], 39_000  # segments for 9,728 columns a row
    X = (np.random.default_rng(1).normal(size=(sum(steps), 8)) + offset).astype(np.float32)
    s = native.Session(native.default_params(n_instances=room, n_features=8, max_epoch=5, device=0, precision=1))
    o = oracle_mod.OracleSession(room, 8, max_epoch=5, precision=1)
    s.set_stats(True)
    c0 = 0
    for rows in steps:
        s.append_host(X[c0 : c0 + rows])
        o.append(X[c0 : c0 + rows])
        c0 += rows
        same_result(s.run(rows, 0, 0), o.run(rows, 0, 0))
        same_state(s, o, tag=f"rows {c0}")
    assert (wide_rows(native, s) > 0) == wide
