"""Allocations that fail (reported by the library's own hook, on the host): a
session that cannot be built leaves nothing behind, one that cannot grow keeps
what it had and frees each buffer once, so that memory of other sessions stays
theirs."""
import numpy as np
import pytest

from gpumap_gb300.datasets import gaussian_mixture

pytestmark = pytest.mark.gpu


def tables(s):
    return [s.copy(b, t) for b, t in (("pub_idx", np.uint32), ("pub_dist", np.float32), ("sigma", np.float32),
                                      ("sched_row", np.int32), ("sched_eps", np.float32))]


def same(a, b):
    return all(np.array_equal(x, y) for x, y in zip(a, b))


def build(native, X, k=15, precision=0, emb=0):
    n, d = X.shape
    s = native.Session(native.default_params(n_instances=n, n_features=d, n_neighbors=k, max_epoch=5, device=0,
                                             precision=precision))
    s.append_host(X)
    s.run(n, 0, emb)
    return s


@pytest.mark.parametrize("precision,overlap", [(0, 0), (1, 1)])
def test_failed_create_leaves_nothing(native, precision, overlap):
    lib = native.load()
    native.release_memory()
    _, used0 = native.memory_held(0)
    p = native.default_params(n_instances=2000, n_features=9, device=0, precision=precision, overlap=overlap)
    made = 0
    for nth in range(1, 200):
        lib.gm_debug_fail_alloc(nth)
        try:
            native.Session(p)
            made = nth
            break
        except MemoryError:
            assert native.memory_held(0)[1] == used0
        finally:
            lib.gm_debug_fail_alloc(0)
    assert made > 40  # every allocation of a session has failed once
    assert native.memory_held(0)[1] == used0


@pytest.mark.parametrize("nth", range(1, 11))
def test_failed_embedding_growth(native, nth):
    lib = native.load()
    X, _ = gaussian_mixture(3000, 12, seed=3)
    Y, _ = gaussian_mixture(2500, 7, seed=4)
    want = tables(build(native, X, emb=3000))
    a = build(native, X, emb=0)  # scratch for a small batch
    other = build(native, Y, precision=1, emb=2500)
    mine = tables(other)
    _, used = native.memory_held(0)
    lib.gm_debug_fail_alloc(nth)
    with pytest.raises(MemoryError):
        a.run(0, 0, 3000)
    lib.gm_debug_fail_alloc(0)
    assert native.memory_held(0)[1] <= used  # nothing half made is held
    third = build(native, Y, emb=2500)  # may take what was freed
    theirs = tables(third)
    a.run(0, 0, 3000)  # grows now
    assert same(tables(a), want)
    assert same(tables(other), mine) and same(tables(third), theirs)
    del a
    fourth = build(native, X, emb=3000)
    assert same(tables(fourth), want) and same(tables(other), mine) and same(tables(third), theirs)


@pytest.mark.parametrize("k", [15, 30])
def test_failed_insertion_growth(native, k):
    lib = native.load()
    X, _ = gaussian_mixture(4000, 12, seed=5)
    n, d = X.shape
    for nth in range(1, 5):
        s = native.Session(native.default_params(n_instances=n, n_features=d, n_neighbors=k, max_epoch=5, device=0))
        s.append_host(X)
        s.run(500, 0, 0)
        _, used = native.memory_held(0)
        lib.gm_debug_fail_alloc(nth)
        with pytest.raises(MemoryError):
            s.run(2000, 0, 0)
        lib.gm_debug_fail_alloc(0)
        assert native.memory_held(0)[1] <= used
        r = s.run(1500, 0, 0)
        assert r.n_insertion_ops == 1500


@pytest.mark.parametrize("failures", [1, 3])
def test_update_with_a_smaller_pool(native, oracle_mod, failures):
    # the join pool of the whole round cannot be had: more passes, the same lists
    from test_gpu_parity import pair, same_result, same_state

    X, _ = gaussian_mixture(2000, 20, seed=6)
    s, o = pair(native, oracle_mod, 2000, 20, k=15, max_epoch=5)
    s.append_host(X)
    o.append(X)
    same_result(s.run(2000, 0, 0), o.run(2000, 0, 0))
    native.load().gm_debug_fail_alloc(-failures)
    same_result(s.run(0, 2000, 0), o.run(0, 2000, 0))
    native.load().gm_debug_fail_alloc(0)
    same_state(s, o, tag="smaller pool")
    same_result(s.run(0, 900, 0), o.run(0, 900, 0))
    same_state(s, o, tag="after it")
