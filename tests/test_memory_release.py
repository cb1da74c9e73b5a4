"""Device memory after sessions have gone: what is kept for the next one is
bounded, a call gives it back, and an allocation beyond what is free takes it."""
import numpy as np
import pytest

from gpumap_gb300.datasets import gaussian_mixture

MB = 1 << 20


def test_nothing_held_without_a_device(native):
    # (host bookkeeping only: no pool is made by asking)
    with pytest.raises(ValueError):
        native.memory_held(-1)
    with pytest.raises(ValueError):
        native.memory_held(64)
    import gpumap_gb300

    assert gpumap_gb300.release_memory is native.release_memory


def session(native, n, d=8, precision=1):
    return native.Session(native.default_params(n_instances=n, n_features=d, device=0, precision=precision))


def free_bytes():
    import torch

    torch.cuda.synchronize()
    return torch.cuda.mem_get_info(0)


@pytest.mark.gpu
def test_release_gives_everything_unused_back(native):
    X, _ = gaussian_mixture(3000, 8, seed=1)
    keep = session(native, 3000, precision=0)
    keep.append_host(X)
    keep.run(3000, 3000, 0)
    before = keep.copy("knn_ids", np.int32)
    for n in (20_000, 60_000, 40_000):
        del_me = session(native, n)
        del del_me
    reserved, used = native.memory_held(0)
    assert reserved - used > 100 * MB  # kept for the next session
    free0, _ = free_bytes()
    native.release_memory()
    r2, u2 = native.memory_held(0)
    free1, _ = free_bytes()
    assert u2 == used and r2 - u2 < 64 * MB and free1 - free0 > 100 * MB
    # live sessions keep theirs, and new ones come as before
    assert np.array_equal(keep.copy("knn_ids", np.int32), before)
    again = session(native, 20_000)
    again.append_host(X[:, :8])
    again.run(3000, 0, 0)


@pytest.mark.gpu
def test_a_large_session_is_given_back_beyond_the_share(native):
    native.release_memory()
    free0, total = free_bytes()
    big = session(native, 1_000_000)  # about 30 GB of exact scratch
    assert free0 - free_bytes()[0] > total // 16
    del big
    assert free0 - free_bytes()[0] <= total // 16 + 256 * MB
    # small sessions after it give the rest up
    for _ in range(20):
        small = session(native, 1000)
        del small
    assert free0 - free_bytes()[0] <= 512 * MB


@pytest.mark.gpu
def test_growth_takes_what_closed_sessions_left(native):
    # free device memory is used up to a rest that the new session fits only with
    # what the pool still holds
    import torch

    native.release_memory()
    first = session(native, 200_000)
    reserved, used = native.memory_held(0)
    del first
    kept = native.memory_held(0)[0] - native.memory_held(0)[1]
    assert kept > used // 2
    free, _ = free_bytes()
    block = torch.empty(free - (3 << 30), dtype=torch.uint8, device="cuda")  # 3 GB stay
    try:
        # more rows, so other block sizes: together no larger than what is kept and free
        second = session(native, 205_000)
        X = np.random.default_rng(0).normal(size=(2000, 8)).astype(np.float32)
        second.append_host(X)
        assert second.run(2000, 0, 2000).n_insertion_ops == 2000
    finally:
        del block
        torch.cuda.empty_cache()
