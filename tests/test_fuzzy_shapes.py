"""The fuzzy set's per-row bisection at the list widths where its lanes change
(16 / 17, the widest 32, the narrowest) and on rows without any positive
distance, whose sigma is a share of the global mean.  Bit for bit against the
oracle."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,k,euclid,zero_rows", [
    (5, 1, 1, 0), (70, 2, 1, 3), (333, 3, 0, 5), (1000, 15, 1, 40), (1001, 16, 0, 0), (1000, 17, 1, 7),
    (700, 32, 0, 700), (3000, 30, 1, 1),
])
def test_fuzzy_schedule_bitexact(native, oracle_mod, n, k, euclid, zero_rows):
    import torch

    rng = np.random.default_rng(n + k)
    # tables with a wide spread of scales, ties, zeros and missing neighbours
    d = np.sort(rng.gamma(0.5, 1.0, size=(n, k)) * 10.0 ** rng.uniform(-6, 4, size=(n, 1)), axis=1).astype(np.float32)
    d[rng.random((n, k)) < 0.05] = 0.0
    d = np.sort(d, axis=1)
    idx = np.stack([(i + 1 + rng.permutation(max(n - 1, k))[:k]) % n for i in range(n)]).astype(np.uint32)
    missing = rng.random((n, k)) < 0.02
    idx[missing], d[missing] = 0xFFFFFFFF, np.finfo(np.float32).max
    z = rng.choice(n, zero_rows, replace=False)
    d[z] = 0.0
    pidx, pdst = np.zeros((n, k + 1), np.uint32), np.zeros((n, k + 1), np.float32)
    pidx[:, :k], pdst[:, :k], pidx[:, k] = idx, d, 1
    batch = np.sort(rng.choice(n, max(1, n // 3), replace=False)).astype(np.int32)
    ref = oracle_mod.fuzzy_schedule(pidx, pdst, k, bool(euclid), batch, n_epochs=100, alpha=1.0)
    dev = torch.device("cuda:0")
    t_idx, t_dst, t_b = (torch.from_numpy(a).to(dev) for a in (pidx.view(np.int32), pdst, batch))
    cap = 2 * len(batch) * k
    ints, vals = torch.zeros(4, cap, dtype=torch.int32, device=dev), torch.zeros(2, cap, device=dev)
    rows = torch.zeros(2, n, device=dev)
    counts, scal = (C.c_int64 * 4)(), (C.c_float * 3)()
    native.check(native.load().gm_op_fuzzy_schedule(
        t_idx.data_ptr(), t_dst.data_ptr(), n, k, euclid, t_b.data_ptr(), len(batch), 100, 1.0, ints[0].data_ptr(),
        ints[1].data_ptr(), vals[0].data_ptr(), ints[2].data_ptr(), ints[3].data_ptr(), vals[1].data_ptr(),
        rows[0].data_ptr(), rows[1].data_ptr(), counts, scal, C.c_void_p(torch.cuda.current_stream().cuda_stream)))
    assert np.array_equal(rows[1].cpu().numpy(), ref["rho"])
    assert np.array_equal(rows[0].cpu().numpy(), ref["sigma"])
    assert (counts[0], counts[1], counts[2], counts[3]) == (ref["nnz"], ref["extras"], ref["nnz2"], ref["max_deg"])
    assert scal[0] == np.float32(ref["mean"]) and scal[1] == np.float32(ref["max_w"])
    nnz, left = counts[0], counts[2]
    for t, key, m in ((ints[0], "coo_row", nnz), (ints[1], "coo_col", nnz), (vals[0], "coo_val", nnz),
                      (ints[2], "t_row", left), (ints[3], "t_col", left), (vals[1], "t_eps", left)):
        assert np.array_equal(t[:m].cpu().numpy(), ref[key]), key


# rows whose bisection has no root or a far one (terms that never reach the
# target, ties that always exceed it, a tail over many scales): where the sum
# is known without forming it, and where it is not
@pytest.mark.parametrize("k", [3, 15, 30])
def test_fuzzy_bisection_extremes(native, oracle_mod, k):
    import torch

    rng = np.random.default_rng(k)
    n = 512
    d = np.empty((n, k), np.float32)
    for i in range(n):
        kind = i % 8
        if kind == 0:
            v = np.full(k, 10.0 ** rng.uniform(-30, 30))  # all equal: every term 1
        elif kind == 1:
            v = 10.0 ** np.linspace(-35, 35, k)  # one scale a term
        elif kind == 2:
            v = np.where(np.arange(k) < k // 2, 1.0, 1e30)
        elif kind == 3:
            v = 1.0 + np.arange(k) * 1e-7  # differences of a rounding step
        elif kind == 4:
            v = np.full(k, 1e-38) * (1 + np.arange(k))  # at the smallest normals
        elif kind == 5:
            v = np.full(k, np.finfo(np.float32).max)  # no valid neighbour but one
            v[0] = 1.0
        elif kind == 6:
            v = 1.0 + rng.gamma(0.05, 1.0, k)  # most terms near 1, a few far
        else:
            v = 10.0 ** rng.uniform(-8, 8) * (5.0 + rng.random(k))
        d[i] = np.sort(v)
    idx = np.stack([(i + 1 + np.arange(k)) % n for i in range(n)]).astype(np.uint32)
    pidx, pdst = np.zeros((n, k + 1), np.uint32), np.zeros((n, k + 1), np.float32)
    pidx[:, :k], pdst[:, :k], pidx[:, k] = idx, d, 1
    batch = np.arange(n, dtype=np.int32)
    dev = torch.device("cuda:0")
    t_idx, t_dst, t_b = (torch.from_numpy(a).to(dev) for a in (pidx.view(np.int32), pdst, batch))
    cap = 2 * n * k
    for euclid in (0, 1):
        ref = oracle_mod.fuzzy_schedule(pidx, pdst, k, bool(euclid), batch, n_epochs=100, alpha=1.0)
        ints, vals = torch.zeros(4, cap, dtype=torch.int32, device=dev), torch.zeros(2, cap, device=dev)
        rows = torch.zeros(2, n, device=dev)
        counts, scal = (C.c_int64 * 4)(), (C.c_float * 3)()
        native.check(native.load().gm_op_fuzzy_schedule(
            t_idx.data_ptr(), t_dst.data_ptr(), n, k, euclid, t_b.data_ptr(), n, 100, 1.0, ints[0].data_ptr(),
            ints[1].data_ptr(), vals[0].data_ptr(), ints[2].data_ptr(), ints[3].data_ptr(), vals[1].data_ptr(),
            rows[0].data_ptr(), rows[1].data_ptr(), counts, scal,
            C.c_void_p(torch.cuda.current_stream().cuda_stream)))
        assert np.array_equal(rows[1].cpu().numpy(), ref["rho"])
        assert np.array_equal(rows[0].cpu().numpy(), ref["sigma"])
        assert (counts[0], counts[2], counts[3]) == (ref["nnz"], ref["nnz2"], ref["max_deg"])
