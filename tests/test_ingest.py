"""Host rows into a session: unaligned arrays, row widths that are not multiples
of four floats, buffers overwritten as soon as append returns, pinned and
pageable memory.  The feature matrix is compared byte for byte."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,pinned,offset", [(1, False, 0), (3, False, 1), (64, False, 0), (64, False, 1),
                                             (131, False, 0), (131, True, 0), (784, False, 3), (784, True, 0)])
def test_append_host_rows(native, d, pinned, offset):
    import torch

    sizes = [1, 7, 500, 2000]
    n, ld = sum(sizes), (d + 3) // 4 * 4
    s = native.Session(native.default_params(n_instances=n, n_features=d, device=0))
    rng = np.random.default_rng(d)
    want, c0 = np.zeros((n, ld), np.float32), 0
    flat = torch.empty(max(sizes) * d + 8, pin_memory=pinned).numpy()
    for m in sizes:
        buf = flat[offset : offset + m * d].reshape(m, d)
        buf[:] = rng.normal(size=(m, d)).astype(np.float32)
        want[c0 : c0 + m, :d] = buf
        s.append_host(buf)
        buf[:] = np.nan  # the caller's buffer again
        c0 += m
    assert np.array_equal(s.copy("x", np.float32).reshape(n, ld), want)
