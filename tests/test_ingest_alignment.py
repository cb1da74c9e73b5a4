"""Host rows at any byte address: which way they take (a host decision, no
GPU), and that rows at odd addresses arrive byte for byte."""
import numpy as np
import pytest

COPY, IN_PLACE, STAGED = 0, 1, 2


@pytest.mark.parametrize("offset", range(16))
def test_route_by_address(native, offset):
    route = native.load().gm_debug_ingest_route
    base = 1 << 20
    assert route(base + offset, 0, 1) == (STAGED if offset % 4 else IN_PLACE)
    assert route(base + offset, 0, 0) == STAGED
    assert route(base + offset, 1, 1) == route(base + offset, 1, 0) == COPY


def test_route_of_arrays_that_numpy_leaves_unaligned(native):
    # the array a caller hands in is passed on as it is: contiguous, not aligned
    raw = bytearray(4 * 64 + 8)
    start = -np.frombuffer(raw, np.uint8).ctypes.data % 4
    for shift in (0, 1, 2, 3):
        a = np.frombuffer(raw, np.float32, 64, offset=start + shift)
        assert np.ascontiguousarray(a, dtype=np.float32).ctypes.data == a.ctypes.data
        want = STAGED if shift else IN_PLACE
        assert native.load().gm_debug_ingest_route(a.ctypes.data, 0, 1) == want


@pytest.mark.gpu
@pytest.mark.parametrize("d", [1, 5, 64, 131])
@pytest.mark.parametrize("shift", [1, 2, 3])
def test_append_rows_at_odd_addresses(native, d, shift):
    sizes = [1, 7, 500, 2000]
    n, ld = sum(sizes), (d + 3) // 4 * 4
    s = native.Session(native.default_params(n_instances=n, n_features=d, device=0))
    rng = np.random.default_rng(d + shift)
    want, c0 = np.zeros((n, ld), np.float32), 0
    raw = np.zeros(max(sizes) * d * 4 + 64, np.uint8)
    start = -raw.ctypes.data % 16 + shift
    for m in sizes:
        buf = np.frombuffer(raw.data, np.float32, m * d, offset=start).reshape(m, d)
        assert buf.ctypes.data % 4 == shift and not buf.flags.aligned
        rows = rng.normal(size=(m, d)).astype(np.float32)
        buf[:] = rows
        want[c0 : c0 + m, :d] = rows
        s.append_host(buf)
        buf[:] = np.nan  # the caller's buffer again
        c0 += m
    assert np.array_equal(s.copy("x", np.float32).reshape(n, ld), want)
