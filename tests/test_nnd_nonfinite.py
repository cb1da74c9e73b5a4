"""NN-Descent (precision 0) with NaN rows: the lists' insertion sorts compare
with a NaN as sequential code does, entry by entry.  Insertion against the oracle;
the update round's merge into the authoritative lists against its restatement
here."""
import numpy as np
import pytest

from gpumap_gb300.datasets import gaussian_mixture

pytestmark = pytest.mark.gpu

FLT_MAX = np.finfo(np.float32).max


def data(n, d, seed, share):
    X, _ = gaussian_mixture(n, d, seed=seed)
    rng = np.random.default_rng(seed)
    X[rng.choice(n, max(1, int(n * share)), replace=False), 0] = np.nan
    return X


@pytest.mark.parametrize("n,k,share", [(900, 20, 0.01), (900, 30, 0.05), (700, 32, 0.2)])
def test_insertion(native, oracle_mod, n, k, share):
    X = data(n, 12, n + k, share)
    s = native.Session(native.default_params(n_instances=n, n_features=12, n_neighbors=k, device=0))
    o = oracle_mod.OracleSession(n, 12, k=k)
    for t in (s, o):
        (t.append_host if t is s else t.append)(X)
        t.run(n, 0, 0)
    assert np.array_equal(s.copy("graph_ids", np.int32), o.copy("graph_ids", np.int32))
    assert np.array_equal(s.copy("graph_dists", np.float32), o.copy("graph_dists", np.float32), equal_nan=True)


def merged(ids, dists, graph_ids, graph_dists, n, row):
    """A row's list after update_graph (insert_to_ordered_list for each working
    entry); whether an entry came in."""
    k, came = len(ids), False
    for nid, nd in zip(graph_ids, graph_dists):
        if nd == FLT_MAX:
            break
        if not 0 <= nid < n or nid == row or nd > dists[k - 1]:
            continue
        if any((e if e >= 0 else -e - 1) == nid for e in ids):
            continue
        at = next((q for q in range(k) if dists[q] > nd), k)
        if at == k:
            continue
        ids[at + 1 :], dists[at + 1 :] = ids[at:-1], dists[at:-1]
        ids[at], dists[at] = nid, nd
        came = True
    return came


def insertion_sorted(ids, dists):
    for a in range(1, len(ids)):
        e, v, b = ids[a], dists[a], a
        while b > 0 and (dists[b - 1] > v or (dists[b - 1] == v and ids[b - 1] > e)):
            ids[b], dists[b] = ids[b - 1], dists[b - 1]
            b -= 1
        ids[b], dists[b] = e, v


@pytest.mark.parametrize("n,k,share", [(700, 32, 0.2), (900, 32, 0.4), (1200, 32, 0.05)])
def test_update_round(native, n, k, share):
    X = data(n, 12, n + k, share)
    s = native.Session(native.default_params(n_instances=n, n_features=12, n_neighbors=k, device=0))
    s.append_host(X)
    s.run(n, 0, 0)

    def lists():
        return [s.copy(b, t).reshape(n, -1).copy() for b, t in (
            ("knn_ids", np.int32), ("knn_dists", np.float32), ("graph_ids", np.int32), ("graph_dists", np.float32))]

    seen = 0
    for _ in range(4):
        ids, dists, g0, d0 = lists()
        seen += int(np.isnan(dists).any(1).sum())
        s.run(0, n, 0)  # one round over every row
        got_ids, got_dists, g1, d1 = lists()
        moved = (g0 != g1).any(1) | (d0.view(np.int32) != d1.view(np.int32)).any(1)
        ids = np.where((ids >= 0) & (ids < n), -ids - 1, ids)  # every new entry was sampled
        for row in range(n):
            i, v = list(ids[row].tolist()), list(dists[row])
            if merged(i, v, g1[row].tolist(), d1[row], n, row) or moved[row]:
                insertion_sorted(i, v)
            assert i == got_ids[row].tolist(), row
            assert np.array_equal(np.array(v, np.float32), got_dists[row], equal_nan=True), row
    assert seen > 0  # lists with NaN distances were merged and sorted
