"""Pull rounds of the single-query SSSP: in-edge rows ordered by weight, read only as far as an
edge can still improve the vertex.  Rows at the edges of a group, a warp and the split over the
grid; both round rules; weights at the limit the rows serve and beyond it; seeds below zero."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _csr(V, src, dst, w):
    order = np.lexsort((dst, src))
    src, dst, w = src[order], dst[order], w[order]
    vl = np.zeros(V + 1, np.int32)
    np.cumsum(np.bincount(src, minlength=V), out=vl[1:])
    return vl, dst.astype(np.int32), w.astype(np.int32)


def _check(vl, el, wl, sources):
    import c2g
    import oracle

    with c2g.Graph.create(vl, el, wl) as g:
        for s in sources:
            ref = oracle.dijkstra(vl, el, wl, [int(s)], [0])
            dist, st = g.sssp(int(s))
            assert st.status_flags == 0
            assert np.array_equal(dist, ref), int(s)


# in-degrees around 4 (a group), 8 (what a lane reads), 32 (the row sort's two forms), 72 (what a
# warp reads: 2 + 16 groups of 4) and far beyond (rows split over the grid)
@pytest.mark.parametrize("wmax", [1, 100, 5000, 147483648])
def test_rows_of_every_length(gpu_available, wmax):
    rng = np.random.default_rng(wmax)
    lengths = [0, 1, 2, 3, 4, 5, 7, 8, 9, 31, 32, 33, 63, 64, 65, 71, 72, 73, 76, 255, 257, 1000, 3001]
    V, base = 4000 + 13, 4000 - 200
    # targets base.. take in-edges from any lower vertex; a chain reaches the lower vertices
    src, dst = [np.arange(base - 1)], [np.arange(1, base)]
    for k, n in enumerate(lengths):
        for copy in range(3):
            src.append(rng.choice(base, n, replace=False))
            dst.append(np.full(n, base + 3 * k + copy))
    tail = base + 3 * len(lengths)
    src.append(rng.integers(base, tail, 400))
    dst.append(rng.integers(tail, V, 400))
    src, dst = np.concatenate(src), np.concatenate(dst)
    w = rng.integers(0, wmax + 1, len(src))
    w[: base - 1] = rng.integers(0, min(wmax, 50) + 1, base - 1)
    _check(*_csr(V, src, dst, w), [0, base - 30, 17])


@pytest.mark.parametrize("V,ef,wmax", [(1, 0, 1), (33, 3, 10), (4097, 8, 1000), (299999, 9, 100), (310001, 9, 100),
                                       (400003, 12, 1000)])
def test_round_rules_vs_dijkstra(gpu_available, V, ef, wmax):
    """Below and above the sizes where every round pulls; a hub that most vertices point to and
    one that points to most."""
    rng = np.random.default_rng(V)
    M = V * ef
    src, dst = rng.integers(0, V, M), rng.integers(0, V, M)
    if M:
        dst[: M // 4] = V // 3
        src[M // 4: M // 2] = V // 2
    keep = src != dst
    key = np.unique(src[keep].astype(np.int64) * V + dst[keep])
    src, dst = key // V, key % V
    vl, el, wl = _csr(V, src, dst, rng.integers(1, wmax + 1, len(src)))
    _check(vl, el, wl, [0, V // 2, V - 1])


@pytest.mark.parametrize("lo,hi", [(147483649, 147483649), (-3, 2)])
def test_weights_the_rows_do_not_serve(gpu_available, lo, hi):
    """Weights above the limit, and below zero (without a negative cycle): push rounds only."""
    import c2g

    V = 40
    src, dst = np.arange(V - 1), np.arange(1, V)
    w = np.full(V - 1, 1)
    w[5], w[20] = lo, hi
    vl, el, wl = _csr(V, src, dst, w)
    ref = np.concatenate([[0], np.cumsum(w)]).astype(np.int64)
    with c2g.Graph.create(vl, el, wl) as g:
        dist, st = g.sssp(0)
        assert st.status_flags == 0 and np.array_equal(dist, ref)


def test_negative_record_weights(gpu_available):
    """Record seeds below zero (the pull rounds' bound assumes none): the source's distances
    follow the seeds."""
    import c2g

    vl = np.array([0, 1, 2, 3, 3], np.int32)
    el = np.array([1, 2, 3], np.int32)
    wl = np.array([10, 10, 10], np.int32)
    with c2g.Graph.create(vl, el, wl) as g:
        g.set_records(np.array([0, 1], np.int32), np.array([2], np.int32), np.array([-7], np.int32),
                      record_vertex=np.array([0], np.int32))
        dist, _ = g.sssp(0, seeds=True, mode=c2g.SEEDS_EXACT)
        assert dist.tolist() == [0, 10, -7, 3]
