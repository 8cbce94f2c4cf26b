"""Pull rounds of the batched SSSP over in-edge rows ordered by weight: rows at the edges of a
group, an item and a segment; every form of the kernel (1, 2, 4 and more query words, more slots
than tracked minima); queries that reach nothing; the sizes on both sides of the default rule."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _csr(V, src, dst, w):
    order = np.lexsort((dst, src))
    src, dst, w = src[order], dst[order], w[order]
    vl = np.zeros(V + 1, np.int32)
    np.cumsum(np.bincount(src, minlength=V), out=vl[1:])
    return vl, dst.astype(np.int32), w.astype(np.int32)


@pytest.fixture(scope="module")
def rows_graph():
    rng = np.random.default_rng(5)
    lengths = [0, 1, 3, 4, 5, 8, 9, 16, 31, 32, 33, 36, 63, 64, 65, 287, 288, 289, 545, 1500]
    V, base = 3007, 2800
    src, dst = [np.arange(base - 1)], [np.arange(1, base)]  # a chain reaches every source
    for k, n in enumerate(lengths):
        for copy in range(3):
            src.append(rng.choice(base, n, replace=False))
            dst.append(np.full(n, base + 3 * k + copy))
    tail = base + 3 * len(lengths)
    src.append(rng.integers(base, tail, 600))
    dst.append(rng.integers(0, V - 5, 600))  # back into the chain, and beyond; 5 vertices stay unreached
    src, dst = np.concatenate(src), np.concatenate(dst)
    w = rng.integers(0, 5001, len(src))
    return _csr(V, src, dst, w)


@pytest.mark.parametrize("n", [1, 33, 65, 130, 1100])
def test_batch_rows_of_every_length(gpu_available, rows_graph, n):
    import c2g
    import oracle

    vl, el, wl = rows_graph
    rng = np.random.default_rng(n)
    src = rng.integers(0, len(vl) - 1, n).astype(np.int32)
    src[0] = len(vl) - 2  # reaches nothing
    with c2g.Graph.create(vl, el, wl) as g:
        for frac in (0.0, 0.2):
            g.sssp_batch_pull(frac)
            dist, st = g.sssp_batch(src)
            assert st.status_flags == 0
            for i in range(0, n, max(1, n // 40)):
                ref = oracle.dijkstra(vl, el, wl, [int(src[i])], [0])
                assert np.array_equal(dist[i], ref), (n, frac, i)


@pytest.mark.parametrize("V,n", [(130001, 256), (120001, 256), (500009, 64)])
def test_batch_default_rule(gpu_available, V, n):
    """Default rule above and below a million (vertex, word) lines, hubs in both directions."""
    import c2g
    import oracle

    rng = np.random.default_rng(V)
    M = 8 * V
    src, dst = rng.integers(0, V, M), rng.integers(0, V, M)
    dst[: M // 8] = V // 3
    src[M // 8: M // 4] = V // 2
    key = np.unique((src.astype(np.int64) * V + dst)[src != dst])
    vl, el, wl = _csr(V, key // V, key % V, rng.integers(1, 1001, len(key)))
    q = rng.integers(0, V, n).astype(np.int32)
    with c2g.Graph.create(vl, el, wl) as g:
        dist, st = g.sssp_batch(q)
        assert st.status_flags == 0
        _, _, shape = g.last_rounds()
        assert bool(shape.max()) == (V * ((n + 31) // 32) >= 1000000)
        for i in range(0, n, n // 8):
            assert np.array_equal(dist[i], oracle.dijkstra(vl, el, wl, [int(q[i])], [0])), i


def test_batch_negative_weights_expand(gpu_available):
    """A weight below zero (no negative cycle): the batch expands, pull fraction or not."""
    import c2g

    V = 50
    w = np.full(V - 1, 2)
    w[7] = -5
    vl, el, wl = _csr(V, np.arange(V - 1), np.arange(1, V), w)
    with c2g.Graph.create(vl, el, wl) as g:
        g.sssp_batch_pull(0.0)
        dist, st = g.sssp_batch([0, 3])
        ref = np.concatenate([[0], np.cumsum(w)])
        assert st.status_flags == 0 and np.array_equal(dist[0], ref)
        _, _, shape = g.last_rounds()
        assert not shape.any()
