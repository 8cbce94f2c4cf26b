"""Label propagation over rows that start, end and cross at the edges of chunks (8 or 32 in-edges), stretches
(8 to 128) and tiles (64 to 1024), both result buffers, seeds without in-edges, no edges at all.

Weights and start values are not negative, so a row's sum is off by at most its additions in sequence:
128 in a stretch, 3 over a tile's stretches, a row's tiles in eighths (20000 / 64 / 8 = 40) and 3 more,
and each iteration multiplies and adds once more.  Per entry: (150 k) 2^-24 of the FP64 value after k
iterations, and 1e-38 for what lies below the normal range."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _graph(lengths, base, seed, extra=0):
    """Rows of the given in-degrees, then ``extra`` random edges."""
    rng = np.random.default_rng(seed)
    V = base + len(lengths) + 5
    dst = np.repeat(np.arange(base, base + len(lengths)), lengths)
    src = rng.integers(0, V, len(dst))
    src = np.concatenate([src, rng.integers(0, V, extra)])
    dst = np.concatenate([dst, rng.integers(0, V, extra)])
    order = np.argsort(src, kind="stable")
    vl = np.zeros(V + 1, np.int32)
    np.cumsum(np.bincount(src, minlength=V), out=vl[1:])
    w = rng.random(len(src)).astype(np.float32)
    return vl, dst[order].astype(np.int32), w


def _check(csr, seed, iterations=(3,)):
    import c2g
    import oracle

    V = len(csr[0]) - 1
    rng = np.random.default_rng(seed)
    pp = rng.dirichlet((1.0, 1.0, 1.0), size=V).astype(np.float32)
    indeg = np.bincount(csr[1], minlength=V)
    seeds = rng.integers(0, V, 16).astype(np.int32)
    seeds[0] = int(np.argmin(indeg))   # no in-edges
    seeds[1] = seeds[0]
    seeds[2] = int(np.argmax(indeg))
    with c2g.Graph.create(csr[0], csr[1], flist=csr[2]) as g:
        for k in iterations:
            Y, st = g.adsorption(seeds, pp[:, 0], pp[:, 1], pp[:, 2], iterations=k)
            ref = oracle.adsorption_labels(*csr, seeds, pp[:, 0], pp[:, 1], k)
            assert (np.abs(Y - ref) <= 150 * k * 2.0**-24 * ref + 1e-38).all(), k
            assert st.iterations == k and st.edges_relaxed == k * len(csr[1])


@pytest.mark.parametrize("n", [1, 2, 7, 8, 9, 31, 32, 33, 63, 64, 255, 256, 257, 511, 512, 513, 1023, 1024, 1025, 5000])
def test_edge_counts_around_a_tile(gpu_available, n):
    _check(_graph([3, n, 1], 9, n), n)


@pytest.mark.parametrize("lengths", [
    [32] * 40, [31, 33] * 40, [1] * 700, [256] * 9, [255, 257] * 5, [20000], [7, 20000, 9, 300, 0, 0, 1],
    [100, 156, 768, 1024, 1, 1023, 0, 2048]])
def test_rows_across_tiles(gpu_available, lengths):
    _check(_graph(lengths, 50, len(lengths)), 3, (0, 1, 2, 3, 10, 3))


@pytest.mark.parametrize("extra", [500000, 3000000, 9000000])
def test_longer_stretches(gpu_available, extra):
    """Graphs large enough for the longer stretches, with rows of many tiles among the short ones."""
    rng = np.random.default_rng(extra)
    _check(_graph(list(rng.integers(0, 9, 30000)) + [20000, 5000, 1024], 60000, 7, extra), 5, (1, 4))


def test_no_edges(gpu_available):
    csr = (np.zeros(41, np.int32), np.zeros(0, np.int32), np.zeros(0, np.float32))
    _check(csr, 2, (0, 1, 2, 3))
