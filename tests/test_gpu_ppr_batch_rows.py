"""Pull rounds of the batched push over chunks of 32 in-edges: rows that start, end and cross at chunk
and item boundaries, edge counts around a chunk, every number of query words, both item sizes.

Tolerance: L1 1e-6 per query for pr and res, the bar of the other batched push tests."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _csr(V, src, dst, w):
    order = np.lexsort((dst, src))
    src, dst, w = src[order], dst[order], w[order]
    vl = np.zeros(V + 1, np.int32)
    np.cumsum(np.bincount(src, minlength=V), out=vl[1:])
    return vl, dst.astype(np.int32), w.astype(np.float32)


def _rows_graph(lengths, base, seed, extra):
    rng = np.random.default_rng(seed)
    V = base + len(lengths) + 3
    src, dst = [np.arange(base)], [(np.arange(base) * 7 + 1) % base]
    for k, n in enumerate(lengths):
        src.append(rng.choice(base, n, replace=False))
        dst.append(np.full(n, base + k))
    src.append(rng.integers(base, base + len(lengths), extra))
    dst.append(rng.integers(0, V, extra))
    src, dst = np.concatenate(src), np.concatenate(dst)
    w = rng.random(len(src)) + 0.01
    w /= np.bincount(src, weights=w, minlength=V)[src]
    return _csr(V, src, dst, w)


def _check(csr, n, seed):
    import c2g
    import oracle

    V = len(csr[0]) - 1
    src = np.random.default_rng(seed).integers(0, V, n).astype(np.int32)
    with c2g.Graph.create(csr[0], csr[1], flist=csr[2]) as g:
        prm = g.ppr_params(alpha=0.15, rmax=1e-7, seeded=0, pr0=0.15, r0=1.0, max_iter=500)
        for ratio in (None, 0.0, 4.0):  # None: the library's own
            if ratio is not None:
                g.ppr_batch_pull(ratio)
            pr, res, st = g.ppr_batch(src, prm)
            assert st.status_flags == 0
            for i in range(0, n, max(1, n // 12)):
                rp, rr, _, _ = oracle.ppr_push(*csr, int(src[i]), 0.15, 1e-7)
                assert np.abs(pr[i].astype(np.float64) - rp).sum() <= 1e-6, (n, ratio, i)
                assert np.abs(res[i].astype(np.float64) - rr).sum() <= 1e-6, (n, ratio, i)


@pytest.mark.parametrize("n", [1, 2, 8, 9, 16, 17, 31, 32, 33, 64, 65, 200])
def test_rows_across_chunks(gpu_available, n):
    lengths = [1, 31, 32, 33, 63, 64, 65, 1, 1, 1, 255, 256, 257, 30, 2, 500] * 2 + [1] * 70
    _check(_rows_graph(lengths, 600, n, 700), n, n)


@pytest.mark.parametrize("extra", [0, 1, 2, 3, 30, 31, 32, 33])
def test_edge_counts_around_a_chunk(gpu_available, extra):
    _check(_rows_graph([5, 9, 16], 34, extra, extra), 40, extra)


def test_items_of_eight_chunks(gpu_available):
    """A graph large enough for whole items, with rows longer than an item."""
    rng = np.random.default_rng(4)
    lengths = list(rng.integers(1, 60, 3000)) + [4000, 2500, 300, 257] + list(rng.integers(1, 9, 20000))
    _check(_rows_graph(lengths, 60000, 9, 2400000), 70, 5)
