"""Pull rounds of the single-query push: rows of every length class and at its edges, rows in segments,
sources and targets without edges, weights that send nothing, residuals that outgrow the float pairs,
the round cap, and mixes of pull and push rounds, against the FP64 push.

Tolerance: L1 1e-6 of the mass in the graph, the bar of the other push tests (pr is FP32: its
rounding alone is 2^-24 of the mass)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _csr(V, src, dst, w):
    order = np.lexsort((dst, src))
    src, dst, w = src[order], dst[order], w[order]
    vl = np.zeros(V + 1, np.int32)
    np.cumsum(np.bincount(src, minlength=V), out=vl[1:])
    return vl, dst.astype(np.int32), w.astype(np.float32)


def _rows_graph(seed, scale=1.0):
    """Targets with 1, 2, ... 1300 in-edges, two of each; every vertex has out-edges but a few."""
    rng = np.random.default_rng(seed)
    lengths = [1, 2, 7, 8, 9, 15, 16, 17, 31, 32, 33, 63, 64, 65, 127, 128, 129, 255, 256, 257, 511, 512, 513, 1300]
    V, base = 2048 + 5, 1400
    src, dst = [np.arange(base)], [(np.arange(base) + 1) % base]
    for k, n in enumerate(lengths):
        for copy in range(2):
            src.append(rng.choice(base, n, replace=False))
            dst.append(np.full(n, base + 2 * k + copy))
    tail = base + 2 * len(lengths)
    src.append(rng.integers(base, tail, 900))
    dst.append(rng.integers(0, V, 900))  # back into the graph; some vertices have no out-edges
    src, dst = np.concatenate(src), np.concatenate(dst)
    w = rng.random(len(src)) + 0.01
    w /= np.bincount(src, weights=w, minlength=V)[src]
    return _csr(V, src, dst, w * scale)


def _compare(g, csr, s, alpha, rmax, tol=1e-6, **kw):
    import oracle

    prm = g.ppr_params(alpha=alpha, rmax=rmax, seeded=0, pr0=alpha, r0=1.0, max_iter=kw.get("max_iter", 500))
    pr, res, st = g.ppr(s, prm)
    rp, rr, rounds, _ = oracle.ppr_push(*csr, s, alpha, rmax, **kw)
    for got, want in ((pr, rp), (res, rr)):
        fits = np.abs(want) < 3e38  # a value beyond FP32 comes back as infinity
        assert np.all(np.isinf(got[np.abs(want) > 3.5e38]))
        off = np.abs(got[fits].astype(np.float64) - want[fits]).sum()
        scale = max(1.0, float(np.abs(want[fits]).sum()))
        assert off <= tol * scale, (s, off, scale)
    return st, rounds


@pytest.mark.parametrize("pull_div", [None, 1 << 30, 3, 1])
@pytest.mark.parametrize("rmax", [1e-7, 3e-5])
def test_rows_of_every_length(gpu_available, pull_div, rmax):
    import c2g

    csr = _rows_graph(7)
    deg, indeg = np.diff(csr[0]), np.bincount(csr[1], minlength=len(csr[0]) - 1)
    sources = [0, 700, 1400 + 47, int(np.flatnonzero(deg == 0)[0])]
    sources += [int(v) for v in np.flatnonzero(indeg == 0)[:2]]
    with c2g.Graph.create(csr[0], csr[1], flist=csr[2]) as g:
        if pull_div is not None:
            g.ppr_config(pull_div=pull_div)
        for s in sources:
            st, rounds = _compare(g, csr, s, 0.15, rmax)
            assert st.status_flags == 0 and abs(st.iterations - rounds) <= 2


@pytest.mark.parametrize("cap", [1, 2, 3, 6])
@pytest.mark.parametrize("pull_div", [None, 4])
def test_round_cap(gpu_available, cap, pull_div):
    import c2g

    csr = _rows_graph(11)
    with c2g.Graph.create(csr[0], csr[1], flist=csr[2]) as g:
        if pull_div is not None:
            g.ppr_config(pull_div=pull_div)
        for s in (3, 1400 + 46):
            st, _ = _compare(g, csr, s, 0.2, 1e-9, max_iter=cap)
            assert st.status_flags & c2g.FLAG_ITER_CAP and st.iterations == cap + 1


def test_weights_that_send_nothing(gpu_available):
    """Zero, negative and subnormal weights among the rows: a push sends only positive messages, so
    the expected result is that of the graph with the negative weights at zero."""
    import c2g

    vl, el, w = _rows_graph(13)
    rng = np.random.default_rng(1)
    w[rng.random(len(w)) < 0.1] = 0.0
    w[rng.random(len(w)) < 0.1] *= -1.0
    w[rng.random(len(w)) < 0.02] = np.float32(1e-40)
    with c2g.Graph.create(vl, el, flist=w) as g:
        _compare(g, (vl, el, np.maximum(w, 0)), 5, 0.15, 1e-7)
        g.ppr_config(pull_div=0)
        _compare(g, (vl, el, np.maximum(w, 0)), 5, 0.15, 1e-7)


def test_growing_residuals_leave_the_pull(gpu_available):
    """Weights that multiply the mass every round: past 2^60 the rounds push in FP64."""
    import c2g

    csr = _rows_graph(17, scale=4000.0)
    with c2g.Graph.create(csr[0], csr[1], flist=csr[2]) as g:
        _compare(g, csr, 0, 0.15, 1e-7, tol=1e-5, max_iter=12)


def test_set_weights_reach_the_pull(gpu_available):
    import c2g

    csr = _rows_graph(19)
    rng = np.random.default_rng(2)
    with c2g.Graph.create(csr[0], csr[1], flist=csr[2]) as g:
        _compare(g, csr, 9, 0.15, 1e-6)
        w = (csr[2] * rng.random(len(csr[2]))).astype(np.float32)
        g.set_weights(w)
        _compare(g, (csr[0], csr[1], w), 9, 0.15, 1e-6)


def test_pull_and_push_rounds_mixed(gpu_available):
    """A graph above the size where every round pulls: dense rounds pull, sparse ones push."""
    import c2g

    rng = np.random.default_rng(3)
    V, M = 300007, 16 * 300007
    src, dst = rng.integers(0, V, M), rng.integers(0, V, M)
    dst[: M // 10] = V // 3
    src[M // 10: M // 5] = V // 2
    key = np.unique(src.astype(np.int64) * V + dst)
    src, dst = key // V, key % V
    w = rng.random(len(key)) + 0.01
    w /= np.bincount(src, weights=w, minlength=V)[src]
    csr = _csr(V, src, dst, w)
    assert len(csr[1]) > 4000000
    with c2g.Graph.create(csr[0], csr[1], flist=csr[2]) as g:
        for s in (V // 2, 12):
            st, rounds = _compare(g, csr, s, 0.15, 1e-7)
            assert st.status_flags == 0 and abs(st.iterations - rounds) <= 2
