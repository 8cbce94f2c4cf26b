"""Single push whose residuals pass 2^60 on the way: the round after, every block leaves the pulls together and
the rounds push in FP64.  Weights that multiply the mass by 34 to 255,000 a round, so that the limit is passed
after few or many pulls; graphs of one row step per warp, of several, and above the size where every round pulls.

Tolerance: pr is FP32 and a vertex takes at most one rounding of 2^-24 per round, so L1 within rounds * 2^-24 of
the mass; the residuals are FP64 and come back rounded once."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _graph(V, ef, scale, seed):
    rng = np.random.default_rng(seed)
    key = np.unique(rng.integers(0, V, V * ef) * V + rng.integers(0, V, V * ef))
    src, dst = key // V, (key % V).astype(np.int32)
    vl = np.zeros(V + 1, np.int32)
    np.cumsum(np.bincount(src, minlength=V), out=vl[1:])
    w = rng.random(len(src)) + 0.01
    return vl, dst, (w * scale / np.bincount(src, weights=w, minlength=V)[src]).astype(np.float32)


@pytest.mark.parametrize("V,ef", [(3000, 8), (120000, 12), (400000, 11)])
@pytest.mark.parametrize("scale,cap", [(40.0, 18), (4000.0, 9), (3e5, 6)])
def test_all_blocks_leave_the_pulls_together(gpu_available, V, ef, scale, cap):
    import c2g
    import oracle

    vl, el, w = _graph(V, ef, scale, V + cap)
    rng = np.random.default_rng(cap)
    with c2g.Graph.create(vl, el, flist=w) as g:
        prm = g.ppr_params(alpha=0.15, rmax=1e-7, seeded=0, pr0=0.15, r0=1.0, max_iter=cap)
        for s in rng.choice(np.flatnonzero(np.diff(vl) > 0), 2):
            rp, rr, _, _ = oracle.ppr_push(vl, el, w, int(s), 0.15, 1e-7, max_iter=cap)
            assert np.abs(rr).max() > 2.0 ** 60  # passed on the way
            for _ in range(6):
                pr, res, st = g.ppr(int(s), prm)
                assert st.status_flags == c2g.FLAG_ITER_CAP
                for got, want in ((pr, rp), (res, rr)):
                    assert np.abs(got.astype(np.float64) - want).sum() <= cap * 2.0 ** -24 * np.abs(want).sum()


def _heavy_records():
    """Vertex 0 has 40 records of weight 3e38; their vertices send all to a hub (weight 1), the hub to 64 leaves
    (1/64), the leaves to one tail (1e-30): the hub's residual is beyond FP32, what comes after it is not."""
    n, hub = 40, 41
    leaf = np.arange(42, 106)
    src = np.concatenate([np.arange(1, n + 1), np.full(64, hub), leaf])
    dst = np.concatenate([np.full(n, hub), leaf, np.full(64, 106)]).astype(np.int32)
    w = np.concatenate([np.ones(n), np.full(64, 1 / 64), np.full(64, 1e-30)]).astype(np.float32)
    V = 107
    vl = np.zeros(V + 1, np.int32)
    np.cumsum(np.bincount(src, minlength=V), out=vl[1:])
    hv = np.full(V + 1, n, np.int32)
    hv[0] = 0
    return (vl, dst, w), (hv, np.arange(1, n + 1, dtype=np.int32), np.full(n, 3e38, np.float32))


def _check_heavy(got, want, rounds):
    fits = np.abs(want) < 3e38
    assert np.isinf(got[~fits]).all() and np.count_nonzero(~fits) <= 1
    assert np.all(np.abs(got[fits].astype(np.float64) - want[fits]) <= rounds * 2.0 ** -24 * np.abs(want[fits]))


def test_records_beyond_the_limit(gpu_available):
    """The first round's residuals are the records': a sum of them overflows FP32, not FP64."""
    import c2g
    import oracle

    csr, (hv, he, hw) = _heavy_records()
    with c2g.Graph.create(csr[0], csr[1], flist=csr[2]) as g:
        g.set_records(hv, he, hw)
        pr, res, st = g.ppr(0, g.ppr_params(alpha=0.15, rmax=1e-7, seeded=1, max_iter=500))
        rp, rr, rounds, _ = oracle.ppr_push(*csr, 0, 0.15, 1e-7, seeded=True, seed_v=he, seed_w=hw)
        assert st.status_flags == 0
        _check_heavy(pr, rp, rounds)
        _check_heavy(res, rr, rounds)


@pytest.mark.parametrize("n", [1, 3, 40])
@pytest.mark.parametrize("records", [True, False])
def test_batches_beyond_the_limit(gpu_available, n, records):
    """The same in batches, which pull from few pushes on when the library decides; and a path whose weights, not
    its records, pass the limit: 1e20, 1e20, 1e-30, 1."""
    import c2g
    import oracle

    csr, (hv, he, hw) = _heavy_records()
    if not records:
        csr = (np.arange(6, dtype=np.int32).clip(0, 4), np.array([1, 2, 3, 4], np.int32),
               np.array([1e20, 1e20, 1e-30, 1.0], np.float32))
        he, hw = [], []
    with c2g.Graph.create(csr[0], csr[1], flist=csr[2]) as g:
        if records:
            g.set_records(hv, he, hw)
        prm = g.ppr_params(alpha=0.15, rmax=1e-7, pr0=0.15, seeded=int(records), max_iter=500)
        rp, rr, rounds, _ = oracle.ppr_push(*csr, 0, 0.15, 1e-7, seeded=records, seed_v=he, seed_w=hw)
        for ratio in (None, 0.0):
            if ratio is not None:
                g.ppr_batch_pull(ratio)
            pr, res, st = g.ppr_batch(np.zeros(n, np.int32), prm)
            assert st.status_flags == 0
            for q in range(n):
                _check_heavy(pr[q], rp, rounds)
                _check_heavy(res[q], rr, rounds)
