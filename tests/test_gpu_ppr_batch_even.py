"""Batched pulls on graphs without long rows, whose items are 2, 4 and 8 chunks of 32 in-edges on far smaller graphs
than those with hubs: rows inside an item, across chunks and across items, one to five query words.

Tolerance: L1 1e-6 per query for pr and res, the bar of the other batched push tests."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("V,ef", [(60000, 15), (120001, 17), (100000, 40)])
@pytest.mark.parametrize("n", [3, 40, 70, 130])
def test_long_items(gpu_available, V, ef, n):
    import c2g
    import oracle

    rng = np.random.default_rng(V)
    key = np.unique(rng.integers(0, V, V * ef) * V + rng.integers(0, V, V * ef))
    src, el = key // V, (key % V).astype(np.int32)
    vl = np.zeros(V + 1, np.int32)
    np.cumsum(np.bincount(src, minlength=V), out=vl[1:])
    f = rng.random(len(el)) + 0.01
    f = (f / np.bincount(src, weights=f, minlength=V)[src]).astype(np.float32)
    assert np.bincount(el, minlength=V).max() <= 256
    ss = rng.choice(V, n).astype(np.int32)
    with c2g.Graph.create(vl, el, flist=f) as g:
        prm = g.ppr_params(alpha=0.15, rmax=1e-6, seeded=0, pr0=0.15, r0=1.0, max_iter=500)
        pr, res, st = g.ppr_batch(ss, prm)
        assert st.status_flags == 0 and 1 in g.last_rounds()[2]
        for i in (0, n // 2, n - 1):
            rp, rr, _, _ = oracle.ppr_push(vl, el, f, int(ss[i]), 0.15, 1e-6)
            assert np.abs(pr[i].astype(np.float64) - rp).sum() <= 1e-6
            assert np.abs(res[i].astype(np.float64) - rr).sum() <= 1e-6
