"""Local queries of the single push, whose frontier stays small (large rmax), and default ones, on graphs around the
sizes where the rule for pull rounds changes: a local query's rounds push above 1.6M edges and pull below, and the
last rounds of a default one all pull below 2.5M.

Tolerance: L1 1e-6 of the mass in the graph, the bar of the other push tests."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("V,ef,always", [(106000, 15, True), (107500, 15, False), (166000, 15, False), (167500, 15, False),
                                         (266000, 15, False), (267500, 15, False)])
def test_local_and_default_queries(gpu_available, V, ef, always):
    import c2g
    import oracle

    rng = np.random.default_rng(V)
    key = np.unique(rng.integers(0, V, V * ef) * V + rng.integers(0, V, V * ef))
    src, el = key // V, (key % V).astype(np.int32)
    vl = np.zeros(V + 1, np.int32)
    np.cumsum(np.bincount(src, minlength=V), out=vl[1:])
    f = rng.random(len(el)) + 0.01
    f = (f / np.bincount(src, weights=f, minlength=V)[src]).astype(np.float32)
    assert (len(el) <= 1600000) == always
    with c2g.Graph.create(vl, el, flist=f) as g:
        for s in rng.choice(V, 2):
            for rmax in (0.1, 1e-3, 1e-7):
                prm = g.ppr_params(alpha=0.15, rmax=rmax, seeded=0, pr0=0.15, r0=1.0, max_iter=500)
                pr, res, st = g.ppr(int(s), prm)
                rp, rr, rounds, _ = oracle.ppr_push(vl, el, f, int(s), 0.15, rmax)
                assert st.status_flags == 0 and abs(st.iterations - rounds) <= 2
                assert np.abs(pr.astype(np.float64) - rp).sum() <= 1e-6
                assert np.abs(res.astype(np.float64) - rr).sum() <= 1e-6
                if rmax == 0.1:  # a pull visits every vertex, a push the targets of its frontier
                    assert (st.touched >= V) == always
