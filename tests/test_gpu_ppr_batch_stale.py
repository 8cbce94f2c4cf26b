"""One-word batches on a handle whose pushed residuals still hold an earlier call's infinities and NaN: a
lane that reads two queries' residuals at once takes only those of active ones.

Tolerance: L1 1e-6 per query for pr and res, the bar of the other batched push tests."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 3, 8, 9, 17, 31])
@pytest.mark.parametrize("ratio", [None, 0.0])
def test_residuals_of_an_earlier_call(gpu_available, tmp_path, n, ratio):
    import c2g
    import oracle

    d = str(tmp_path)
    c2g.rmat_write(d, 10, 8, n, 1, 100)
    o = oracle.load_dataset(d, "origin")
    rng = np.random.default_rng(n)
    src = rng.choice(np.flatnonzero(np.diff(o["vlist"]) > 0), n + 1).astype(np.int32)
    with c2g.Graph.load(d, "origin") as g:
        if ratio is not None:
            g.ppr_batch_pull(ratio)
        # an rmax below 1e-30 never pulls: infinite residuals wherever the queries come in 6 rounds
        g.ppr_batch(src, g.ppr_params(alpha=0.15, rmax=1e-31, seeded=0, pr0=0.15, r0=np.inf, max_iter=6))
        prm = g.ppr_params(alpha=0.15, rmax=1e-7, seeded=0, pr0=0.15, r0=1.0, max_iter=500)
        pr, res, st = g.ppr_batch(src[:n], prm)
        assert st.status_flags == 0 and st.iterations < 200
        for i in range(n):
            rp, rr, _, _ = oracle.ppr_push(o["vlist"], o["elist"], o["flist"], int(src[i]), 0.15, 1e-7)
            assert np.abs(pr[i].astype(np.float64) - rp).sum() <= 1e-6, i
            assert np.abs(res[i].astype(np.float64) - rr).sum() <= 1e-6, i
