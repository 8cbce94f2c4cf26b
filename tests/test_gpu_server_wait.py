"""A kind that is alone at work has the whole GPU for 4 rounds at a time, however long the server's epochs are: a
request of another kind that arrives meanwhile waits for the end of that epoch, not of the other kind's queries."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("epoch_rounds", [2, 4, 1000])
def test_epochs_of_a_kind_alone(gpu_available, tmp_path, epoch_rounds):
    import c2g

    d = str(tmp_path)
    c2g.rmat_write(d, 12, 8, 6, 1, 100)
    with c2g.Graph.load(d, "origin") as g:
        s = int(np.argmax(np.diff(np.fromfile(d + "/origin/vlist.bin", dtype=np.int32))))
        prm = g.ppr_params(alpha=0.15, rmax=1e-7, seeded=0, pr0=0.15, r0=1.0, max_iter=500)
        pr, _, st = g.ppr(s, prm)
        dist, ss = g.sssp(s)
        rounds = {c2g.REQ_PPR: st.iterations, c2g.REQ_SSSP: ss.iterations}
        with c2g.Server(g, max_batch=8, alpha=0.15, rmax=1e-7, epoch_rounds=epoch_rounds) as srv:
            for kind, want in ((c2g.REQ_PPR, pr), (c2g.REQ_SSSP, dist)):
                out = np.empty_like(want)
                status, _ = srv.wait(srv.submit(kind, source=s, out=out), timeout=60.0)
                assert status == c2g.OK and np.abs(out.astype(np.float64) - want).max() <= 1e-6
                # (the batch's rounds may differ from the single query's by one or two)
                assert srv.stats().batches[kind] >= (rounds[kind] - 2) / min(epoch_rounds, 4)
