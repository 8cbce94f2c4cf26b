"""A kind that is alone at work takes the whole GPU; another that arrives meanwhile waits for the end of
its epoch, and both then run on a third each.  Waves that make each kind start, in turn, while the other
is alone, and stay alone after it: every request ends, each result as the query run alone."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("epoch_rounds", [1, 4])
def test_arrivals_while_another_kind_is_alone(gpu_available, tmp_path, epoch_rounds):
    import c2g
    import oracle

    d = str(tmp_path / "g")
    c2g.rmat_write(d, 13, 16, 4, 1, 100)
    o = oracle.load_dataset(d, "origin")
    V = len(o["vlist"]) - 1
    rng = np.random.default_rng(epoch_rounds)
    pp = rng.dirichlet((1.0, 1.0, 1.0), size=V).astype(np.float32)
    src = rng.choice(np.flatnonzero(np.diff(o["vlist"]) > 0), 8)
    seeds = rng.choice(V, 16, replace=False).astype(np.int32)
    order = [c2g.REQ_PPR, c2g.REQ_SSSP, c2g.REQ_ADSORPTION]
    done = []
    with c2g.Graph.load(d, "origin") as g:
        labels, _ = g.adsorption(seeds, pp[:, 0], pp[:, 1], pp[:, 2], 30)
        with c2g.Server(g, max_batch=32, alpha=0.15, rmax=1e-7, ads_iterations=30, p_inj=pp[:, 0], p_cont=pp[:, 1],
                        p_abnd=pp[:, 2], epoch_rounds=epoch_rounds) as srv:
            for wave in range(9):
                tickets = []
                for k in range(3):
                    kind = order[(wave + k) % 3]
                    out = np.empty((V, 16), np.float32) if kind == c2g.REQ_ADSORPTION else np.empty(
                        V, np.int32 if kind == c2g.REQ_SSSP else np.float32)
                    s = int(src[(wave + k) % 8])
                    tickets.append(srv.submit(kind, source=s, seeds=seeds if kind == c2g.REQ_ADSORPTION else None,
                                              out=out))
                    done.append((kind, s, out))
                    time.sleep(0.0004 * (wave % 4))
                for t in tickets:
                    status, _ = srv.wait(t, timeout=60.0)
                    assert status == c2g.OK
    for kind, s, out in done:
        if kind == c2g.REQ_SSSP:
            assert np.array_equal(out, oracle.dijkstra(o["vlist"], o["elist"], o["wlist"], [s], [0]))
        elif kind == c2g.REQ_PPR:
            rp, _, _, _ = oracle.ppr_push(o["vlist"], o["elist"], o["flist"], s, 0.15, 1e-7)
            assert float(np.abs(out.astype(np.float64) - rp).sum()) <= 1e-6
        else:
            assert float(np.abs(out.astype(np.float64) - labels).max()) <= 1e-6
