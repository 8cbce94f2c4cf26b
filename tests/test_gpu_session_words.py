"""Resident push batches whose running queries fill one, two, three or more query words of larger slot
counts, at word boundaries, before and after others leave: each query's result is the FP64 push's within
L1 1e-6, the bar of the other session tests."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("slots,first,second", [
    (64, 8, 1), (64, 9, 30), (64, 16, 17), (64, 32, 32), (64, 33, 20), (128, 17, 64), (128, 40, 60), (256, 3, 250),
    (256, 64, 70), (320, 100, 200)])
def test_running_queries_in_some_of_the_words(gpu_available, tmp_path, slots, first, second):
    import c2g
    import oracle

    d = str(tmp_path / "g")
    c2g.rmat_write(d, 12, 12, 6, 1, 100)
    o = oracle.load_dataset(d, "origin")
    rng = np.random.default_rng(slots + first)
    cand = np.flatnonzero(np.diff(o["vlist"]) > 0)
    with c2g.Graph.load(d, "origin") as g:
        for ratio in (0.0, 8.0):
            g.ppr_batch_pull(ratio)
            prm = g.ppr_params(alpha=0.15, rmax=1e-7, seeded=0, pr0=0.15, r0=1.0, max_iter=500)
            with c2g.Session(g, c2g.REQ_PPR, slots, prm) as s:
                source, left = {}, 0
                for src in rng.choice(cand, first):
                    source[s.admit(int(src))] = int(src)
                more = list(rng.choice(cand, second))
                for epoch in range(400):
                    done, _ = s.step(3)
                    for slot in done:
                        src = source.pop(slot)
                        left += 1
                        (pr, res), _ = s.read(slot, want_res=True)
                        if left % 7 == 1:
                            rp, rr, _, _ = oracle.ppr_push(o["vlist"], o["elist"], o["flist"], src, 0.15, 1e-7)
                            assert np.abs(pr.astype(np.float64) - rp).sum() <= 1e-6
                            assert np.abs(res.astype(np.float64) - rr).sum() <= 1e-6
                    if epoch == 2:
                        while more and len(source) < slots:
                            src = int(more.pop())
                            source[s.admit(src)] = src
                    if not source:
                        break
                assert not source and left == first + second
