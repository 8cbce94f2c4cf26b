"""Resident SSSP batches whose running queries fill one, two, three or more query words of larger slot counts, at
word boundaries, before and after others leave, in epochs that pull every round and in the library's own: each
query's distances are Dijkstra's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("slots,first,second", [
    (32, 1, 31), (64, 8, 1), (64, 32, 32), (64, 33, 20), (128, 17, 64), (128, 40, 60), (256, 3, 250), (256, 64, 70),
    (320, 100, 200), (1024, 5, 40)])
def test_running_queries_in_some_of_the_words(gpu_available, tmp_path, slots, first, second):
    import c2g
    import oracle

    d = str(tmp_path / "g")
    c2g.rmat_write(d, 12, 12, 6, 1, 100)
    o = oracle.load_dataset(d, "origin")
    rng = np.random.default_rng(slots + first)
    cand = np.flatnonzero(np.diff(o["vlist"]) > 0)
    with c2g.Graph.load(d, "origin") as g:
        for frac in (0.0, 0.001, 0.3):
            g.sssp_batch_pull(frac)
            with c2g.Session(g, c2g.REQ_SSSP, slots) as s:
                source, left = {}, 0
                for src in rng.choice(cand, first):
                    source[s.admit(int(src))] = int(src)
                more = list(rng.choice(cand, second))
                for epoch in range(100):
                    done, _ = s.step(3)
                    for slot in done:
                        src = source.pop(slot)
                        left += 1
                        dist, _ = s.read(slot)
                        if left % 5 == 1:
                            assert np.array_equal(dist, oracle.dijkstra(o["vlist"], o["elist"], o["wlist"], [src], [0]))
                    if epoch == 1:
                        while more and len(source) < slots:
                            src = int(more.pop())
                            source[s.admit(src)] = src
                    if not source:
                        break
                assert not source and left == first + second
