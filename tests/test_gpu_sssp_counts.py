"""vertices_popped and edges_relaxed of a query whose hub row is lowered by both parts of one pull round: the row's
first groups give the hub a distance, its later ones, read by the whole grid, a smaller one.  It is popped once.

source -> 8 vertices (weight 90) -> hub (weight 1), source -> n vertices (weight 5) -> hub (weight 50); each of
those m = n + 8 vertices has 3 edges more and the hub 2 m, to vertices without out-edges (weight 1).  The counts
follow: the source (m edges), the m vertices (4 each), the hub (2 m), once each; where every round pulls, the
source's edges are relaxed before the first round and the m vertices are in no round's frontier."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# pulls only, with kept words and without; push, pull, pull by the frontier's out-edges
@pytest.mark.parametrize("V", [4000, 200000, 300001])
@pytest.mark.parametrize("n", [130, 1000])
def test_hub_lowered_in_both_parts(gpu_available, V, n):
    import c2g

    m, hub = n + 8, V - 1
    mid, leaf = np.arange(1, m + 1), m + 1 + np.arange(2 * m)
    src = np.concatenate([np.zeros(m), np.repeat(mid, 4), np.full(2 * m, hub)]).astype(np.int64)
    to = np.column_stack([leaf[:m], leaf[:m], leaf[m:], np.full(m, hub)])
    to[:, 1] = np.roll(leaf[:m], 1)
    wt = np.column_stack([np.ones((m, 3)), np.where(mid <= 8, 1, 50)])
    dst = np.concatenate([mid, to.ravel(), leaf]).astype(np.int32)
    w = np.concatenate([np.where(mid <= 8, 90, 5), wt.ravel(), np.ones(2 * m)]).astype(np.int32)
    vl = np.zeros(V + 1, np.int32)
    np.cumsum(np.bincount(src, minlength=V), out=vl[1:])
    with c2g.Graph.create(vl, dst, w) as g:
        dist, st = g.sssp(0)
    assert dist[hub] == 55 and np.array_equal(dist[mid], w[:m])
    between = 0 if V <= 300000 else m
    assert st.vertices_popped == 2 + between
    assert st.edges_relaxed == m + 4 * between + 2 * m
