"""A handle whose round shapes were set and set back to the defaults decides by itself again: its rounds are those of
a handle that was never set, push and pull alike."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture
def graph(gpu_available, tmp_path):
    import c2g

    d = str(tmp_path)
    c2g.rmat_write(d, 13, 8, 1, 1, 100)
    with c2g.Graph.load(d, "origin") as g:
        yield g


def test_single_push(graph):
    prm = graph.ppr_params(alpha=0.15, rmax=1e-7, seeded=0, pr0=0.15, r0=1.0, max_iter=500)
    unset = graph.ppr(5, prm)[2].touched  # a pull visits every vertex, a push the targets of its frontier
    graph.ppr_config(dense_div=16)
    assert graph.ppr(5, prm)[2].touched == unset
    graph.ppr_config(pull_div=0)
    assert graph.ppr(5, prm)[2].touched < unset
    graph.ppr_config()
    assert graph.ppr(5, prm)[2].touched == unset


def _shapes(graph, call):
    call()
    return list(graph.last_rounds()[2])


def test_batched_push(graph):
    prm = graph.ppr_params(alpha=0.15, rmax=1e-7, seeded=0, pr0=0.15, r0=1.0, max_iter=500)
    call = lambda: graph.ppr_batch(np.array([5, 9, 70], np.int32), prm)  # noqa: E731
    unset = _shapes(graph, call)
    assert 1 in unset
    graph.ppr_batch_pull(-1.0)
    assert 1 not in _shapes(graph, call)
    graph.ppr_batch_pull()
    assert _shapes(graph, call) == unset


def test_batched_sssp(graph):
    call = lambda: graph.sssp_batch(np.arange(100, dtype=np.int32))  # noqa: E731
    assert 1 not in _shapes(graph, call)  # a small batch
    graph.sssp_batch_pull(0.5)
    assert 1 in _shapes(graph, call)
    graph.sssp_batch_pull(0.3)
    assert 1 not in _shapes(graph, call)
