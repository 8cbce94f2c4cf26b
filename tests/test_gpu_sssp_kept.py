"""Single-query SSSP on graphs of at most one map word per warp (each warp keeps its vertices' first
in-edges and distances for all rounds), just within and beyond that limit, with hub rows that go to the
whole grid in several rounds.  Distances are whole numbers: equal to Dijkstra's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _csr(V, src, dst, w):
    order = np.lexsort((dst, src))
    src = src[order]
    vl = np.zeros(V + 1, np.int32)
    np.cumsum(np.bincount(src, minlength=V), out=vl[1:])
    return vl, dst[order].astype(np.int32), w[order].astype(np.int32)


def _check(csr, sources):
    import c2g
    import oracle

    with c2g.Graph.create(csr[0], csr[1], wlist=csr[2]) as g:
        for s in sources:
            dist, st = g.sssp(int(s))
            assert st.status_flags == 0
            assert np.array_equal(dist, oracle.dijkstra(*csr, [int(s)], [0])), s


@pytest.mark.parametrize("over", [-33, -1, 0, 1, 33])
def test_vertices_around_the_resident_words(gpu_available, over):
    import torch

    V = torch.cuda.get_device_properties(0).multi_processor_count * 32 * 32 + over
    rng = np.random.default_rng(abs(over))
    src, dst = rng.integers(0, V, 6 * V), rng.integers(0, V, 6 * V)
    _check(_csr(V, src, dst, rng.integers(0, 1000, 6 * V)), [0, V - 1])


@pytest.mark.parametrize("V", [1, 2, 31, 32, 33, 511, 512, 513, 5000])
@pytest.mark.parametrize("wmax", [1, 100000])
def test_hub_rows_over_several_rounds(gpu_available, V, wmax):
    """Every 9th vertex takes in-edges from up to 900 others; a chain of small weights keeps lowering them."""
    rng = np.random.default_rng(V + wmax)
    src, dst, w = [np.arange(V - 1)], [np.arange(1, V)], [rng.integers(0, 3, V - 1)]
    for h in range(0, V, max(9, V // 40)):
        n = min(V, 900)
        src.append(rng.choice(V, n, replace=False))
        dst.append(np.full(n, h))
        w.append(rng.integers(0, wmax + 1, n))
    src, dst, w = np.concatenate(src), np.concatenate(dst), np.concatenate(w)
    extra = rng.integers(0, V, (2, 3 * V))
    _check(_csr(V, np.concatenate([src, extra[0]]), np.concatenate([dst, extra[1]]),
                np.concatenate([w, rng.integers(0, wmax + 1, 3 * V)])), {0, V // 2, V - 1})
