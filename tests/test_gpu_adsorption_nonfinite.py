"""Label propagation with p_cont that is infinite or NaN: its product with a sum of no in-edges is NaN, as with a
zero sum, and spreads along the out-edges like any label.  The classes (finite, infinite, NaN) of all entries are
those of the formula in 64 bits; finite ones are within 20 k 2^-24 (rows of at most 12 in-edges)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("V", [300, 40000])  # 64-edge tiles, larger ones
@pytest.mark.parametrize("bad", [np.inf, np.nan])
def test_rows_without_in_edges(gpu_available, V, bad):
    import c2g

    rng = np.random.default_rng(V)
    bare = V // 10  # the first vertices have out-edges only
    src, dst = rng.integers(0, V, 3 * V), rng.integers(bare, V, 3 * V)
    key = np.unique(src * V + dst)
    key = key[rng.random(len(key)) < 0.9]
    src, dst = key // V, key % V
    vl = np.zeros(V + 1, np.int32)
    np.cumsum(np.bincount(src, minlength=V), out=vl[1:])
    w = rng.random(len(src)).astype(np.float32)
    pp = rng.dirichlet((1.0, 1.0, 1.0), size=V).astype(np.float32)
    pi, pc = pp[:, 0].copy(), pp[:, 1].copy()
    seeds = rng.integers(bare, V, 16).astype(np.int32)
    seeds[:3] = 0, 1, 1
    pc[[1, 2, 3, bare + 1]] = bad  # seeded and not, with and without in-edges
    inject = np.zeros((V, 16))
    np.add.at(inject, (seeds, np.arange(16)), 1.0)
    y = inject
    with c2g.Graph.create(vl, dst.astype(np.int32), flist=w) as g, np.errstate(all="ignore"):
        for k in range(5):
            got = g.adsorption(seeds, pi, pc, pp[:, 2], iterations=k)[0].astype(np.float64)
            assert np.array_equal(np.isnan(got), np.isnan(y)) and np.array_equal(np.isinf(got), np.isinf(y))
            fin = np.isfinite(y)
            assert (np.abs(got - y)[fin] <= 20 * k * 2.0**-24 * y[fin] + 1e-38).all()
            total = np.zeros((V, 16))
            np.add.at(total, dst, w[:, None].astype(np.float64) * y[src])
            y = pi[:, None].astype(np.float64) * inject + pc[:, None].astype(np.float64) * total
