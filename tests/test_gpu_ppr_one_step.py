"""Single-query push on graphs whose rows are about one step per resident warp: the kept-rows loop just
within and just beyond its limit, against the FP64 push, with and without rows in segments.

Tolerance: L1 1e-6 of the mass in the graph, the bar of the other push tests."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("over", [-40, -1, 0, 1, 40])
@pytest.mark.parametrize("long_rows", [0, 3])
def test_steps_around_the_resident_warps(gpu_available, over, long_rows):
    import c2g
    import oracle
    import torch

    warps = torch.cuda.get_device_properties(0).multi_processor_count * 32
    rng = np.random.default_rng(100 + over)
    V = warps + 200
    # rows of 129 to 200 in-edges are one step each, 700 in-edges three (segments of 256)
    lengths = np.concatenate([np.full(long_rows, 700), rng.integers(129, 201, warps + over - 3 * long_rows)])
    dst = np.repeat(np.arange(len(lengths)), lengths)
    src = rng.integers(0, V, len(dst))
    order = np.lexsort((dst, src))
    src, dst = src[order], dst[order].astype(np.int32)
    vl = np.zeros(V + 1, np.int32)
    np.cumsum(np.bincount(src, minlength=V), out=vl[1:])
    w = rng.random(len(src)) + 0.01
    w = (w / np.bincount(src, weights=w, minlength=V)[src]).astype(np.float32)
    with c2g.Graph.create(vl, dst, flist=w) as g:
        for s in (0, V - 1):  # the last one has no in-edges
            prm = g.ppr_params(alpha=0.15, rmax=1e-7, seeded=0, pr0=0.15, r0=1.0, max_iter=500)
            pr, res, st = g.ppr(s, prm)
            rp, rr, rounds, _ = oracle.ppr_push(vl, dst, w, s, 0.15, 1e-7)
            assert st.status_flags == 0 and abs(st.iterations - rounds) <= 2
            assert np.abs(pr.astype(np.float64) - rp).sum() <= 1e-6
            assert np.abs(res.astype(np.float64) - rr).sum() <= 1e-6
