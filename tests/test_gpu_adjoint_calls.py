"""Gradient calls on one handle: target lists that grow and shrink (the kept workspace), repeated targets,
calls without pi, lambda and loss, results on the device, another graph's handle in between.

A call is compared with the same call on a fresh handle.  Below 4M edges every round of the pushes pulls,
each row summed in one order, so the two agree to the last bit; the loss is the sum, in the order of the
list, of pi at the targets."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_calls_on_one_handle(gpu_available, tmp_path):
    import torch

    import c2g

    d = str(tmp_path / "g")
    c2g.rmat_write(d, 11, 8, 4, 1, 100)
    rng = np.random.default_rng(2)
    with c2g.Graph.load(d, "origin") as g, c2g.Graph.load(d, "origin") as other:
        prm = g.ppr_params(alpha=0.15, rmax=1e-8, seeded=0, pr0=0.15, r0=1.0, max_iter=500)
        for n in (1, 64, 3, 1000, 64, 5000):
            targets = rng.integers(0, g.V, n).astype(np.int32)
            source = int(rng.integers(0, g.V))
            grad, pi, lam, loss, _ = g.ppr_adjoint(source, targets, prm, rmax_backward=1e-8)
            with c2g.Graph.load(d, "origin") as fresh:
                g2, p2, l2, loss2, _ = fresh.ppr_adjoint(source, targets, prm, rmax_backward=1e-8)
            assert np.array_equal(grad, g2) and np.array_equal(pi, p2) and np.array_equal(lam, l2)
            want = 0.0
            for t in targets:
                want += float(pi[t])
            assert loss == want and loss2 == want
            other.ppr_adjoint(source, targets[: n // 2 + 1], prm, rmax_backward=1e-8)
            # gradient alone, on the device
            dg = torch.full((g.E,), -1.0, dtype=torch.float32, device="cuda")
            st = c2g.Stats()
            rc = c2g.lib().c2g_ppr_adjoint(g._h, source, ctypes.byref(prm), n, targets.ctypes.data_as(ctypes.c_void_p),
                                           1e-8, ctypes.c_void_p(dg.data_ptr()), None, None, None, 1, ctypes.byref(st))
            assert rc == c2g.OK
            assert np.array_equal(dg.cpu().numpy(), grad)
