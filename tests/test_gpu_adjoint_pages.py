"""Gradient calls into host arrays large enough that their pages are made ready beside the pushes (4 MB and
more): the gradient alone (few vertices), and pi and lambda read in several pieces, the last one ragged (more
vertices than edges).

Compared with the same call into device arrays, to the last bit: up to 1.6M edges every round of the pushes
pulls, each row summed in one order."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("V", [100_001, 2_300_003])
def test_large_host_arrays(gpu_available, V):
    import torch

    import c2g

    E = 1_100_003
    rng = np.random.default_rng(V)
    src = np.sort(rng.integers(0, V // 2, E))
    row = np.zeros(V + 1, np.int32)
    row[1:] = np.cumsum(np.bincount(src, minlength=V))
    w = rng.random(E) + 0.01
    w = (w / np.bincount(src, weights=w, minlength=V)[src]).astype(np.float32)
    with c2g.Graph.create(row, rng.integers(0, V // 2, E).astype(np.int32), flist=w) as g:
        prm = g.ppr_params(alpha=0.15, rmax=1e-7, seeded=0, pr0=0.15, r0=1.0, max_iter=500)
        targets = rng.integers(0, V // 2, 40).astype(np.int32)
        for source in (int(src[0]), int(src[-1])):
            grad, pi, lam, loss, _ = g.ppr_adjoint(source, targets, prm, rmax_backward=1e-7)
            out = [torch.full((n,), -1.0, dtype=torch.float32, device="cuda") for n in (E, V, V)]
            dloss = ctypes.c_double()
            rc = c2g.lib().c2g_ppr_adjoint(g._h, source, ctypes.byref(prm), len(targets),
                                           targets.ctypes.data_as(ctypes.c_void_p), 1e-7,
                                           *(ctypes.c_void_p(t.data_ptr()) for t in out), ctypes.byref(dloss), 1, None)
            assert rc == c2g.OK
            for host, dev in zip((grad, pi, lam), out):
                assert np.array_equal(host, dev.cpu().numpy())
            assert loss == dloss.value and pi[source] > 0 and np.count_nonzero(lam) >= len(set(targets.tolist()))
