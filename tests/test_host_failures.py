"""Failures on the library's host side, made by a CUDA runtime without a device (fake_cudart.cpp): allocations that
do not fit and launches that are refused or end with status flags.  Device memory is host memory and kernels do
nothing, so these tests read status codes, the kernels that were launched and what the caller's arrays hold.
No GPU."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from conftest import PKG, REPO


@pytest.fixture(scope="module")
def fake_lib(built, tmp_path_factory):
    """The library's objects linked against the fake runtime."""
    d = str(tmp_path_factory.mktemp("fake"))
    csrc = os.path.join(PKG, "csrc")
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    objs = [os.path.join(PKG, "lib", "obj", f + ".o") for f in os.listdir(csrc) if f.endswith((".cu", ".cpp"))]
    subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", "-I", os.path.join(cuda, "include"), "-I", csrc, "-c",
                    os.path.join(REPO, "tests", "fake_cudart.cpp"), "-o", d + "/fake.o"], check=True)
    subprocess.run(["g++", "-shared", "-fopenmp", "-Wl,-Bsymbolic", "-o", d + "/libfake.so", d + "/fake.o"] + objs +
                   ["-lpthread"], check=True)
    return d + "/libfake.so"


@pytest.fixture
def fake(fake_lib, monkeypatch):
    import c2g

    monkeypatch.setattr(c2g, "LIB_PATH", fake_lib)
    monkeypatch.setattr(c2g, "_lib", None)
    L = c2g.lib()
    L.fake_budget.argtypes = [ctypes.c_size_t]
    L.fake_in_use.restype = ctypes.c_size_t
    L.fake_launched.restype = ctypes.c_char_p
    L.fake_reset()
    yield L
    L.fake_reset()


def _graph(V=4096, ef=16, kinds="wf"):
    import c2g

    rng = np.random.default_rng(3)
    src = np.sort(rng.integers(0, V, V * ef))
    vl = np.zeros(V + 1, np.int32)
    np.cumsum(np.bincount(src, minlength=V), out=vl[1:])
    E = len(src)
    return c2g.Graph.create(vl, rng.integers(0, V, E).astype(np.int32),
                            wlist=rng.integers(1, 9, E).astype(np.int32) if "w" in kinds else None,
                            flist=rng.random(E).astype(np.float32) if "f" in kinds else None)


def test_a_call_that_does_not_fit_leaves_no_error_behind(fake):
    import c2g

    with _graph() as g:
        g.ppr_config(pull_div=0)  # no in-edges, which the call could do without
        fake.fake_fail_malloc(2)
        with pytest.raises(c2g.C2GError) as e:
            g.ppr(0)
        assert e.value.code == c2g.ERR_OOM
        g.ppr(0)  # its launches are checked for errors


@pytest.mark.parametrize("on_device", [0, 1])
def test_set_weights_that_do_not_fit_change_nothing(fake, on_device):
    import c2g

    with _graph(kinds="f") as g:
        w = np.ones(g.E, np.float32)
        for n in range(2 - on_device):  # each of the call's allocations
            fake.fake_reset()
            fake.fake_fail_malloc(n)
            held = fake.fake_in_use()
            assert fake.c2g_graph_set_weights(g._h, c2g._ptr(w), on_device) == c2g.ERR_OOM
            assert fake.fake_launched() == b"" and fake.fake_in_use() == held
        fake.fake_reset()
        g.set_weights(w)
        assert b"set_weight_bits" in fake.fake_launched() and b"in_scatter" in fake.fake_launched()


@pytest.mark.parametrize("push", [0, 1])
def test_a_failed_adjoint_leaves_the_results_alone(fake, push):
    """A push that ends with an error (here: its grid barrier gave up) returns it before anything is written."""
    import c2g

    with _graph() as g:
        prm = g.ppr_params(alpha=0.15, rmax=1e-7, seeded=0)
        targets = np.array([5, 7], np.int32)
        out = [np.full(n, 7.0, np.float32) for n in (g.E, g.V, g.V)]
        loss = ctypes.c_double(7.0)
        call = lambda: fake.c2g_ppr_adjoint(  # noqa: E731
            g._h, 1, ctypes.byref(prm), 2, c2g._ptr(targets), 1e-7, *(c2g._ptr(a) for a in out), ctypes.byref(loss), 0, None)
        fake.fake_flag_launch(push, c2g.FLAG_BARRIER_TIMEOUT)
        assert call() == c2g.ERR_OVERFLOW
        assert all((a == 7.0).all() for a in out) and loss.value == 7.0
        fake.fake_reset()
        assert call() == c2g.OK and not any((a == 7.0).any() for a in out)


def test_each_kind_of_call_builds_its_own_in_edges(fake):
    """A graph with both kinds of weights is made without in-edges; one with a single kind with that kind's."""
    with _graph() as g:
        assert b"in_count" not in fake.fake_launched()
        for call, rows, lists in ((lambda: g.sssp(0), 1, 0), (lambda: g.ppr(0), 1, 1), (lambda: g.sssp(1), 1, 1),
                                  (lambda: g.ppr(1), 1, 1)):
            call()
            log = fake.fake_launched()
            assert log.count(b"in_sort_short") == rows and (b"row_classes" in log) == bool(lists)
    fake.fake_reset()
    with _graph(kinds="w") as g:
        assert b"in_sort_short" in fake.fake_launched() and b"row_classes" not in fake.fake_launched()
    fake.fake_reset()
    with _graph(kinds="f") as g:
        assert b"in_sort_short" not in fake.fake_launched() and b"row_classes" in fake.fake_launched()


_SOURCES = np.arange(3, dtype=np.int32)
_CALLS = {"sssp": ("w", lambda g: g.sssp(0)), "sssp_batch": ("w", lambda g: g.sssp_batch(_SOURCES)),
          "ppr": ("f", lambda g: g.ppr(0)), "ppr after sssp": ("wf", lambda g: (g.sssp(0), g.ppr(0))),
          "ppr_batch after sssp": ("wf", lambda g: (g.sssp(0), g.ppr_batch(_SOURCES))),
          "adsorption after sssp": ("wf", lambda g: (g.sssp(0), g.adsorption(np.arange(16), *np.ones((3, g.V), np.float32)))),
          "adjoint after sssp": ("wf", lambda g: (g.sssp(0), g.ppr_adjoint(0, _SOURCES)))}


@pytest.mark.parametrize("name", sorted(_CALLS))
def test_workspaces_that_fit_only_without_in_edges(fake, name):
    """In-edges that leave too little room for a call's workspace go, where no session shares them."""
    import c2g

    kinds, call = _CALLS[name]
    before = fake.fake_in_use()
    with _graph(kinds=kinds) as g:
        call(g)
        held = fake.fake_in_use()
    assert fake.fake_in_use() == before
    with _graph(kinds=kinds) as g:
        fake.fake_budget(held - 1000)
        call(g)
        assert fake.fake_in_use() <= held - 1000
        call(g)
    assert fake.fake_in_use() == before
    if name == "sssp_batch":  # a session's view keeps them
        fake.fake_reset()
        with _graph(kinds=kinds) as g, c2g.Session(g, c2g.REQ_SSSP, 32):
            fake.fake_budget(fake.fake_in_use() + 1000)
            with pytest.raises(c2g.C2GError) as e:
                call(g)
            assert e.value.code == c2g.ERR_OOM
