"""Kept buffers (mpm_alloc.cpp): a dropped solver's are reused and given back on
request, large ones are not enlarged, and dropping objects leaves graph captures
of other threads alone."""
import threading

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


def solver(n=20):
    import cumpm_b200 as cu

    g = np.stack(np.meshgrid(np.arange(3), np.arange(3), np.arange(3)), axis=-1).reshape(-1, 3)[:n] * 3.0
    s = cu.dipole_solver(np.array([30.0, 31.0, 32.0]), np.array([-3.0 + 0.4j, -2.5 + 0.4j]), radius=1.0, tol=1e-3,
                         quiet=True)
    s.compute(g)
    return s


def field(box=20.0, n=14):
    from cumpm_b200 import capi

    f = capi.Field(capi.FIELD_MONO, (box,) * 3, 1e-3, 0.5)
    f.set_positions(np.random.default_rng(0).uniform(0, box, (n, 3)))
    return f


def test_a_solvers_buffers_are_kept_within_bounds_and_given_back():
    from cumpm_b200 import capi

    solver()
    capi.empty_cache()
    base = capi.buffer_stats()
    assert base["kept_device"] == base["kept_host"] == 0
    a = solver().get_dipoles()
    kept = capi.buffer_stats()
    assert 0 < kept["kept_device"] <= 256 << 20 and 0 < kept["kept_host"] <= 64 << 20
    assert kept["live_device"] == base["live_device"] and kept["live_host"] == base["live_host"]
    assert (solver().get_dipoles() == a).all()               # on the kept blocks
    again = capi.buffer_stats()
    assert again["kept_device"] <= 256 << 20 and again["kept_host"] <= 64 << 20
    capi.empty_cache()
    none = capi.buffer_stats()
    assert none["kept_device"] == none["kept_host"] == 0


def test_a_fields_buffers_are_kept_unless_a_graph_may_use_them():
    from cumpm_b200 import capi

    X = torch.ones((42, 3), dtype=torch.complex128, device="cuda")
    Y = torch.empty_like(X)
    capi.empty_cache()
    f = field()
    other = torch.cuda.Stream()
    for s in (torch.cuda.current_stream(), other):           # on two streams
        f.apply(X, Y, stream=s)
    del f
    assert capi.buffer_stats()["kept_device"] > 0
    torch.cuda.synchronize()
    f = field()
    f.apply(X, Y)
    torch.cuda.synchronize()
    ref = Y.clone()
    capi.empty_cache()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        f.apply(X, Y)
    Y.zero_()
    g.replay()
    torch.cuda.synchronize()
    assert (Y == ref).all()
    del f
    assert capi.buffer_stats()["kept_device"] == 0


def test_large_buffers_are_not_enlarged():
    """A grid of 1.1 GB: what a field holds beyond its requests is less than the
    quarter by which small blocks may be rounded up."""
    from cumpm_b200 import capi

    box, m = 180.0, 12
    f = field(box, 50)
    before = capi.buffer_stats()["live_device"]
    f.apply(torch.zeros((150, m), dtype=torch.complex128, device="cuda"), recip_fp32=True)
    g = f.info()["grid"]
    grid = 8 * 3 * m * g[0] * g[1] * g[2]
    assert grid > 256 << 20
    assert grid <= capi.buffer_stats()["live_device"] - before < grid + (64 << 20)


@pytest.mark.parametrize("mode", ["thread_local", "relaxed"])
@pytest.mark.parametrize("make", [field, solver])
def test_dropping_an_object_leaves_a_capture_of_another_thread_alone(make, mode):
    held = [make()]
    go, done = threading.Event(), threading.Event()

    def drop():
        go.wait(30)
        held.pop()
        done.set()

    t = threading.Thread(target=drop)
    t.start()
    a = torch.ones(1024, device="cuda")
    b = torch.zeros_like(a)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    try:
        with torch.cuda.graph(g, capture_error_mode=mode):
            b.copy_(a * 2)
            go.set()
            assert done.wait(30)
            b.add_(1)
    finally:
        go.set()
        t.join()
    g.replay()
    torch.cuda.synchronize()
    assert (b == 3).all()
