"""Kept buffers (mpm_alloc.cpp): a dropped solver's are reused and given back on
request."""
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
