"""The per-frame spread plan (contributor lists of every tile) of fields with
targets of their own: kept for a field that its owner may apply any number of
times, left out of a near field, which is applied once per set of positions.
Seen by the lists' bytes: 64 entries of a weight in both precisions and an index
for each of the 8 x 8 columns of a tile of 8 planes."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

BOX = 40.0


def growth(make):
    """(object, device bytes that it holds)"""
    from cumpm_b200 import capi

    before = capi.buffer_stats()["live_device"]
    obj = make()
    return obj, capi.buffer_stats()["live_device"] - before


def lists(grid):
    return int(np.prod([-(-g // 8) for g in grid])) * 64 * 64 * 16


def test_interaction_field_keeps_a_plan():
    from cumpm_b200 import capi

    rng = np.random.default_rng(0)
    pos, pts = rng.uniform(0, BOX, (300, 3)), rng.uniform(0, BOX, (200, 3))
    f = capi.Field(capi.FIELD_MONO, (BOX,) * 3, 1e-3, 0.5, mode=capi.MODE_INTERACTION)
    f.set_field_points(pts)
    _, held = growth(lambda: f.set_positions(pos))
    info = f.info()
    assert not info["pruned"]
    assert held > lists(info["grid"])


def test_near_field_has_none():
    import cumpm_b200 as cu
    from cumpm_b200 import capi

    rng = np.random.default_rng(0)
    pos, pts = rng.uniform(0, BOX, (300, 3)), rng.uniform(0, BOX, (200, 3))
    g = capi.ewald_geometry((BOX,) * 3, 1e-3, 0.5)["grid"]

    def make():
        nf = cu.Near_Field(np.array([BOX] * 3), np.array([1.0, 0, 0], complex), 1.0, xi=0.5, errortol=1e-3)
        nf.set_dipoles(np.ones((300, 3), complex))
        nf.set_dipole_positions(pos)
        nf.set_field_points(pts)
        nf.calculate()
        return nf

    nf, held = growth(make)
    assert 0 < held < lists(g)
