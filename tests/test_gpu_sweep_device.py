"""The frequency-by-frequency sweep whose guesses, right-hand sides and self
coefficients are made on the device, against every frequency solved by a solver
of its own (no guess from its neighbours): each guess type, both solvers, one to
four frequencies (the extrapolation starts at the third), two frames, several
materials, an epsilon that two frequencies share (the extrapolation's run is
zero there) and one equal to the medium's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def run(eps, pos, **kw):
    import cumpm_b200 as cu

    s = cu.dipole_solver(np.array([30.0, 31.0, 32.0]), eps, radius=1.0, eps_m=1.2, tol=1e-9, quiet=True,
                         precision="double", **kw)
    s.compute(pos)
    return s.get_dipoles(), s.get_eff_polarizability()


@pytest.mark.parametrize("field_type", ["auto", "direct"])
@pytest.mark.parametrize("guess", ["derivative", "previous", "mean_field"])
@pytest.mark.parametrize("W,solver", [(1, "gmres"), (2, "bicgstab"), (4, "gmres"), (4, "bicgstab")])
def test_sweep_matches_single_frequencies(W, solver, guess, field_type):
    rng = np.random.default_rng(W)
    n = 20
    g = np.stack(np.meshgrid(np.arange(3), np.arange(3), np.arange(3)), axis=-1).reshape(-1, 3)[:n]
    frames = [g * 3.0 + rng.uniform(-0.3, 0.3, (n, 3)) for _ in range(2)]
    omega = np.linspace(0.4, 0.8, W)
    eps = (4 - 1.8 ** 2 / (omega ** 2 + 0.1j * omega))[:, None] + np.where(np.arange(n) % 2, 1.5, 0.0)[None, :]
    if W == 4:
        eps[2] = eps[1]
        eps[:, 0] = 1.2          # the medium's own
    d, a = run(eps, np.stack(frames), guess_type=guess, solver_type=solver, field_type=field_type)
    d, a = d.reshape(2, W, n, 3, 3), a.reshape(W, 3, 3)
    for f in range(2):
        for w in range(W):
            ref = run(eps[w:w + 1], frames[f], solver_type=solver, field_type=field_type)[0].reshape(n, 3, 3)
            assert np.abs(d[f, w] - ref).max() < 1e-6 * np.abs(ref).max(), (f, w)
    np.testing.assert_allclose(a, d.mean(axis=(0, 2)), rtol=1e-10, atol=1e-10 * np.abs(a).max())


def test_extrapolation_from_an_epsilon_close_to_the_mediums():
    """(eps + 2) / (eps - 1) whose divisor's square vanishes in 64 bits."""
    g = np.stack(np.meshgrid(np.arange(2), np.arange(2), np.arange(2)), axis=-1).reshape(-1, 3) * 3.0
    eps = 1.2 * np.array([1.0 + 0.5j, 1.0 + 1e-170j, 1.0 + 2e-170j, 2.0 + 0.1j])
    d, _ = run(eps, g, guess_type="derivative", field_type="direct")
    d = d.reshape(4, 8, 3, 3)
    assert np.isfinite(d).all()
    ref = run(eps[3:], g, field_type="direct")[0].reshape(8, 3, 3)
    assert np.abs(d[3] - ref).max() < 1e-6 * np.abs(ref).max()


def test_unknown_guess_is_refused_at_the_second_frequency():
    g = np.array([[0.0, 0, 0], [3.0, 0, 0]])
    run(np.array([2.0 + 0.1j]), g, guess_type="none")
    with pytest.raises(RuntimeError, match="not supported"):
        run(np.array([2.0 + 0.1j, 2.1 + 0.1j]), g, guess_type="none")
