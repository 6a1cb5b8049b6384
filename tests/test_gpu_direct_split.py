"""The open-boundary dipole sum (k_direct) against the plain pair sum in 64
bits, over the column counts of its instantiations (1, 2-3, more than 3 with a
partial last chunk), targets on both sides of a CTA's 8 and 32 and of a source
tile's 64, radii that overlap, and field points that are not particles.
Tolerance: N rounded terms per value."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


def reference(pos, tgt, rad, X, sc, solver_ax):
    N, T = len(pos), len(tgt)
    Y = np.zeros((T, 3, X.shape[1]), complex)
    P = X.reshape(N, 3, -1)
    k = (-1.0 if solver_ax else 1.0) / (4 * np.pi)
    for j in range(T):
        r = pos - tgt[j]
        r2 = np.sum(r * r, axis=1)
        use = np.arange(N) != j if solver_ax else np.ones(N, bool)
        inside = r2 < rad ** 2
        far = np.sqrt(r2) > 1e-9
        scl = np.where(inside & far, rad / np.sqrt(np.where(far, r2, 1.0)), 1.0)
        r = r * scl[:, None]
        r2 = np.where(inside, rad ** 2, r2)
        u = r / np.sqrt(r2)[:, None]
        pu = np.einsum("nc,ncm->nm", u, P)
        E = (3 * u[:, :, None] * pu[:, None, :] - P) * (k / r2 ** 1.5)[:, None, None]
        Y[j] = E[use].sum(axis=0)
        if solver_ax:
            Y[j] += (sc[j] + 1 / (4 * np.pi * rad[j] ** 3)) * P[j]
    return Y.reshape(3 * T, -1)


@pytest.mark.parametrize("fp32", [False, True])
@pytest.mark.parametrize("N,M", [(1, 1), (7, 3), (64, 2), (65, 7), (130, 12), (33, 4)])
def test_direct_sum(N, M, fp32):
    from cumpm_b200 import capi

    rng = np.random.default_rng(N * 100 + M)
    pos = rng.uniform(0, 2.5 * N ** (1 / 3) + 1, (N, 3))     # some pairs overlap
    rad = rng.uniform(0.8, 1.2, N)
    X = rng.standard_normal((3 * N, M)) + 1j * rng.standard_normal((3 * N, M))
    sc = rng.standard_normal((N, M)) + 1j
    F = capi.Field(capi.FIELD_DIRECT, radius=rad)
    F.set_positions(pos)
    t = lambda a: torch.tensor(a, dtype=torch.complex128, device="cuda")
    Y = F.apply(t(X), self_coef=t(sc), recip_fp32=fp32).cpu().numpy()
    ref = reference(pos, pos, rad, X, sc, True)
    tol = (2e-6 if fp32 else 4e-15) * max(4, N) ** 0.5
    assert np.abs(Y - ref).max() < tol * np.abs(ref).max()
    J = F.apply(t(X), self_coef=t(sc), jacobi=True, recip_fp32=fp32).cpu().numpy()
    want = (ref.reshape(N, 3, M) / sc[:, None, :]).reshape(3 * N, M)
    assert np.abs(J - want).max() < 4 * tol * np.abs(want).max()


@pytest.mark.parametrize("N,T", [(5, 70), (70, 5), (64, 9)])
def test_direct_field_points(N, T):
    from cumpm_b200 import capi

    rng = np.random.default_rng(N + T)
    pos, tgt = rng.uniform(0, 12, (N, 3)), rng.uniform(0, 12, (T, 3))
    rad = np.full(N, 0.7)
    X = rng.standard_normal((3 * N, 2)) + 1j * rng.standard_normal((3 * N, 2))
    F = capi.Field(capi.FIELD_DIRECT, radius=rad, mode=capi.MODE_INTERACTION)
    F.set_positions(pos)
    F.set_field_points(tgt)
    Y = F.apply(torch.tensor(X, dtype=torch.complex128, device="cuda")).cpu().numpy()
    ref = reference(pos, tgt, rad, X, None, False)
    assert np.abs(Y - ref).max() < 1e-13 * np.abs(ref).max()
