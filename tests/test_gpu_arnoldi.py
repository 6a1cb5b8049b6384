"""GMRES around the Arnoldi step's two forms (fewer than 16 columns: three
launches whose last CTAs reduce and finish; more: one kernel per pass), the
back substitution and the shifted solve's member updates: every column's
solution against a dense solve, over column counts on both sides of the line
and of the reductions' lane groups, restarts that do and do not end a cycle
early, and a zero right-hand side."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


def problem(N, M, seed, zero=False):
    rng = np.random.default_rng(seed)
    pos = np.stack(np.meshgrid(*[np.arange(5)] * 3), axis=-1).reshape(-1, 3)[:N] * 2.4 + rng.uniform(-0.15, 0.15, (N, 3))
    eps = (4 - 1.8 ** 2 / (np.linspace(0.35, 0.9, M) ** 2 + 0.1j * np.linspace(0.35, 0.9, M))) / 1.77
    sc = np.repeat((3 / (4 * np.pi * (eps - 1)))[None, :], N, axis=0)
    B = rng.standard_normal((3 * N, M)) + 1j * rng.standard_normal((3 * N, M))
    if zero:
        B[:, M // 2] = 0
    A0 = np.zeros((3 * N, 3 * N))
    for j in range(N):
        for i in range(N):
            if i != j:
                r = pos[i] - pos[j]
                d = np.linalg.norm(r)
                A0[3 * j:3 * j + 3, 3 * i:3 * i + 3] = -(3 * np.outer(r, r) / d ** 2 - np.eye(3)) / d ** 3 / (4 * np.pi)
    X = np.stack([np.linalg.solve(A0 + np.diag(np.repeat(sc[:, m] + 1 / (4 * np.pi), 3)), B[:, m]) for m in range(M)],
                 axis=1)
    return pos, sc, B, X


@pytest.mark.parametrize("restart", [4, 12, 50])
@pytest.mark.parametrize("M", [1, 2, 3, 5, 8, 9, 15, 16, 33])
def test_columns_against_dense(M, restart):
    from cumpm_b200 import capi

    N = 40
    pos, sc, B, ref = problem(N, M, 10 * M + restart, zero=M > 4)
    F = capi.Field(capi.FIELD_DIRECT, radius=np.ones(N))
    F.set_positions(pos)
    t = lambda a: torch.tensor(a, dtype=torch.complex128, device="cuda")
    X = torch.zeros((3 * N, M), dtype=torch.complex128, device="cuda")
    r = F.batch_solve(t(B), X, t(sc), tol=1e-11, restart=restart, maxiter=3000, recip_fp32=False)
    assert r["num_converged"] == M
    err = np.abs(X.cpu().numpy() - ref).max() / np.abs(ref).max()
    assert err < 1e-8, err


@pytest.mark.parametrize("W", [2, 6, 20])
def test_shifted_members_against_dense(W):
    """One material, shared right-hand sides: W frequencies on three seeds."""
    from cumpm_b200 import capi

    N = 60
    pos, sc, _, _ = problem(N, W, W)
    M = 3 * W
    S = np.repeat(sc, 3, axis=1)
    B = np.zeros((3 * N, M), complex)
    for m in range(M):
        B[m % 3::3, m] = 1
    box = np.array([40.0, 40.0, 40.0])
    F = capi.Field(capi.FIELD_MONO, box, 1e-8, 0.5)
    F.set_positions(pos)
    t = lambda a: torch.tensor(a, dtype=torch.complex128, device="cuda")
    X = torch.zeros((3 * N, M), dtype=torch.complex128, device="cuda")
    r = F.batch_solve(t(B), X, t(S), tol=1e-8, refine=True)
    assert r["num_converged"] == M and r["shift_seeds"] == 3
    Y = torch.zeros_like(X)
    F.batch_solve(t(B), Y, t(S), tol=1e-12, recip_fp32=False, shifted=False, maxiter=3000)
    assert (X - Y).abs().max().item() < 1e-6 * Y.abs().max().item()
