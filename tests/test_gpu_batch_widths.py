"""Every column of a batched operator application against the column applied
alone: the spread, contraction and pair kernels choose lane groups, columns per
CTA and chunks by the batch width, so the widths here lie on both sides of each
line.  Sums of one column run in another order for other widths; tolerance: a
few hundred rounded terms."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

WIDTHS = [2, 3, 4, 5, 6, 8, 9, 11, 16, 17, 33, 49, 97]


def packing(n, L, seed):
    rng = np.random.default_rng(seed)
    k = int(np.ceil(n ** (1 / 3)))
    g = np.stack(np.meshgrid(*[np.arange(k)] * 3, indexing="ij"), axis=-1).reshape(-1, 3)[:n]
    return (g + 0.5) * (L / k) + rng.uniform(-0.2, 0.2, (n, 3))


def check(F, rows, n, fp32, seed, widths=WIDTHS):
    rng = np.random.default_rng(seed)
    M = max(widths)
    X = torch.tensor(rng.standard_normal((rows, M)) + 1j * rng.standard_normal((rows, M)), device="cuda")
    S = torch.tensor(rng.standard_normal((n, M)) + 1j * rng.standard_normal((n, M)), device="cuda")
    col = lambda t, m: t[:, m:m + 1].contiguous()
    alone = torch.cat([F.apply(col(X, m), self_coef=col(S, m), recip_fp32=fp32) for m in range(M)], dim=1)
    tol = (1e-6 if fp32 else 2e-14) * alone.abs().max().item()
    for w in widths:
        Y = F.apply(X[:, :w].contiguous(), self_coef=S[:, :w].contiguous(), recip_fp32=fp32)
        assert (Y - alone[:, :w]).abs().max().item() < tol, w


@pytest.mark.parametrize("fp32", [False, True])
def test_polydisperse(fp32):
    from cumpm_b200 import capi

    n, L = 60, 19.0
    rad = np.random.default_rng(3).uniform(1.0, 1.4, n)
    F = capi.Field(capi.FIELD_POLY, np.full(3, L), 1e-5, 0.5, radius=rad)
    F.set_positions(packing(n, L, 4))
    check(F, 3 * n, n, fp32, 5)


@pytest.mark.parametrize("fp32", [False, True])
@pytest.mark.parametrize("layout", ["cube", "slab", "layer"])
def test_monodisperse(layout, fp32):
    from cumpm_b200 import capi

    n = 64
    if layout == "cube":
        box, pos = np.array([17.0, 18.0, 19.0]), packing(n, 17.0, 6)
    else:
        box = np.array([24.0, 21.0, 150.0])
        rng = np.random.default_rng(7)
        g = np.stack(np.meshgrid(np.arange(8), np.arange(8), indexing="ij"), axis=-1).reshape(-1, 2)
        pos = np.concatenate([g * [3.0, 2.6] + rng.uniform(-0.2, 0.2, (n, 2)), np.zeros((n, 1))], axis=1)
        if layout == "slab":
            pos[:, 2] = rng.uniform(-0.6, 0.6, n)
    F = capi.Field(capi.FIELD_MONO, box, 1e-6, 0.5)
    F.set_positions(pos)
    info = F.info()
    assert bool(info["pruned"]) == (layout != "cube") and bool(info["single_layer"]) == (layout == "layer")
    check(F, 3 * n, n, fp32, 8)


@pytest.mark.parametrize("fp32", [False, True])
def test_quadrupoles(fp32):
    from cumpm_b200 import capi

    n = 40
    F = capi.Field(capi.FIELD_MONO, np.array([16.0, 16.5, 17.0]), 1e-6, 0.5, quad_idxs=np.arange(0, n, 2))
    F.set_positions(packing(n, 16.0, 9))
    check(F, 3 * n + 5 * (n // 2), n, fp32, 10, widths=[2, 3, 5, 9, 17, 33])
