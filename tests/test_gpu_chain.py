"""Kernels scheduled while their predecessor still runs: operator applications
queued back to back, each on inputs that the launch just before it wrote and
with the last one's inputs overwritten right behind it, are bit for bit what
they are with a synchronisation around each; on the default stream and on one
of the caller's, and two operators on two streams at once."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


def operator(kind):
    from cumpm_b200 import capi

    rng = np.random.default_rng(1)
    k, n = 4, 64
    g = np.stack(np.meshgrid(*[np.arange(k)] * 3, indexing="ij"), axis=-1).reshape(-1, 3)
    pos = g * 4.5 + 1.0 + rng.uniform(-0.3, 0.3, (n, 3))
    box = np.full(3, 18.0)
    if kind == "poly":
        F = capi.Field(capi.FIELD_POLY, box, 1e-4, 0.5, radius=rng.uniform(1.0, 1.4, n))
    elif kind == "layer":
        pos = np.concatenate([g[:, :2] * 4.0 + 1.0 + 16.0 * (g[:, 2:] % 2) * [1, 0]
                              + 16.0 * (g[:, 2:] // 2) * [0, 1], np.zeros((n, 1))], axis=1)
        F = capi.Field(capi.FIELD_MONO, np.array([32.0, 32.0, 150.0]), 1e-4, 0.5)
    else:
        F = capi.Field(capi.FIELD_MONO, box, 1e-4, 0.5)
    F.set_positions(pos)
    return F, n


def chain(F, X, S, fp32, steps, sync):
    out = []
    buf = torch.empty_like(X)
    for k in range(steps):
        torch.mul(X, 1.0 + 0.125 * k, out=buf)
        if sync:
            torch.cuda.synchronize()
        out.append(F.apply(buf, self_coef=S, recip_fp32=fp32))
        if sync:
            torch.cuda.synchronize()
        buf.fill_(float("nan"))
    torch.cuda.synchronize()
    return torch.stack(out)


@pytest.mark.parametrize("M", [1, 3, 20])
@pytest.mark.parametrize("fp32", [False, True])
@pytest.mark.parametrize("kind", ["mono", "layer", "poly"])
def test_back_to_back_applications(kind, fp32, M):
    rng = np.random.default_rng(M)
    F, n = operator(kind)
    X = torch.tensor(rng.standard_normal((3 * n, M)) + 1j * rng.standard_normal((3 * n, M)), device="cuda")
    S = torch.tensor(rng.standard_normal((n, M)) + 1j * rng.standard_normal((n, M)), device="cuda")
    ref = chain(F, X, S, fp32, 6, True)
    assert torch.isfinite(torch.view_as_real(ref)).all()
    assert torch.equal(chain(F, X, S, fp32, 6, False), ref)
    torch.cuda.synchronize()
    st = [torch.cuda.Stream(), torch.cuda.Stream()]
    G, _ = operator(kind)
    res = []
    for f, s in ((F, st[0]), (G, st[1])):
        with torch.cuda.stream(s):
            buf = X * 1.0
            res.append([f.apply(buf, self_coef=S, recip_fp32=fp32) for _ in range(4)])
            buf.fill_(float("nan"))
    torch.cuda.synchronize()
    for r in res:
        for y in r:
            assert torch.equal(y, ref[0])
