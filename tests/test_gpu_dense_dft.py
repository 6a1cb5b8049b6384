"""Line transforms by table products (mpm_dense.cu) against numpy in 64 bits,
at the sizes where they can go wrong: one and two points per product, even
middles, the longest product in one sum and the first in blocks (47, 53 points),
tables that stay in global memory (m above 191, in fp64 127), radices up to 16 in
front, composite rests (260, 286, 352; 1144 = 13 * 88), columns that do not fill a tile, and few columns per line (lines and
columns enumerated together).  Tolerance: a product sums m / 2 rounded terms, so
its error is at most about sqrt(m) roundings of the result's root mean square."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fp64", [False, True])
@pytest.mark.parametrize("n", [3, 17, 22, 47, 53, 84, 109, 131, 137, 251, 260, 272, 286, 352, 366, 1144])
def test_product_transform(n, fp64):
    from cumpm_b200 import capi

    eps = 2.0 ** -53 if fp64 else 2.0 ** -24
    rng = np.random.default_rng(n)
    for ncols, nouter in ((1, 1), (3, 7), (9, 40), (70, 3)):
        for layout in ("z", "x"):
            shape, axis = ((nouter, n, ncols), 1) if layout == "z" else ((n, nouter, ncols), 0)
            es, os = (ncols, n * ncols) if layout == "z" else (nouter * ncols, ncols)
            a = rng.standard_normal(shape) + 1j * rng.standard_normal(shape)
            a = a.astype(np.complex128 if fp64 else np.complex64)
            sc = rng.uniform(0.5, 1.5, (n, nouter, ncols)).astype(np.float64 if fp64 else np.float32)
            f = np.fft.fft(a.astype(np.complex128), axis=axis)
            fac = sc.transpose(1, 0, 2) if layout == "z" else sc
            for mode, ref in ((0, f), (1, np.fft.ifft(a.astype(np.complex128), axis=axis) * n),
                              (2, np.fft.ifft(f * fac, axis=axis) * n)):
                d = torch.tensor(a, device="cuda").contiguous()
                s = torch.tensor(sc, device="cuda").contiguous()
                capi.line_fft(d, n, es, ncols, os, nouter, mode=mode, scale=s if mode == 2 else None, sz=ncols, sb=1)
                err = np.linalg.norm(d.cpu().numpy() - ref) / np.linalg.norm(ref)
                assert err < 4 * np.sqrt(n) * eps, (layout, ncols, nouter, mode, err)
