"""Line transforms by Rader's convolution (mpm_rader.cu: long primes, with a
radix in front or without) against numpy, at the lengths on both sides of the
rule that chooses them, in both directions, with column groups that are partly
empty, and with the fused scale and few columns, which other kernels take.
Tolerance: no stage sums more than 16 terms and there are seven, so the error is
at most sqrt(7 * 16) roundings of the result's root mean square."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fp64", [False, True])
@pytest.mark.parametrize("n,split", [(131, (1, 131)), (181, (1, 181)), (211, (1, 211)), (257, (1, 257)),
                                     (302, (2, 151)), (362, (2, 181)), (386, (2, 193)), (514, (2, 257)),
                                     (1965, (15, 131))])
def test_rader_transform(n, split, fp64):
    from cumpm_b200 import capi

    eps = 2.0 ** -53 if fp64 else 2.0 ** -24
    rng = np.random.default_rng(n)
    for ncols, nouter, layout in ((16, 3, "z"), (17, 2, "x"), (33, 2, "z"), (5, 3, "x")):
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
            got = capi.line_fft(d, n, es, ncols, os, nouter, mode=mode, scale=s if mode == 2 else None, sz=ncols, sb=1)
            assert got == split, (ncols, mode, got)
            err = np.linalg.norm(d.cpu().numpy() - ref) / np.linalg.norm(ref)
            assert err < np.sqrt(7 * 16) * np.sqrt(2 if mode == 2 else 1) * eps, (layout, ncols, nouter, mode, err)
