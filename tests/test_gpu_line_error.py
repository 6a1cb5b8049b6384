"""Rounding errors of the line transforms whose prime part is a product with
cosine and sine tables (mpm_dense.cu), against numpy in more bits.  A rounding
is at most u, of variance u^2 / 3 of its value.  Of a sum of H terms the partial
sums have variance q = 1 .. H of a term's:
* fp32, sums of 20 terms and then the sum of those B = H / 20: (20 + 1) / 2 + B / 2
  roundings of a term per term, and two more for the pair's sum and the table;
* fp64, one sum: H / 2, and two more; a table entry from an angle rounded to 64
  bits would bring in about two more by itself, and the twiddles likewise.
The relative rms error is at most u sqrt(roundings / 3)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


def rms_error(n, fp64, ncols=18, nouter=48):
    from cumpm_b200 import capi

    rng = np.random.default_rng(n)
    a = rng.standard_normal((nouter, n, ncols)) + 1j * rng.standard_normal((nouter, n, ncols))
    a = a.astype(np.complex128 if fp64 else np.complex64)
    ref = np.fft.fft(a.astype(np.clongdouble if fp64 else np.complex128), axis=1)
    d = torch.tensor(a, device="cuda").contiguous()
    assert capi.line_fft(d, n, ncols, ncols, n * ncols, nouter) == (1, n)
    return float(np.linalg.norm(d.cpu().numpy() - ref) / np.linalg.norm(ref))


@pytest.mark.parametrize("n", [109, 151, 199, 251, 277])
def test_fp32_product_sums_in_blocks(n):
    H = n // 2
    assert rms_error(n, False) < 2.0 ** -24 * np.sqrt((10.5 + H / 40 + 2) / 3)


@pytest.mark.parametrize("n", [37, 61, 109])
def test_fp64_tables_hold_all_their_digits(n):
    H = n // 2
    assert rms_error(n, True) < 2.0 ** -53 * np.sqrt((H / 2 + 3) / 3)
