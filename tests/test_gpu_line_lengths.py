"""The mixed-radix line FFT at the lengths where its schedule changes: one,
two and three radices, the largest radices, large primes (alone, with a small
factor, two of them), along each axis, on the line passes and on the slab
passes built from it, against the float64 oracle.

Tolerance: float32 rounding u = 6e-8 grows as sqrt(terms) along a sum of a
large prime's q / 2 products and as sqrt(log2 n) along the other steps; a
subband makes two transforms of three axes, so the relative 2-norm error stays
below 2 u (sqrt(q) + 3 sqrt(log2 n)) < 5e-6 for every length here.
"""

import numpy as np
import pytest

from oracle import ns as N

TOL = 5e-6
LENGTHS = [2, 7, 17, 19, 20, 23, 29, 34, 45, 46, 77, 91, 100, 109, 125, 150, 200, 242, 250, 251, 437, 529, 667, 1000,
           2048]


@pytest.mark.gpu
@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("n", LENGTHS)
@pytest.mark.parametrize("pipeline", ["lines", "mixed"])
def test_line_lengths_match_oracle(sfl, n, axis, pipeline):
    dims = [6, 5, 8]
    dims[axis] = n
    dims = tuple(dims)
    x = np.random.default_rng(n).standard_normal(dims).astype(np.float32)
    ws = sfl.make_workspace(sfl.HourglassFB(bernstein_order=6), "float32", dims)
    if pipeline == "mixed" and n >= 1000:
        pytest.skip("tiles of this length leave no room for a slab")
    ws.set_pipeline(pipeline)
    bands = sfl.hourglass_decompose(ws, sfl.to_device(x))
    ref = N.hourglass_decompose(x, dims, 6, 1)
    for b, r in zip(bands, ref):
        assert np.linalg.norm(sfl.to_host(b) - r) <= TOL * max(np.linalg.norm(r), 1e-3 * np.linalg.norm(x))
    y = sfl.to_host(sfl.hourglass_reconstruct(ws, bands))
    assert np.linalg.norm(y - x) <= TOL * np.linalg.norm(x)


# the lengths compiled for the slab and axis-3 passes: products of two radices up to 16
TWO_RADIX = [n for n in range(16, 257) if any(n % a == 0 and 2 <= n // a <= 16 for a in range(2, 17))]


@pytest.mark.gpu
@pytest.mark.parametrize("n", TWO_RADIX)
def test_two_radix_lengths_match_oracle(sfl, n):
    for axis in range(3):
        dims = [18, 21, 16]
        dims[axis] = n
        dims = tuple(dims)
        x = np.random.default_rng(n + axis).standard_normal(dims).astype(np.float32)
        ws = sfl.make_workspace(sfl.HourglassFB(bernstein_order=6), "float32", dims)
        assert ws.tuning()[0] == "mixed"
        bands = sfl.hourglass_decompose(ws, sfl.to_device(x))
        for b, r in zip(bands, N.hourglass_decompose(x, dims, 6, 1)):
            assert np.linalg.norm(sfl.to_host(b) - r) <= TOL * max(np.linalg.norm(r), 1e-3 * np.linalg.norm(x))
        y = sfl.to_host(sfl.hourglass_reconstruct(ws, bands))
        assert np.linalg.norm(y - x) <= TOL * np.linalg.norm(x)
        # the denoiser at threshold 0 is the round trip, bit for bit
        z = sfl.to_host(sfl.denoise(ws, sfl.to_device(x), np.zeros(3, np.float32)))
        assert np.array_equal(z, y)
