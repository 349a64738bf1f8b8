"""Error against the float64 oracle, relative to what it was: the bars are the
rms errors measured with radix-2/3/4/5/8 line passes and one compensated step a
subband, on the same kind of input (standard normal; they vary by 0.3 % from one
input to the next)."""

import numpy as np
import pytest

from oracle import ns as N

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


# lengths of the radices 10, 15, 6 and 12: with twiddles inside those radices the errors were 2.49e-7, 2.47e-7, 2.45e-7
@pytest.mark.parametrize("dims,bar", [((100, 60, 20), 2.313e-7), ((120, 100, 90), 2.351e-7), ((150, 120, 60), 2.341e-7)])
def test_analysis_error_of_composite_radices(sfl, dims, bar):
    x = np.random.default_rng(6).standard_normal(dims).astype(np.float32)
    ws = sfl.make_workspace(sfl.NSSurfacelet(direction_levels=[1, 2]), "float32", dims)
    c = sfl.to_host(sfl.analyze(ws, sfl.to_device(x)))
    assert _rel(c, N.analyze(N.make_tables(N.NSParams.make(direction_levels=[1, 2]), dims), x)) <= bar
