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


# axis 3 of two radices, of run-time radices, of a large prime; and the line pipeline
@pytest.mark.parametrize("dims,pipeline", [((32, 32, 32), "mixed"), ((40, 36, 60), "mixed"), ((24, 20, 34), "mixed"),
                                           ((20, 24, 37), "mixed"), ((32, 32, 32), "lines")])
def test_subbands_of_a_group_add_with_compensation(sfl, dims, pipeline):
    """The four wedges of hourglass 3 have the same mask where both transverse
    frequencies are zero.  Impulses at the origin transform exactly, so there
    the sum is m (2^24 + 3 x 0.45): each 0.45 m is at most 0.45 units in the
    last place of the first term and lost by plain additions, the three
    together are 0.67 to 1.35 units."""
    ws = sfl.make_workspace(sfl.NSSurfacelet(direction_levels=[2], bernstein_order=6), "float32", dims)
    ws.set_pipeline(pipeline)
    ops = sfl.LibRanges(ws)
    S = ws.nsubbands

    def spectrum(values):
        c = ops.new_subbands(S)
        c.zero_()
        for s, v in zip(range(10, 14), values):   # subbands of hourglass 3 (1-based), at their stream positions
            c[0, 0, 0, ops.stream_order.index(s)] = v
        A = ops.new_spectrum()
        ops.accumulate_range(c, 0, S, A, True)
        return A.reshape(dims[2], dims[1], -1)[:, 0, 0].real.cpu().numpy().astype(np.float64)

    one, all4 = spectrum([2.0 ** 24, 0, 0, 0]), spectrum([2.0 ** 24, 0.45, 0.45, 0.45])
    on = one > 1e-3 * one.max()
    assert on.sum() >= 4
    more = (all4 - one)[on]
    assert (more > 0).all()
    assert (np.abs(more - one[on] * 3 * 0.45 / 2 ** 24) <= np.spacing(one[on].astype(np.float32))).all()
