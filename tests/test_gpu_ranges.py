"""Item ranges added to a spectrum the caller holds: onto a zeroed spectrum
without `clear`, in the first call on a plan, over several ranges, and under
stream capture; with four accumulators, two and one, on every pipeline.

Tolerance: the ranges add the same terms as the plain synthesis, grouped
otherwise; their float32 sums differ by a few roundings (6e-8 each), bar 1e-6."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

CASES = [   # (n1 / 2 + 1) n2 up to 3000: four accumulators, up to 10000: two, above: one
    ((32, 32, 32), "mixed", "float32"),
    ((64, 64, 64), "slabs", "complex64"),
    ((128, 128, 32), "slabs", "float32"),
    ((120, 100, 18), "mixed", "complex64"),
    ((160, 160, 16), "slabs", "float32"),
    ((40, 36, 48), "lines", "complex64"),
]


def _fresh(sfl, dims, pipeline, dtype):
    """A workspace whose device memory last held NaN, and its subbands' volumes in stream order."""
    junk = torch.full((1 << 28,), float("nan"), device="cuda")
    torch.cuda.synchronize()
    del junk
    torch.cuda.empty_cache()
    t = sfl.NSSurfacelet(direction_levels=[1, 2], bernstein_order=6)
    ws = sfl.make_workspace(t, dtype, dims)
    if ws.tuning()[0] != pipeline:
        ws.set_pipeline(pipeline)
    rng = np.random.default_rng(5)
    c = rng.standard_normal(dims + (ws.nsubbands,)).astype(np.float32)
    if dtype == "complex64":
        c = (c + 1j * rng.standard_normal(c.shape)).astype(np.complex64)
    return ws, sfl.LibRanges(ws), sfl.to_device(c)


def _rel(a, b):
    return float(torch.linalg.vector_norm(a - b) / torch.linalg.vector_norm(b))


@pytest.mark.parametrize("dims,pipeline,dtype", CASES)
@pytest.mark.parametrize("clear_first", [False, True])
def test_ranges_add_to_a_held_spectrum(sfl, dims, pipeline, dtype, clear_first):
    ws, ops, c = _fresh(sfl, dims, pipeline, dtype)
    S = ws.nsubbands
    A, y = ops.new_spectrum(), ops.new_volume()
    A.fill_(float("nan") if clear_first else 0)
    for r in range(3):
        f, n = sfl.shard(S, 3, r)
        cr = sfl.as_colmajor(torch.stack([c[..., s - 1] for s in ops.stream_order[f:f + n]], -1))
        ops.accumulate_range(cr, f, n, A, clear_first and r == 0)
    kept = A.clone()
    ops.accumulate_range(cr, 0, 0, A, False)   # an empty range leaves the spectrum alone
    assert torch.equal(A, kept)
    ops.inverse_spectrum(A, y)
    assert _rel(y, sfl.synthesize(ws, c)) <= 1e-6


@pytest.mark.parametrize("dims,pipeline,dtype", CASES)
def test_first_range_of_a_plan_under_capture(sfl, dims, pipeline, dtype):
    warm, wops, c = _fresh(sfl, dims, pipeline, dtype)   # another plan of the size loads the kernels
    ws, ops, _ = _fresh(sfl, dims, pipeline, dtype)
    S = ws.nsubbands
    call = sfl.as_colmajor(torch.stack([c[..., s - 1] for s in ops.stream_order], -1))
    A, B, y = ops.new_spectrum(), ops.new_spectrum(), ops.new_volume()
    wops.accumulate_range(call, 0, S, B, True)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        ops.accumulate_range(call, 0, S, A, True)
    A.fill_(float("nan"))
    g.replay()
    assert torch.equal(A, B)
    ops.inverse_spectrum(A, y)
    assert _rel(y, sfl.synthesize(ws, c)) <= 1e-6
