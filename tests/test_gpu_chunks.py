"""Launch chunks of the slab pipeline that span mask groups: equal bit for bit
to chunks of one mask group each (a group size that leaves the mask groups
whole and the work slots at that size), real and complex, analysis, synthesis
and the denoiser.  No tolerance: the terms, their order and the Kahan steps
are the same."""

import numpy as np
import pytest
import torch


@pytest.mark.gpu
@pytest.mark.parametrize("dims,levels,dtype", [
    ((64, 64, 64), [2, 2, 3], "float32"),          # every subband in one chunk
    ((128, 128, 128), [2, 2, 3], "float32"),       # chunks of several small boxes, then one group each
    ((64, 96, 32), [1, 1, 1, 3], "float32"),       # more mask groups than scales share a box
    ((96, 64, 64), [1, 2], "complex64"),
    ((64, 64, 16), [4, 4], "float32"),             # mask groups of more than 8 subbands split at 8
])
def test_chunks_do_not_change_results(sfl, dims, levels, dtype):
    rng = np.random.default_rng(3)
    x = rng.standard_normal(dims).astype(np.float32)
    if dtype == "complex64":
        x = (x + 1j * rng.standard_normal(dims)).astype(np.complex64)
    x = sfl.to_device(x)
    t = sfl.NSSurfacelet(direction_levels=levels, bernstein_order=6)
    a = sfl.make_workspace(t, dtype, dims)
    assert a.tuning() == ("slabs", 8)
    b = sfl.make_workspace(t, dtype, dims, group=9 if max(levels) < 4 else 8)
    if max(levels) < 4:
        assert b.tuning() == ("slabs", 9)
    ca, cb = sfl.analyze(a, x), sfl.analyze(b, x)
    assert torch.equal(ca, cb)
    assert torch.equal(sfl.synthesize(a, ca), sfl.synthesize(b, ca))
    assert torch.equal(sfl.adjoint_synthesize(a, x), sfl.adjoint_synthesize(b, x))
    if dtype == "float32":
        assert torch.equal(sfl.denoise(a, x, 0.3), sfl.denoise(b, x, 0.3))
