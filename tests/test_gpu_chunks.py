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


@pytest.mark.gpu
@pytest.mark.parametrize("dims", [(16, 18, 20), (17, 19, 21), (32, 32, 32)])
def test_bf16_packing_is_the_float_subbands_rounded(sfl, dims):
    """Four values a step (volumes of a multiple of four) and one: exact, since
    packing rounds the float32 subband by its power-of-two scale once."""
    x = sfl.to_device(np.random.default_rng(4).standard_normal(dims).astype(np.float32))
    ws = sfl.make_workspace(sfl.NSSurfacelet(direction_levels=[1, 2], bernstein_order=6), "float32", dims)
    c = sfl.analyze(ws, x)
    q, scales = sfl.analyze_bf16(ws, x)
    peak = c.abs().amax((0, 1, 2))
    assert torch.equal(scales, torch.ldexp(torch.ones_like(peak), torch.frexp(peak)[1]))
    assert torch.equal(q, (c / scales).to(torch.bfloat16))
    y = sfl.synthesize_bf16(ws, q, scales)
    assert torch.equal(y, sfl.synthesize(ws, sfl.as_colmajor(q.float() * scales)))
