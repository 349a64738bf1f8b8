"""The slab pipeline on the mixed-radix FFT ("mixed", the default for sizes
without compile-time slabs): against the float64 oracle at odd, ragged and
prime sizes, small and wide boxes, tight and not; and its equalities bit for
bit: streaming, item ranges, complex data as two channels, the denoiser.

Tolerance against the oracle: the transform's own 1e-5 bar (float32 rounding
measures 2e-7 to 5e-7 here)."""

import numpy as np
import pytest
import torch

from oracle import ns as N

pytestmark = pytest.mark.gpu

CASES = [
    ((20, 12, 18), dict(direction_levels=[1, 2], bernstein_order=6)),
    ((15, 21, 9), dict(direction_levels=[2], bernstein_order=6)),
    ((33, 34, 35), dict(direction_levels=[1, 3], bernstein_order=6)),              # odd pairs, a factor 17
    ((46, 29, 31), dict(direction_levels=[1, 2], bernstein_order=6)),              # large primes on every axis
    ((48, 80, 40), dict(direction_levels=[1, 2, 3], bernstein_order=8)),
    ((100, 60, 20), dict(direction_levels=[1, 2], bernstein_order=8, tight=False)),
    ((32, 32, 32), dict(direction_levels=[2, 2, 3])),                              # coarse boxes of a few rows
    ((200, 24, 16), dict(direction_levels=[1, 5], bernstein_order=4)),             # mask groups above 8 subbands
    ((17, 200, 24), dict(direction_levels=[1, 1], bernstein_order=4)),
]


def rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


@pytest.mark.parametrize("dims,kw", CASES)
def test_mixed_matches_oracle(sfl, dims, kw):
    rng = np.random.default_rng(1)
    x = rng.standard_normal(dims).astype(np.float32)
    T = N.make_tables(N.NSParams.make(**kw), dims)
    ws = sfl.make_workspace(sfl.NSSurfacelet(**kw), "float32", dims)
    assert ws.tuning()[0] == "mixed"
    c = sfl.to_host(sfl.analyze(ws, sfl.to_device(x)))
    ref = N.analyze(T, x)
    for i in range(ref.shape[-1]):
        assert np.linalg.norm(c[..., i] - ref[..., i]) <= 1e-5 * max(np.linalg.norm(ref[..., i]), 1e-3 * np.linalg.norm(x))
    cr = rng.standard_normal(ref.shape).astype(np.float32)
    cd = sfl.to_device(cr)
    assert rel(sfl.to_host(sfl.synthesize(ws, cd)), N.synthesize(T, cr)) <= 1e-5
    assert rel(sfl.to_host(sfl.adjoint_analyze(ws, cd)), N.adjoint_analyze(T, cr)) <= 1e-5
    assert rel(sfl.to_host(sfl.adjoint_synthesize(ws, sfl.to_device(x))), N.adjoint_synthesize(T, x)) <= 1e-5


@pytest.mark.parametrize("dims,levels", [((20, 12, 18), [1, 2]), ((33, 34, 35), [1, 3]), ((48, 80, 40), [2, 2, 3]),
                                         ((128, 100, 64), [2, 3])])
def test_mixed_equalities(sfl, dims, levels):
    rng = np.random.default_rng(2)
    t = sfl.NSSurfacelet(direction_levels=levels, bernstein_order=6)
    xr, xi = (rng.standard_normal(dims).astype(np.float32) for _ in range(2))
    ws, wc = sfl.make_workspace(t, "float32", dims), sfl.make_workspace(t, "complex64", dims)
    assert ws.tuning()[0] == "mixed" and wc.tuning()[0] == "mixed"
    x = sfl.to_device(xr)
    c = sfl.analyze(ws, x)
    y = sfl.synthesize(ws, c)
    # streaming
    bands = {}
    sfl.analyze(lambda i, b: bands.__setitem__(i, b.clone()), ws, x)
    assert all(torch.equal(bands[i], c[..., i - 1]) for i in bands) and len(bands) == ws.nsubbands
    ys = sfl.volume_like(dims)
    sfl.synthesize_(lambda i: bands[i], ys, ws)
    assert torch.equal(ys, y)
    # complex data are two real channels
    cc = sfl.analyze(wc, sfl.to_device((xr + 1j * xi).astype(np.complex64)))
    ci = sfl.analyze(ws, sfl.to_device(xi))
    assert torch.equal(cc.real, c) and torch.equal(cc.imag, ci)
    yc = sfl.synthesize(wc, cc)
    assert torch.equal(yc.real, y) and torch.equal(yc.imag, sfl.synthesize(ws, ci))
    # the denoiser is its three calls
    cs = torch.sign(c) * (c.abs() - 0.2).clamp(min=0)
    cs[..., 0] = c[..., 0]
    assert torch.equal(sfl.denoise(ws, x, 0.2), sfl.synthesize(ws, sfl.as_colmajor(cs)))
    # item ranges
    ops = sfl.LibRanges(ws)
    X, A, yr = ops.new_spectrum(), ops.new_spectrum(), ops.new_volume()
    ops.forward_spectrum(x, X)
    cr = ops.new_subbands(ws.nsubbands)
    ops.analyze_range(X, 0, ws.nsubbands, cr)
    ops.accumulate_range(cr, 0, ws.nsubbands, A, True)
    ops.inverse_spectrum(A, yr)
    assert torch.equal(yr, y)
    # the line pipeline to rounding
    wl = sfl.make_workspace(t, "float32", dims)
    wl.set_pipeline("lines")
    d = sfl.analyze(wl, x) - c
    assert float(d.norm() / c.norm()) <= 1e-6


def test_sizes_whose_slabs_do_not_fit_take_lines(sfl):
    ws = sfl.make_workspace(sfl.NSSurfacelet(direction_levels=[1], bernstein_order=4), "float32", (300, 250, 8))
    assert ws.tuning()[0] == "lines"
    with pytest.raises(sfl.ArgumentError, match="mixed-radix slab pipeline does not support"):
        ws.set_pipeline("mixed")
