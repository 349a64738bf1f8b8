"""The pipeline a plan starts with, and the ones that can be selected: a long
axis beside lengths with compile-time line passes takes lines (where the mixed
pipeline is slower), other lengths the mixed pipeline where the slabs fit;
either gives the same subbands."""

import numpy as np
import pytest
import torch

from oracle import ns as N

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,default", [
    ((256, 20, 32), "mixed"), ((258, 32, 32), "lines"), ((258, 20, 32), "mixed"), ((32, 257, 16), "lines"),
    ((16, 32, 512), "mixed"), ((16, 32, 513), "lines"), ((16, 18, 513), "mixed"), ((512, 64, 32), "lines"),
    ((32, 400, 32), "lines"), ((16, 16, 1000), "lines"), ((64, 64, 64), "slabs"), ((250, 250, 20), "lines"),
])
def test_default_pipeline(sfl, dims, default):
    t = sfl.NSSurfacelet(direction_levels=[1], bernstein_order=4)
    ws = sfl.make_workspace(t, "float32", dims)
    assert ws.tuning()[0] == default
    if default == "slabs" or dims[:2] == (250, 250):
        return
    other = sfl.make_workspace(t, "float32", dims)
    other.set_pipeline("lines" if default == "mixed" else "mixed")   # both stay selectable
    x = sfl.to_device(np.random.default_rng(3).standard_normal(dims).astype(np.float32))
    a, b = sfl.analyze(ws, x), sfl.analyze(other, x)
    # two orders of the same float32 transform: each within about 3e-7 of 64 bits
    assert float(torch.linalg.vector_norm(a - b) / torch.linalg.vector_norm(a)) <= 1e-6
    y, z = sfl.synthesize(ws, a), sfl.synthesize(other, a)
    assert float(torch.linalg.vector_norm(y - z) / torch.linalg.vector_norm(y)) <= 1e-6


@pytest.mark.parametrize("dims", [(1000, 8, 8), (10, 600, 12), (12, 6, 520), (521, 8, 10), (8, 8, 541), (258, 34, 6)])
def test_long_lines_in_small_tiles(sfl, dims):
    """Few long lines run in tiles of one to eight lines: against the float64
    oracle, bar 1e-5 (float32 rounding measures 2e-7 to 5e-7)."""
    kw = dict(direction_levels=[1], bernstein_order=4)
    rng = np.random.default_rng(8)
    x = rng.standard_normal(dims).astype(np.float32)
    T = N.make_tables(N.NSParams.make(**kw), dims)
    ws = sfl.make_workspace(sfl.NSSurfacelet(**kw), "float32", dims)
    ws.set_pipeline("lines")
    ref = N.analyze(T, x)
    c = rng.standard_normal(ref.shape).astype(np.float32)
    assert np.linalg.norm(sfl.to_host(sfl.analyze(ws, sfl.to_device(x))) - ref) <= 1e-5 * np.linalg.norm(ref)
    y = N.synthesize(T, c)
    assert np.linalg.norm(sfl.to_host(sfl.synthesize(ws, sfl.to_device(c))) - y) <= 1e-5 * np.linalg.norm(y)


@pytest.mark.parametrize("n3", [6, 18, 20, 27, 34, 40, 45, 60, 63, 75, 90, 108, 143, 150, 208, 225])
def test_masked_lines_of_two_radices(sfl, n3):
    """The line pipeline's masked axis-3 pass takes the smaller radix first:
    against the float64 oracle (bar 1e-5), ragged counts of lines."""
    dims, kw = (22, 18, n3), dict(direction_levels=[1], bernstein_order=4)
    x = np.random.default_rng(9).standard_normal(dims).astype(np.float32)
    ws = sfl.make_workspace(sfl.NSSurfacelet(**kw), "float32", dims)
    ws.set_pipeline("lines")
    ref = N.analyze(N.make_tables(N.NSParams.make(**kw), dims), x)
    assert np.linalg.norm(sfl.to_host(sfl.analyze(ws, sfl.to_device(x))) - ref) <= 1e-5 * np.linalg.norm(ref)


@pytest.mark.parametrize("dims,levels", [((64, 200, 20), [1, 2]), ((34, 18, 12), [1]), ((17, 13, 19), [1]), ((109, 34, 16), [2]),
                                         ((20, 111, 18), [1, 2]), ((200, 96, 16), [1, 3]), ((12, 14, 10), [1])])
def test_denoiser_of_run_time_slabs(sfl, dims, levels):
    """Slabs of run-time radices threshold into the spectrum's own block between
    two passes: bit for bit the three calls, odd counts of columns among them."""
    ws = sfl.make_workspace(sfl.NSSurfacelet(direction_levels=levels, bernstein_order=4), "float32", dims)
    assert ws.tuning()[0] == "mixed"
    x = sfl.to_device(np.random.default_rng(10).standard_normal(dims).astype(np.float32))
    c = sfl.analyze(ws, x)
    s = torch.sign(c) * (c.abs() - 0.1).clamp(min=0)
    s[..., 0] = c[..., 0]
    y = sfl.denoise(ws, x, 0.1)
    assert torch.equal(y, sfl.synthesize(ws, sfl.as_colmajor(s)))
    assert torch.equal(y, sfl.denoise(ws, x, 0.1))


@pytest.mark.parametrize("dims,dtype", [((64, 64, 160), "float32"), ((64, 64, 96), "complex64"), ((96, 96, 96), "complex64"),
                                        ((30, 20, 96), "float32"), ((128, 64, 160), "float32")])
def test_accumulators_summed_ahead_of_the_inverse(sfl, dims, dtype):
    """Two and four accumulators with 96 and 160 points along axis 3: against the
    line pipeline's one (a few float32 roundings apart, bar 1e-6), and streamed
    bit for bit."""
    rng = np.random.default_rng(11)
    t = sfl.NSSurfacelet(direction_levels=[1, 2], bernstein_order=6)
    ws, wl = sfl.make_workspace(t, dtype, dims), sfl.make_workspace(t, dtype, dims)
    wl.set_pipeline("lines")
    c = rng.standard_normal(dims + (ws.nsubbands,)).astype(np.float32)
    if dtype == "complex64":
        c = (c + 1j * rng.standard_normal(c.shape)).astype(np.complex64)
    c = sfl.to_device(c)
    y, z = sfl.synthesize(ws, c), sfl.synthesize(wl, c)
    assert float(torch.linalg.vector_norm(y - z) / torch.linalg.vector_norm(z)) <= 1e-6
    s = sfl.volume_like(dims, dtype)
    sfl.synthesize_(lambda i: c[..., i - 1], s, ws)
    assert torch.equal(s, y)
