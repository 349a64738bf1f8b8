"""Transposes of the decimated transform where a plane of two axes does not fit
shared memory, so that the hourglass across it runs a launch per checkerboard
stage while the others take the plane pass: against the float64 oracle's
forward operators, as dot products and at single points.

The bars are those of the transposes on small planes: 2e-5 on dot products of
correlated vectors, 1e-5 of the vector's rms at a point (float32 rounding
measures 3e-7)."""

import numpy as np
import pytest

from oracle import decimated as D

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,levels", [((256, 128, 16), [2]), ((256, 16, 128), [1]), ((16, 256, 128), [2]),
                                         ((128, 256, 32), [1, 2]), ((240, 144, 24), [1])])
def test_transposes_across_large_planes(sfl, dims, levels):
    kw = dict(scales=len(levels), direction_levels=levels, pyramid_ratio=1.5 if dims[0] == 240 else 2, checkerboard_order=8)
    T = D.make_tables(D.SurfParams.make(**kw), dims)
    ws = sfl.make_workspace(sfl.Surfacelet(**kw), "float32", dims)
    rng = np.random.default_rng(12)
    x = rng.standard_normal(dims).astype(np.float32)
    Ax = D.analyze(T, x.astype(np.float64))
    c = (Ax + rng.standard_normal(Ax.shape)).astype(np.float32)
    Atc = sfl.to_host(sfl.adjoint_analyze(ws, sfl.to_device(c), dims=dims)).astype(np.float64)
    lhs = float(np.dot(Ax, c))
    assert abs(lhs - float(np.sum(x * Atc))) <= 2e-5 * abs(lhs)
    cc = rng.standard_normal(Ax.shape).astype(np.float32)
    Sc = D.synthesize(T, cc.astype(np.float64))
    y = (Sc + rng.standard_normal(dims)).astype(np.float32)
    Sty = sfl.adjoint_synthesize(ws, sfl.to_device(y)).cpu().numpy().astype(np.float64)
    lhs = float(np.sum(Sc * y))
    assert abs(lhs - float(np.dot(cc, Sty))) <= 2e-5 * abs(lhs)
    for _ in range(2):   # A^T c at a point, S^T y at a coefficient
        at = tuple(int(rng.integers(n)) for n in dims)
        e = np.zeros(dims)
        e[at] = 1
        assert abs(float(np.dot(D.analyze(T, e), c)) - Atc[at]) <= 1e-5 * np.sqrt(np.mean(Atc ** 2))
        i = int(rng.integers(Ax.size))
        e = np.zeros(Ax.shape)
        e[i] = 1
        assert abs(float(np.sum(D.synthesize(T, e) * y)) - Sty[i]) <= 1e-5 * np.sqrt(np.mean(Sty ** 2))
