"""Device memory of NSSurfacelet plans: a group that is set bounds the work
spectra, the default's own number too."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _held(sfl, dims, dtype, group):
    """Bytes a plan holds, before and after a bfloat16 call."""
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    before = torch.cuda.mem_get_info()[0]
    ws = sfl.make_workspace(sfl.NSSurfacelet(direction_levels=[2, 2, 3]), dtype, dims, group=group)
    first = before - torch.cuda.mem_get_info()[0]
    second = 0
    if dtype == "float32":
        sfl.analyze_bf16(ws, torch.zeros(dims[::-1], device="cuda").permute(2, 1, 0))
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        second = before - torch.cuda.mem_get_info()[0]
    tuning = ws.tuning()
    ws.close()
    return first, second, tuning


@pytest.mark.parametrize("dims,pipeline,dtype", [((64, 64, 64), "slabs", "float32"), ((64, 64, 64), "slabs", "complex64"),
                                                 ((60, 72, 60), "mixed", "float32")])
def test_a_set_group_bounds_the_work_spectra(sfl, dims, pipeline, dtype):
    _held(sfl, dims, dtype, None)   # loads the kernels
    spec = 8 * (dims[0] // 2 + 1) * dims[1] * dims[2] * (2 if dtype == "complex64" else 1)
    first, second, tuning = _held(sfl, dims, dtype, None)
    assert tuning == (pipeline, 8)
    for group in (8, 4):
        a, b, t = _held(sfl, dims, dtype, group)
        assert t == (pipeline, group)
        # 49 subbands: the default holds several times the group's spectra (allocations come in 2 MB blocks)
        assert first - a >= 20 * spec - (8 << 20)
        if second:
            assert second - b >= 20 * (spec + 4 * dims[0] * dims[1] * dims[2]) - (8 << 20)
