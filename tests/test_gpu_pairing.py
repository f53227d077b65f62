"""Launches on either side of the rules that choose the vectors a lane and the segments
of a lone plane: samples within the segments' 4e-7 of the largest magnitude (1 code) of
whole vectors'."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = [("bicubic", 1920, 1080, 1, "f32"), ("bicubic", 1920, 1080, 2, "f32"), ("lanczos", 3840, 2160, 1, "f32"),
         ("bilinear", 1920, 1080, 5, "f32"), ("bilinear", 3840, 2160, 24, "f32"), ("lanczos", 1920, 1080, 2, "u16"),
         ("bicubic", 4100, 2050, 1, "f32")]


@pytest.mark.parametrize("kernel,w,h,planes,sample", CASES)
def test_pairing(gb, executor, whole_executor, kernel, w, h, planes, sample):
    import torch
    ow, oh = w * 2 // 3, h * 2 // 3
    hp, vp = (gb.AxisPlan(gb.AxisRequest(n, m, float(m), 0.0, kernel, 3, 0.0, 0.5, 1.0, "symmetric", 0))
              for n, m in ((w, ow), (h, oh)))
    gen = torch.Generator(device="cuda").manual_seed(w)
    x = torch.rand((planes, h, w), generator=gen, device="cuda")
    code, conversion = (0, None) if sample == "f32" else (2, gb.integer_conversion(16, False, False))
    if code:
        x = (x * 65535).to(torch.int32).to(torch.int16)
    outs = []
    for ex in (executor, whole_executor):
        out = torch.zeros((planes, oh, ow), dtype=x.dtype, device="cuda")
        batch = ex.prepare_batch([gb.PlaneTask(hp, vp, x[i].data_ptr(), w, out[i].data_ptr(), ow, code, 0, conversion)
                                  for i in range(planes)])
        torch.cuda.synchronize()
        batch.launch(0)
        batch.check(0)
        torch.cuda.synchronize()
        outs.append(out)
    if code:
        assert int(((outs[0].int() & 65535) - (outs[1].int() & 65535)).abs().max()) <= 1
    else:
        assert float((outs[0] - outs[1]).abs().max()) <= 4e-7 * max(1.0, float(outs[1].abs().max()))
