"""Sweep scoring at the edges of its two kernels (score.cu): odd frames, tiles of
256 and warps of 64 columns cut short, row blocks of 16 and segments cut short,
every compiled window, operators that only the general form reads, an odd frame
pitch; against the oracle's CPU descale re-upscaled in Float64, within the bar
of test_gpu_sweep.py (2e-5 absolute plus 1e-3 relative)."""
import numpy as np
import pytest

from test_gpu_sweep import _oracle_score, _scores

pytestmark = pytest.mark.gpu

# kernel, taps, blur, border, source / destination; windows 2, 4, 6 and 8, then
# wider operators, borders without entries and windows of fewer rows.
OPERATORS = [("bilinear", 3, 1.0, "symmetric", 1.4), ("bilinear", 3, 1.0, "symmetric", 3.7),
             ("bicubic", 3, 1.0, "mirror", 1.5), ("spline36", 3, 1.0, "repeat", 1.2),
             ("lanczos", 3, 1.0, "zero", 1.9), ("lanczos", 4, 1.0, "symmetric", 1.3),
             ("lanczos", 5, 1.0, "symmetric", 1.5), ("bicubic", 3, 1.1, "symmetric", 1.6),
             ("bilinear", 3, 1.0, "zero", 1.0)]


@pytest.mark.parametrize("width,height,pitch", [(131, 77, 131), (64, 33, 66), (259, 140, 260), (517, 16, 520)])
def test_edges(gb, executor, width, height, pitch):
    import torch
    rng = np.random.default_rng(width)
    frame = rng.random((height, width), dtype=np.float32)
    wide = torch.zeros((height, pitch), dtype=torch.float32, device="cuda")
    wide[:, :width] = torch.from_numpy(frame).cuda()
    requests, pairs = [], []
    for kernel, taps, blur, border, ratio in OPERATORS:
        pair = []
        for n in (width, height):
            out = max(8, int(round(n / ratio)))
            pair.append(gb.AxisRequest(n, out, float(out), 0.0, kernel, taps, 0.0, 0.5, blur, border, 0))
        requests.append(pair)
        pairs.append(tuple(gb.AxisPlan(r, cached=False) for r in pair))
    got, _ = _scores(gb, executor, wide, pairs)
    fixed, _ = _scores(gb, executor, wide, pairs, autotune=False, graph=False)
    for score, again, (h, v) in zip(got, fixed, requests):
        want = _oracle_score(frame, h, v)
        assert abs(score - want) <= 2e-5 + 1e-3 * want, (h, v, score, want)
        assert abs(again - score) <= 1e-6 * score + 1e-12
