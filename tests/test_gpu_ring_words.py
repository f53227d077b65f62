"""Planes that no tensor map admits (not 16-byte aligned) but whose rows lie in whole
words come to the ring kernels word by word: the same samples, bit for bit, as their
aligned copies, whatever lies in the pitch's padding, at one and two vectors a lane,
for sizes on either side of blocks; rows that begin inside a word too."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DTYPES = {"f32": (np.float32, 0, None), "u16": (np.int16, 2, 16), "u8": (np.uint8, 1, 8)}
# Sample, kernel, blur, axes, width, height, words of padding a row, samples ahead of the first, planes.
CASES = [("f32", "lanczos", 1.0, "both", 131, 97, 2, 1, 1), ("f32", "bicubic", 1.0, "both", 641, 360, 1, 0, 130),
         ("f32", "spline64", 1.1, "both", 319, 213, 3, 3, 2), ("f32", "spline64", 1.1, "both", 319, 213, 0, 0, 90),
         ("f32", "bicubic", 1.0, "rows", 257, 131, 1, 1, 2), ("f32", "lanczos", 1.0, "rows", 255, 130, 2, 2, 300),
         ("f32", "bicubic", 1.0, "columns", 131, 257, 2, 1, 2), ("f32", "lanczos", 1.0, "columns", 131, 223, 1, 3, 300),
         ("f32", "bilinear", 1.0, "both", 29, 23, 1, 1, 3),
         ("u16", "lanczos", 1.0, "both", 130, 97, 1, 2, 2), ("u16", "bicubic", 1.0, "both", 641, 360, 1, 0, 100),
         ("u16", "bicubic", 1.0, "both", 129, 65, 0, 1, 2),
         ("u8", "spline36", 1.0, "both", 360, 240, 0, 4, 2), ("u8", "spline36", 1.0, "both", 359, 240, 2, 0, 150),
         ("u8", "bicubic", 1.0, "both", 127, 65, 0, 0, 2), ("u8", "spline64", 1.1, "both", 260, 131, 1, 0, 2)]


@pytest.mark.parametrize("sample,kernel,blur,axes,w,h,pad,ahead,planes", CASES)
def test_words(gb, whole_executor, sample, kernel, blur, axes, w, h, pad, ahead, planes):
    import torch
    dtype, code, bits = DTYPES[sample]
    size = np.dtype(dtype).itemsize
    ow, oh = (w * 3 // 4 if axes != "columns" else w), (h * 3 // 4 if axes != "rows" else h)
    plan = lambda n, m: gb.AxisPlan(gb.AxisRequest(n, m, float(m), 0.0, kernel, 3, 0.0, 0.5, blur, "symmetric", 0))
    hp = plan(w, ow) if axes != "columns" else None
    vp = plan(h, oh) if axes != "rows" else None
    conversion = gb.integer_conversion(bits, False, False) if code else None
    # Whole words a row (rows that begin inside a word where there is no padding).
    pitch = (-(-w * size // 4) * 4 + 4 * pad) // size if pad or w * size % 4 == 0 else w
    aligned = -(-w * size // 16) * 16 // size
    rng = np.random.default_rng(w)
    x = rng.random((planes, h, w), dtype=np.float32)
    x = x if code == 0 else (x * ((1 << bits) - 1)).astype(np.int64).astype(dtype)
    fill = np.nan if code == 0 else -1 if size == 2 else 255
    flat = np.full(ahead + planes * h * pitch, fill, dtype)
    flat[ahead:].reshape(planes, h, pitch)[:, :, :w] = x
    whole = np.zeros((planes, h, aligned), dtype)
    whole[:, :, :w] = x
    results = []
    for data, stride, first in ((flat, pitch, ahead), (whole.reshape(-1), aligned, 0)):
        data = torch.from_numpy(data).cuda()
        out = torch.zeros((planes, oh, ow), dtype=data.dtype, device="cuda")
        vectors = {"both": 0, "rows": h, "columns": w}[axes]
        batch = whole_executor.prepare_batch(
            [gb.PlaneTask(hp, vp, data.data_ptr() + (first + i * h * stride) * size, stride, out[i].data_ptr(), ow, code,
                          vectors, conversion) for i in range(planes)])
        torch.cuda.synchronize()
        for _ in range(2):
            batch.launch(0)
        batch.check(0)
        torch.cuda.synchronize()
        results.append(out)
    assert torch.isfinite(results[1].float()).all()
    assert torch.equal(*results)
