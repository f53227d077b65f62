"""Prepared batches of Float32 planes on both sides of the line between one part and two
(a share of the resident warp slots, by kernel): the part count, and samples within the
segments' 4e-7 of the largest magnitude of whole vectors'.  Integer planes keep two parts."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# Kernel, blur, the share of the warp slots, rows of a plane (32 a warp), sample.
CASES = [("bicubic", 1.0, 3, 2048, np.float32), ("bilinear", 1.0, 4, 2048, np.float32),
         ("spline64", 1.1, 6, 1024, np.float32), ("bicubic", 1.0, None, 256, np.uint16)]


@pytest.mark.parametrize("kernel,blur,share,rows,dtype", CASES)
def test_parts(gb, executor, whole_executor, kernel, blur, share, rows, dtype):
    import torch
    slots = torch.cuda.get_device_properties(0).multi_processor_count * 16
    most = slots // share // (rows // 32) if share else 8
    w, ow, oh = 95, 61, rows * 2 // 3 - 1
    code, conversion = (0, None) if dtype == np.float32 else (2, gb.integer_conversion(16, False, False))
    h, v = (gb.AxisPlan(gb.AxisRequest(n, m, float(m), 0.0, kernel, 3, 0.0, 0.5, blur, "symmetric", 0))
            for n, m in ((w, ow), (rows, oh)))
    rng = np.random.default_rng(rows)
    for planes in (8, most, most + 1):
        x = rng.random((planes, rows, w), dtype=np.float32)
        x = torch.from_numpy(x if code == 0 else (x * 65535).astype(dtype).view(np.int16)).cuda()
        got, want = (torch.zeros((planes, oh, ow), dtype=x.dtype, device="cuda") for _ in range(2))
        torch.cuda.synchronize()
        parts = []
        for ex, out in ((executor, got), (whole_executor, want)):
            batch = ex.prepare_batch([gb.PlaneTask(h, v, x[i].data_ptr(), w, out[i].data_ptr(), ow, code, 0, conversion)
                                      for i in range(planes)])
            parts.append(batch.info()["parts"])
            for _ in range(2):
                batch.launch(0)
            batch.check(0)
        assert parts == [1 if share and planes <= most else 2, 2]
        if code:
            assert int(((got.int() & 65535) - (want.int() & 65535)).abs().max()) <= 1
        else:
            assert float((got - want).abs().max()) <= 4e-7 * float(want.abs().max())
