"""Vectors a lane of the launches with the ring in tensor memory: two in every one of them under
DSMVC_GB_PAIRED=1, read from a captured graph's grids, the samples those of one a lane; a sweep's
scores do not depend on what its tuning chose."""
import numpy as np
import pytest

import oracle as O
from conftest import _executor_with
from test_gpu_launch_order import call, captured
from test_gpu_ring import make_input, pair

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def two_a_lane(gb):
    ex = _executor_with(gb, "DSMVC_GB_PAIRED", "1", DSMVC_GB_SEGMENTS="1")
    yield ex
    ex.close()


def grids(batch, x):
    """Blocks of each launch of `batch`."""
    import torch
    stream = torch.cuda.Stream()

    def work():
        with torch.cuda.stream(stream):
            x.add_(0)
            batch.launch(stream.cuda_stream)

    x.add_(0)
    torch.cuda.synchronize()
    (_, *own), graph = captured(stream, work)
    out = [p.grid[0] for _, p in own]
    call("cuGraphDestroy", graph)
    return out


@pytest.mark.parametrize("kernel,taps,blur,axes", [("bicubic", 3, 1.0, "both"), ("spline64", 3, 1.1, "both"),
                                                   ("bicubic", 3, 1.0, "rows"), ("bicubic", 3, 1.0, "columns")])
def test_two_vectors_everywhere(gb, whole_executor, two_a_lane, kernel, taps, blur, axes):
    import torch
    w, h = 701, 513
    ow, oh = 467 if axes != "columns" else w, 342 if axes != "rows" else h
    plan = lambda n, m: gb.AxisPlan(gb.AxisRequest(n, m, float(m), 0.0, kernel, taps, 0.0, 0.5, blur, "symmetric", 0))
    hp, vp = plan(w, ow) if ow != w else None, plan(h, oh) if oh != h else None
    x = torch.from_numpy(np.random.default_rng(1).random((h, w), dtype=np.float32)).cuda()
    outs = []
    for ex, lanes in ((whole_executor, 1), (two_a_lane, 2)):
        y = torch.zeros((oh, ow), dtype=torch.float32, device="cuda")
        batch = ex.prepare_batch([gb.PlaneTask(hp, vp, x.data_ptr(), w, y.data_ptr(), ow, 0,
                                               {"both": 0, "rows": h, "columns": w}[axes])])
        vectors = {"both": [h, ow], "rows": [h], "columns": [w]}[axes]
        assert grids(batch, x) == [-(-n // (128 * lanes)) for n in vectors]
        batch.launch(0)
        batch.check(0)
        outs.append(y)
    assert torch.equal(*outs)


def test_scores_do_not_depend_on_the_tuning(gb, executor):
    import torch
    w, h = 500, 300
    frame = torch.from_numpy(np.random.default_rng(2).random((h, w), dtype=np.float32)).cuda()
    plan = lambda n, m, k: gb.AxisPlan(gb.AxisRequest(n, m, float(m), 0.0, k, 3, 0.0, 0.5, 1.0, "symmetric", 0))
    pairs = [(plan(w, m * w // h, k), plan(h, m, k)) for k in ("bicubic", "lanczos", "spline36") for m in (180, 211, 240)]
    torch.cuda.synchronize()
    scores = []
    for tuned in (False, True):
        sweep = gb.Sweep(executor, pairs, frame.data_ptr(), w, autotune=tuned)
        sweep.run(0)
        scores.append(sweep.scores(0))
        sweep.close()
    assert np.array_equal(*scores)


@pytest.fixture(scope="module")
def exact_two_a_lane(gb):
    ex = _executor_with(gb, "DSMVC_GB_EXACT", "1", DSMVC_GB_SEGMENTS="1", DSMVC_GB_PAIRED="1")
    yield ex
    ex.close()


# Half-bandwidths 3, 5, 9 and 11; vectors on either side of 64 a warp, 256 a CTA.
@pytest.mark.parametrize("width,height", [(90, 33), (97, 64), (131, 129), (388, 257)])
@pytest.mark.parametrize("kernel,taps,ratio", [("bicubic", 3, 1.5), ("lanczos", 3, 1.4), ("spline64", 3, 1.5),
                                               ("lanczos", 5, 1.3), ("lanczos", 6, 1.2)])
def test_two_pass_kernels(gb, exact_two_a_lane, kernel, taps, ratio, width, height):
    """Two-pass kernels at two vectors a lane: the reference CUDA order bit for bit."""
    h, v, oh, ov = pair(gb, kernel, taps, ratio, width, height)
    for sample in ("f32", "u16", "u8"):
        conv = gb.integer_conversion({"u16": 16, "u8": 8}[sample], False, False) if sample != "f32" else None
        x = make_input(height, width, sample, 6)
        want = O.inverse_2d_gpu_order(oh, ov, x, conv) if conv else O.inverse_2d_gpu_order(oh, ov, x)
        assert np.array_equal(exact_two_a_lane.inverse_2d(h, v, x, conv), want), sample


@pytest.mark.parametrize("pitch", [112, 97])
@pytest.mark.parametrize("sample", ["f32", "u16", "u8"])
def test_large_two_pass_batches(gb, whole_executor, sample, pitch):
    """Enough planes in one part for two vectors a lane in both passes, rows that a tensor map
    admits and rows that none does: the samples of batches at one."""
    import torch
    w, h, ow, oh = 97, 97, 65, 61
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    planes = -(-8 * sms // -(-ow // 32))
    dtype = {"f32": torch.float32, "u16": torch.int16, "u8": torch.uint8}[sample]
    code, size = {"f32": (0, 4), "u16": (2, 2), "u8": (1, 1)}[sample]
    conv = gb.integer_conversion(8 * size, False, False) if code else None
    hp, vp = (gb.AxisPlan(gb.AxisRequest(n, m, float(m), 0.0, "spline64", 3, 0.0, 0.5, 1.1, "symmetric", 0))
              for n, m in ((w, ow), (h, oh)))
    x = np.random.default_rng(size).random((planes, h, pitch), dtype=np.float32)
    x = torch.from_numpy(x if not code else (x * ((1 << 8 * size) - 1)).astype(np.int64)).to(dtype).cuda()
    outs = [torch.zeros((planes, oh, ow), dtype=dtype, device="cuda") for _ in range(2)]
    task = lambda i, out: gb.PlaneTask(hp, vp, x[i].data_ptr(), pitch, out[i].data_ptr(), ow, code, 0, conv)
    torch.cuda.synchronize()
    for out, group, lanes in ((outs[0], planes, 2), (outs[1], 40, 1)):
        for first in range(0, planes, group):
            part = range(first, min(first + group, planes))
            batch = whole_executor.prepare_batch([task(i, out) for i in part], parts=1)
            if first == 0:
                spare = torch.zeros(8, device="cuda")
                assert grids(batch, spare) == [-(-len(part) * -(-n // (32 * lanes)) // 4) for n in (h, ow)]
            batch.launch(0)
            batch.check(0)
    assert torch.equal(*outs)
