"""Launches that start while the ones ahead of them end wait for their results: frames behind
one another, their input rewritten by another kernel in between and their output read by one,
give the bytes of frames run one at a time - on streams, in a graph, and for one- and two-pass
routes, small and larger than the device."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# Width, height, planes, kernel, taps, and whether both axes are descaled.
CASES = [(48, 32, 1, "bicubic", 3, "both"), (640, 360, 3, "lanczos", 3, "both"), (700, 330, 2, "spline64", 3, "both"),
         (1920, 1080, 6, "bilinear", 3, "both"), (701, 333, 3, "lanczos", 3, "both"), (701, 333, 2, "bicubic", 3, "rows"),
         (701, 333, 2, "bicubic", 3, "columns"), (640, 360, 2, "bicubic", 3, "rows"), (640, 360, 2, "lanczos", 4, "columns")]


@pytest.mark.parametrize("w,h,planes,kernel,taps,axes", CASES)
def test_frames_behind_one_another(gb, whole_executor, w, h, planes, kernel, taps, axes):
    import torch
    ex = whole_executor
    ow, oh = (w * 2 // 3 if axes != "columns" else w), (h * 2 // 3 if axes != "rows" else h)
    plan = lambda n, m: gb.AxisPlan(gb.AxisRequest(n, m, float(m), 0.0, kernel, taps, 0.0, 0.5, 1.0, "symmetric", 0))
    hp = plan(w, ow) if axes != "columns" else None
    vp = plan(h, oh) if axes != "rows" else None
    frames = [torch.from_numpy(np.random.default_rng(i).random((planes, h, w), dtype=np.float32)).cuda()
              for i in range(6)]
    x = torch.zeros((planes, h, w), dtype=torch.float32, device="cuda")
    y = torch.zeros((planes, oh, ow), dtype=torch.float32, device="cuda")
    vectors = {"both": 0, "rows": h, "columns": w}[axes]
    batch = ex.prepare_batch([gb.PlaneTask(hp, vp, x[i].data_ptr(), w, y[i].data_ptr(), ow, 0, vectors)
                              for i in range(planes)])

    def one(stream, k, got):
        x.copy_(frames[k])
        batch.launch(stream)
        got[k].copy_(y)

    want = torch.zeros((len(frames),) + tuple(y.shape), dtype=torch.float32, device="cuda")
    stream = torch.cuda.Stream()
    for k in range(len(frames)):
        with torch.cuda.stream(stream):
            one(stream.cuda_stream, k, want)
        torch.cuda.synchronize()
    batch.check(stream.cuda_stream)
    assert not torch.equal(want[0], want[1])

    got = torch.zeros_like(want)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        for k in range(len(frames)):
            one(torch.cuda.current_stream().cuda_stream, k, got)

    def streamed(s):
        with torch.cuda.stream(s):
            for k in range(len(frames)):
                one(s.cuda_stream, k, got)

    for run in (lambda: streamed(stream), lambda: streamed(torch.cuda.default_stream()), graph.replay):
        for _ in range(3):
            got.zero_()
            torch.cuda.synchronize()
            run()
            torch.cuda.synchronize()
            batch.check(stream.cuda_stream)
            assert torch.equal(got, want)
