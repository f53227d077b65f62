"""Prepared batches whose passes are many launches run them side by side on forked
streams: the same samples as the launches one after another, repeated, on the
caller's stream and replayed from a graph."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# Plans of different kernels: half-bandwidths 1, 3, 5, 7 and 9, a forced Float64.
PLANS = [("bilinear", 3, 1.0, 0), ("bicubic", 3, 1.0, 0), ("lanczos", 3, 1.0, 0), ("lanczos", 4, 1.0, 0),
         ("spline64", 3, 1.1, 0), ("bicubic", 3, 1.0, 2)]


def test_mixed_batch(gb, whole_executor):
    import torch
    ex = whole_executor
    tasks, outs, kept = [], [], []
    for i, (kernel, taps, blur, f64) in enumerate(PLANS):
        h, v = (gb.AxisPlan(gb.AxisRequest(n, m, float(m), 0.0, kernel, taps, 0.0, 0.5, blur, "symmetric", f64))
                for n, m in ((200 + 8 * i, 131), (120, 83)))
        x = torch.from_numpy(np.random.default_rng(i).random((120, 200 + 8 * i), dtype=np.float32)).cuda()
        out = torch.zeros((83, 131), dtype=torch.float32, device="cuda")
        tasks.append(gb.PlaneTask(h, v, x.data_ptr(), x.shape[1], out.data_ptr(), 131))
        outs.append(out)
        kept.append((x, h, v))
    torch.cuda.synchronize()
    want = []
    for task, out in zip(tasks, outs):
        ex.run_batch([task])
        want.append(out.clone())
    batch = ex.prepare_batch(tasks)
    assert batch.info()["parts"] == 1 and batch.info()["kernel_launches"] >= 2 * len(PLANS) - 2
    stream = torch.cuda.Stream()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        batch.launch(torch.cuda.current_stream().cuda_stream)
    for run in (lambda: batch.launch(stream.cuda_stream), graph.replay):
        for _ in range(3):
            for out in outs:
                out.zero_()
            torch.cuda.synchronize()
            run()
            torch.cuda.synchronize()
            batch.check(stream.cuda_stream)
            for out, w in zip(outs, want):
                assert torch.equal(out, w)
