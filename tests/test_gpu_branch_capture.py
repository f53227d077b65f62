"""A batch whose launches run side by side on streams of its own may be launched on one stream
while another still captures it, and from several threads: the samples of one launch alone."""
import ctypes as C
import threading

import numpy as np
import pytest

from test_gpu_launch_order import call

pytestmark = pytest.mark.gpu

KERNELS = [("bilinear", 3, 1.0), ("bicubic", 3, 1.0), ("lanczos", 3, 1.0), ("lanczos", 4, 1.0), ("spline64", 3, 1.1)]


@pytest.fixture(scope="module", params=[1, 2])
def mixed(request, gb, whole_executor):
    """A batch of planes of several kernels in one part or two, its outputs and their samples."""
    import torch
    tasks, outs, kept = [], [], []
    for i, (kernel, taps, blur) in enumerate(KERNELS):
        h, v = (gb.AxisPlan(gb.AxisRequest(n, m, float(m), 0.0, kernel, taps, 0.0, 0.5, blur, "symmetric", 0))
                for n, m in ((200, 131), (120, 83)))
        x = torch.from_numpy(np.random.default_rng(i).random((120, 200), dtype=np.float32)).cuda()
        outs.append(torch.zeros((83, 131), device="cuda"))
        tasks.append(gb.PlaneTask(h, v, x.data_ptr(), 200, outs[-1].data_ptr(), 131))
        kept.append((x, h, v))
    batch = whole_executor.prepare_batch(tasks, parts=request.param)
    torch.cuda.synchronize()
    batch.launch(0)
    batch.check(0)
    want = [out.clone() for out in outs]
    torch.cuda.synchronize()
    yield batch, outs, want, kept
    batch.close()


def same(outs, want):
    import torch
    torch.cuda.synchronize()
    result = all(torch.equal(o, w) for o, w in zip(outs, want))
    for out in outs:
        out.zero_()
    torch.cuda.synchronize()
    return result


def test_launch_while_captured(mixed):
    import torch
    batch, outs, want, _ = mixed
    same(outs, want)
    one, two = torch.cuda.Stream(), torch.cuda.Stream()
    graph, ready = C.c_void_p(), C.c_void_p()
    call("cuStreamBeginCapture_v2", C.c_void_p(one.cuda_stream), 2)
    try:
        batch.launch(one.cuda_stream)
        batch.launch(two.cuda_stream)
    finally:
        call("cuStreamEndCapture", C.c_void_p(one.cuda_stream), C.byref(graph))
    assert same(outs, want)
    call("cuGraphInstantiateWithFlags", C.byref(ready), graph, C.c_ulonglong(0))
    call("cuGraphLaunch", ready, C.c_void_p(two.cuda_stream))
    assert same(outs, want)
    batch.launch(two.cuda_stream)
    assert same(outs, want)
    call("cuGraphExecDestroy", ready)
    call("cuGraphDestroy", graph)


def test_launch_from_threads(mixed):
    import torch
    batch, outs, want, _ = mixed
    same(outs, want)
    stream = torch.cuda.Stream()
    for _ in range(20):
        threads = [threading.Thread(target=lambda: [batch.launch(stream.cuda_stream) for _ in range(4)]) for _ in range(4)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        assert same(outs, want)
