"""How a prepared batch's launches order themselves behind what is ahead of them, read from
a captured graph: the first one, behind the caller's own kernel, allocates its tensor memory
late; those behind it, whose grid ahead is the batch's own, need not."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


class EdgeData(C.Structure):
    _fields_ = [("from_port", C.c_ubyte), ("to_port", C.c_ubyte), ("type", C.c_ubyte), ("reserved", C.c_ubyte * 5)]


class KernelParams(C.Structure):
    _fields_ = [("func", C.c_void_p), ("grid", C.c_uint * 3), ("block", C.c_uint * 3), ("shared", C.c_uint),
                ("params", C.POINTER(C.c_void_p)), ("extra", C.c_void_p), ("kern", C.c_void_p), ("ctx", C.c_void_p)]


def call(name, *args):
    rc = getattr(C.CDLL("libcuda.so.1"), name)(*args)
    assert rc == 0, (name, rc)


def captured(stream, work):
    """[(programmatic edge into it, its arguments)] of each kernel captured, in order."""
    graph = C.c_void_p()
    call("cuStreamBeginCapture_v2", C.c_void_p(stream.cuda_stream), 2)
    try:
        work()
    finally:
        call("cuStreamEndCapture", C.c_void_p(stream.cuda_stream), C.byref(graph))
    count = C.c_size_t()
    call("cuGraphGetEdges_v2", graph, None, None, None, C.byref(count))
    tail, head, data = (C.c_void_p * count.value)(), (C.c_void_p * count.value)(), (EdgeData * count.value)()
    call("cuGraphGetEdges_v2", graph, tail, head, data, C.byref(count))
    after = {tail[i]: (head[i], data[i].type == 1) for i in range(count.value)}
    node = next(iter(set(after) - {h for h, _ in after.values()}))
    out, edge = [], False
    while node is not None:
        p = KernelParams()
        call("cuGraphKernelNodeGetParams_v2", C.c_void_p(node), C.byref(p))
        out.append((edge, p))
        node, edge = after.get(node, (None, False))
    return out, graph


@pytest.mark.parametrize("kernel,taps,blur,axes", [("bicubic", 3, 1.0, "both"), ("spline64", 3, 1.1, "both"),
                                                   ("lanczos", 3, 1.0, "rows")])
def test_first_launch_allocates_late(gb, executor, kernel, taps, blur, axes):
    import torch
    w, h, ow, oh = 320, 200, 240, 150 if axes == "both" else 200
    plan = lambda n, m: gb.AxisPlan(gb.AxisRequest(n, m, float(m), 0.0, kernel, taps, 0.0, 0.5, blur, "symmetric", 0))
    hp, vp = plan(w, ow), plan(h, oh) if axes == "both" else None
    x = torch.from_numpy(np.random.default_rng(0).random((h, w), dtype=np.float32)).cuda()
    y = torch.zeros((oh, ow), dtype=torch.float32, device="cuda")
    batch = executor.prepare_batch([gb.PlaneTask(hp, vp, x.data_ptr(), w, y.data_ptr(), ow, 0, 0 if vp else h)])
    stream = torch.cuda.Stream()
    x.add_(0.0)
    torch.cuda.synchronize()

    def work():
        with torch.cuda.stream(stream):
            x.add_(0.0)
            batch.launch(stream.cuda_stream)

    (foreign, *own), graph = captured(stream, work)
    assert len(own) == batch.info()["kernel_launches"]
    late = [edge and bool(C.cast(p.params[2], C.POINTER(C.c_ubyte))[0]) for edge, p in own]
    early = [edge for edge, _ in own]
    assert late[0] or not early[0]
    assert early[1:] == [True] * (len(own) - 1) and not any(late[1:])
    call("cuGraphDestroy", graph)


@pytest.mark.parametrize("axes", ["both", "rows"])
def test_input_of_another_stream(gb, whole_executor, axes):
    """Input written on another stream, its event waited for behind the pass before: a first
    launch that starts early still waits for it."""
    import torch
    w, h, ow, oh = 640, 360, 427, 240 if axes == "both" else 360
    plan = lambda n, m: gb.AxisPlan(gb.AxisRequest(n, m, float(m), 0.0, "bicubic", 3, 0.0, 0.5, 1.0, "symmetric", 0))
    hp, vp = plan(w, ow), plan(h, oh) if axes == "both" else None
    frames = torch.from_numpy(np.random.default_rng(3).random((8, h, w), dtype=np.float32)).cuda()
    x, y = torch.zeros((h, w), device="cuda"), torch.zeros((oh, ow), device="cuda")
    batch = whole_executor.prepare_batch([gb.PlaneTask(hp, vp, x.data_ptr(), w, y.data_ptr(), ow, 0, 0 if vp else h)])
    want, got = (torch.zeros((8, oh, ow), device="cuda") for _ in range(2))
    load = torch.rand(1 << 24, device="cuda")
    for k in range(8):
        x.copy_(frames[k])
        torch.cuda.synchronize()
        batch.launch(0)
        batch.check(0)
        want[k].copy_(y)
    torch.cuda.synchronize()
    one, two = torch.cuda.Stream(), torch.cuda.Stream()
    for _ in range(4):
        got.zero_()
        torch.cuda.synchronize()
        for k in range(8):
            with torch.cuda.stream(two):
                two.wait_stream(one)
                load.add_(0.0)
                x.copy_(frames[k])
            with torch.cuda.stream(one):
                batch.launch(one.cuda_stream)            # the frame before, or this one: overwritten below
                one.wait_stream(two)
                batch.launch(one.cuda_stream)
                got[k].copy_(y)
        torch.cuda.synchronize()
        assert torch.equal(got, want)
