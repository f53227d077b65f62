"""Vectors a lane of the launches with the ring in tensor memory: two in every one of them under
DSMVC_GB_PAIRED=1, read from a captured graph's grids, the samples those of one a lane; a sweep's
scores do not depend on what its tuning chose."""
import numpy as np
import pytest

from conftest import _executor_with
from test_gpu_launch_order import call, captured

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
