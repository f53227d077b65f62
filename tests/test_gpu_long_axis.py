"""One vector, or a few, of more than 2^23 samples: the one-axis ring kernels against the
reference CUDA order, within the streaming kernels' tolerance (4e-7 of the largest
magnitude, test_gpu_parity.py)."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("axis,vectors", [("rows", 1), ("columns", 4)])
def test_long_axis(gb, executor, axis, vectors):
    size, out = 8_400_000, 3_000_000
    request = (size, out, float(out), 0.0, "bilinear", 3, 0.0, 0.5, 1.0, "symmetric", 0)
    plan, checker = gb.AxisPlan(gb.AxisRequest(*request), cached=False), O.Plan(O.make_request(*request))
    assert plan.stream_ring()["window"]
    x = np.random.default_rng(vectors).random((vectors, size), dtype=np.float32)
    want = O.inverse_rows_gpu_order(checker, x)
    got = executor.inverse_rows(plan, x) if axis == "rows" else executor.inverse_columns(plan, np.ascontiguousarray(x.T)).T
    assert float(np.abs(got - want).max()) <= 4e-7 * float(np.abs(want).max())
