"""Axes of millions of samples: the records of the kernels with the ring in tensor memory
hold every group's refill target, on either side of 2^23 samples."""
import numpy as np
import pytest


@pytest.mark.parametrize("size,out", [(8_388_600, 3_000_000), (8_400_000, 4_200_000)])
def test_refill_targets(gb, size, out):
    plan = gb.AxisPlan(gb.AxisRequest(size, out, float(out), 0.0, "bilinear", 3, 0.0, 0.5, 1.0, "symmetric", 0),
                       cached=False)
    ring = plan.stream_ring()
    window = ring["window"]
    assert window
    info = plan.stream_info(records=True)
    own = info["forward"][:, 0].copy().view(np.int32)
    heads = np.ascontiguousarray(ring["forward"][:, :4]).view(np.uint32)
    starts = np.minimum(own, size - window).reshape(-1, 4)
    assert np.array_equal(heads & 255, starts % ring["columns"])
    targets = (heads[:, 0] >> 8).astype(np.int64) * 16
    ends = starts[:, 3].astype(np.int64) + window
    assert np.array_equal(targets, (ends + 15) // 16 * 16)
    assert targets[-1] >= size - 2 * window
