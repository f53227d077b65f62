"""The packed records of the kernels with the ring in tensor memory, as the kernels read them:
replayed from the first chunk and from every chunk at which a range may start, each
destination's weights meet their samples, and its factors are the plan's.  Chunk-delayed plans
and plans of the two-pass kernels alone (half-bandwidths 9 and 11, slow decay)."""
import numpy as np
import pytest

DUP, STEP, CHUNK = 16, 16, 32
KERNELS = [("bilinear", 3), ("bicubic", 3), ("lanczos", 2), ("lanczos", 3), ("lanczos", 4), ("lanczos", 5), ("lanczos", 6),
           ("spline16", 3), ("spline36", 3), ("spline64", 3)]


def windows(heads, first, columns, window):
    """Samples (or -1) in each destination's window, its ring refilled from sample `first` on to
    the groups' targets."""
    ring, have, out = np.full(columns + DUP, -1), first, []
    for head in heads:
        while have < (int(head[0]) >> 8) * STEP:
            at = np.arange(have, have + STEP)
            ring[at % columns] = at
            again = at[at % columns < DUP]
            ring[again % columns + columns] = again
            have += STEP
        out += [ring[int(h & 255):int(h & 255) + window].copy() for h in head]
    return np.array(out)


@pytest.mark.parametrize("seed", range(4))
def test_records(gb, seed):
    rng = np.random.default_rng(100 + seed)
    admitted, exact_only = 0, 0
    for _ in range(110):
        size = int(np.exp(rng.uniform(np.log(4), np.log(1200))))
        out = max(1, int(size / np.exp(rng.uniform(0, np.log(7)))))
        kernel, taps = KERNELS[int(rng.integers(len(KERNELS)))]
        request = gb.AxisRequest(size, out, float(out), float(rng.choice([0.0, 0.25, -1.5])), kernel, taps, 0.0, 0.5,
                                 float(rng.choice([1.0, 1.1])),
                                 str(rng.choice(["symmetric", "repeat", "zero", "mirror"])), 1)
        try:
            plan = gb.AxisPlan(request, cached=False)
        except (ValueError, RuntimeError):
            continue
        ring = plan.stream_ring()
        window, hb, n = ring["window"], plan.half_bandwidth, plan.destination_size
        if not window:
            continue
        info = plan.stream_info(records=True)
        admitted += 1
        exact_only += not info["eligible"]
        forward, backward = ring["forward"], ring["backward"]
        heads = np.ascontiguousarray(forward[:, :4]).view(np.uint32).astype(np.int64)
        weights = forward[:, 8:8 + 4 * window].reshape(-1, window)
        own = info["forward"]
        starts = own[:, 0].copy().view(np.int32)
        assert np.array_equal(forward[:, 4:8].reshape(-1), own[:, 1])
        lower = forward[:, 8 + 4 * window:8 + 4 * window + 4 * hb].reshape(-1, hb)
        assert np.array_equal(lower, own[:, 4 + info["window"]:4 + info["window"] + hb])
        assert np.array_equal(backward[:, :4 * hb].reshape(-1, hb), info["backward"][:, :hb])
        for chunk, first in [(0, 0)] + list(enumerate(ring["first_blocks"])):
            if chunk > 2 and chunk % 5:
                continue                     # the first ones, then every fifth
            seen = windows(heads[chunk * CHUNK // 4:], int(first), ring["columns"], window)
            for j in range(chunk * CHUNK, n):
                read, w = seen[j - chunk * CHUNK], weights[j]
                want = {int(starts[j]) + k: x for k, x in enumerate(own[j, 4:4 + info["window"]]) if x}
                assert {int(read[k]): w[k] for k in np.flatnonzero(w)} == want, (request, chunk, j)
    assert admitted > 25 and exact_only > 5, (admitted, exact_only)
