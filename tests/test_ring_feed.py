"""The refill of the chunk-delayed 2D kernels' ring (tring_impl.cuh), replayed on
the CPU: 48 columns a vector, refilled 16 samples at a time up to the end of a
group of four destinations' last window, the first 16 columns stored again
after the ring.  Every plan that the chunk-delayed kernels admit must find its
windows there, at any ratio that their feed allows."""
import numpy as np
import pytest

COLUMNS, DUP, STEP = 48, 16, 16


def compiled_window(hb, window):
    """ring_window (stream_plan.cpp): the compiled window that serves a plan."""
    if hb == 1 and window <= 4:
        return 4
    if hb <= 5 and window <= 8:
        return 8
    if hb >= 3 and window <= 12:
        return 12
    return 16 if window <= 16 else 0


def replay(starts, window, size):
    """Windows (as sample indices per destination) read from the replayed ring."""
    ring = np.full(COLUMNS + DUP, -1)
    have, read = 0, []
    for g in range(0, len(starts), 4):
        need = min(size, starts[g + 3] + window)
        while have < need:
            for s in range(have, have + STEP):
                column = s % COLUMNS
                ring[column] = s
                if column < DUP:
                    ring[column + COLUMNS] = s
            have += STEP
        read += [ring[s % COLUMNS:s % COLUMNS + window].copy() for s in starts[g:g + 4]]
    return np.array(read)


@pytest.mark.parametrize("seed", range(4))
def test_admitted_plans_fit_the_ring(gb, seed):
    rng = np.random.default_rng(seed)
    kernels = [("bilinear", 3), ("bicubic", 3), ("lanczos", 2), ("lanczos", 3), ("lanczos", 4), ("spline16", 3),
               ("spline36", 3)]
    admitted = 0
    for _ in range(150):
        size = int(np.exp(rng.uniform(np.log(4), np.log(2000))))
        out = max(1, int(size / np.exp(rng.uniform(0, np.log(9)))))
        kernel, taps = kernels[int(rng.integers(len(kernels)))]
        request = gb.AxisRequest(size, out, float(out), float(rng.choice([0.0, 0.25, -1.5])), kernel, taps, 0.0, 0.5,
                                 float(rng.choice([1.0, 1.1])),
                                 str(rng.choice(["symmetric", "repeat", "zero", "mirror"])), 1)
        try:
            plan = gb.AxisPlan(request, cached=False)
        except (ValueError, RuntimeError):
            continue
        info = plan.stream_info(records=True)
        if not (info["eligible"] and info["ring_ok_transposed"]):
            continue
        admitted += 1
        window = compiled_window(plan.half_bandwidth, info["window"])
        assert window >= info["window"]
        own = info["forward"][:, 0].copy().view(np.int32).astype(int)
        starts = np.minimum(own, max(0, size - window))
        read = replay(starts, window, size)
        # Every sample a destination weighs is in its place; columns never
        # filled (a source shorter than the window) meet zero weights.
        for j in range(plan.destination_size):
            for k in np.flatnonzero(info["forward"][j, 4:4 + info["window"]]):
                s = own[j] + k
                assert read[j, s - starts[j]] == s, (request, j, k)
    assert admitted > 30
