"""Chunk-delayed 2D kernels with the ring in tensor memory (tring_impl.cuh): each
compiled half-bandwidth and window at the edges of their warps, chunks and
staged blocks, one and two vectors a lane, 16-byte aligned planes and not."""
import numpy as np
import pytest

import oracle as O
from common import F32_MAX_ABS, F32_MEAN_ABS, INT_MAX_CODES, make_input

pytestmark = pytest.mark.gpu

# kernel, taps, source / destination: half-bandwidths 1, 3, 5, 7 and every
# compiled window of them (4, 8, 12, 16).
PLANS = [("bilinear", 3, 1.3), ("bilinear", 3, 2.2), ("bilinear", 3, 4.5), ("bicubic", 3, 1.4), ("bicubic", 3, 2.3),
         ("lanczos", 3, 1.25), ("lanczos", 3, 1.6), ("lanczos", 3, 2.2), ("lanczos", 4, 1.3), ("lanczos", 4, 1.8)]
# Vectors of both passes around 32, 64 and 128; sources around the staged
# blocks (32, 64 and 128 samples); destinations around a chunk of 32.
SIZES = [(66, 33), (129, 64), (127, 65), (258, 31)]


def pair(gb, kernel, taps, ratio, width, height):
    def requests(n):
        out = max(9, int(round(n / ratio)))
        return n, out, float(out), 0.0, kernel, taps, 0.0, 0.5, 1.0, "symmetric", 0
    h, v = requests(width), requests(height)
    return (gb.AxisPlan(gb.AxisRequest(*h)), gb.AxisPlan(gb.AxisRequest(*v)),
            O.Plan(O.make_request(*h)), O.Plan(O.make_request(*v)))


@pytest.mark.parametrize("width,height", SIZES)
@pytest.mark.parametrize("kernel,taps,ratio", PLANS)
def test_edges(gb, executor, whole_executor, paired_executor, kernel, taps, ratio, width, height):
    h, v, oh, ov = pair(gb, kernel, taps, ratio, width, height)
    for sample in ("f32", "u16", "u8"):
        bits = {"f32": 16, "u16": 16, "u8": 8}[sample]
        conv = gb.integer_conversion(bits, False, False) if sample != "f32" else None
        x = make_input(height, width, sample, 3)
        want = O.inverse_2d(oh, ov, x, conv) if conv else O.inverse_2d(oh, ov, x)
        whole = whole_executor.inverse_2d(h, v, x, conv)
        assert np.array_equal(whole, paired_executor.inverse_2d(h, v, x, conv))
        for got in (whole, executor.inverse_2d(h, v, x, conv)):
            err = np.abs(got.astype(np.float64) - want)
            if sample == "f32":
                assert err.max() <= F32_MAX_ABS and err.mean() <= F32_MEAN_ABS, (sample, err.max())
            else:
                assert err.max() <= INT_MAX_CODES, (sample, err.max())


# Half-bandwidths 9 and 11 too, and a ratio beyond the ring's group refill.
@pytest.mark.parametrize("width,height", SIZES)
@pytest.mark.parametrize("kernel,taps,ratio", PLANS + [("spline64", 3, 1.5), ("lanczos", 5, 1.3), ("lanczos", 6, 1.2),
                                                       ("bilinear", 3, 7.3)])
def test_two_pass_edges(gb, exact_executor, kernel, taps, ratio, width, height):
    """Two-pass kernels (xring_impl.cuh) in whole vectors: the reference CUDA
    order bit for bit."""
    h, v, oh, ov = pair(gb, kernel, taps, ratio, width, height)
    for sample in ("f32", "u16", "u8"):
        bits = {"f32": 16, "u16": 16, "u8": 8}[sample]
        conv = gb.integer_conversion(bits, False, False) if sample != "f32" else None
        x = make_input(height, width, sample, 4)
        want = O.inverse_2d_gpu_order(oh, ov, x, conv) if conv else O.inverse_2d_gpu_order(oh, ov, x)
        assert np.array_equal(exact_executor.inverse_2d(h, v, x, conv), want), sample


@pytest.mark.parametrize("sample", ["f32", "u16", "u8"])
def test_unaligned_and_paired_batches(gb, whole_executor, sample):
    """Planes whose rows no tensor map admits (an odd pitch) and a batch large
    enough for two vectors a lane: each plane as alone, bit for bit."""
    import torch
    dtype = {"f32": np.float32, "u16": np.uint16, "u8": np.uint8}[sample]
    bits = {"f32": 16, "u16": 16, "u8": 8}[sample]
    code = gb.SAMPLES[np.dtype(dtype)]
    conv = gb.integer_conversion(bits, False, False)
    h, v, _, _ = pair(gb, "lanczos", 3, 1.25, 61, 5003)
    planes = [make_input(5003, 61, sample, s) for s in range(8)]
    for pitch in (61, 64):
        tasks, outs, kept = [], [], []
        for x in planes:
            wide = np.zeros((x.shape[0], pitch), dtype)
            wide[:, :61] = x
            dev = torch.from_numpy(wide.view(np.uint8)).cuda()
            out = torch.zeros((v.destination_size, h.destination_size * dev.shape[1] // pitch), dtype=torch.uint8,
                              device="cuda")
            tasks.append(gb.PlaneTask(h, v, dev.data_ptr(), pitch, out.data_ptr(), h.destination_size, code, 0, conv))
            outs.append(out)
            kept.append(dev)
        torch.cuda.synchronize()
        whole_executor.run_batch(tasks)
        for x, out in zip(planes, outs):
            got = out.cpu().numpy().view(dtype)
            assert np.array_equal(got, whole_executor.inverse_2d(h, v, x, conv if sample != "f32" else None))


@pytest.mark.parametrize("vectors,size", [(31, 66), (33, 515), (100, 1301), (129, 1024)])
@pytest.mark.parametrize("kernel,taps,ratio", PLANS)
def test_one_axis(gb, executor, whole_executor, kernel, taps, ratio, vectors, size):
    """One-axis passes: within the streaming kernels' tolerance (4e-7 of the
    largest magnitude, test_gpu_parity.py) of the reference CUDA order, and the
    same bits in segments as in whole vectors; rows whose pitch no tensor map
    admits alike."""
    h, _, oh, _ = pair(gb, kernel, taps, ratio, size, 64)
    x = make_input(vectors, size, "f32", 5)
    want = O.inverse_rows_gpu_order(oh, x)
    whole = whole_executor.inverse_rows(h, x)
    assert np.max(np.abs(whole - want)) <= 4e-7 * np.max(np.abs(want))
    assert np.array_equal(whole, executor.inverse_rows(h, x))
    wide = np.zeros((vectors, -(-size // 4) * 4 + 4), np.float32)
    wide[:, :size] = x
    out = np.zeros((vectors, -(-h.destination_size // 4) * 4 + 8), np.float32)
    assert np.array_equal(whole, executor.inverse_rows(h, wide[:, :size], out[:, :h.destination_size]))
    assert not out[:, h.destination_size:].any()
    columns = whole_executor.inverse_columns(h, np.ascontiguousarray(x.T))
    assert np.array_equal(columns, executor.inverse_columns(h, np.ascontiguousarray(x.T)))
    assert np.max(np.abs(columns.T - want)) <= 4e-7 * np.max(np.abs(want))
