"""The calls by which this executor is measured: the work of its public entry
points over the sizes, formats and kernels that a frame server, a batch job
or a native-resolution search gives it.

Kinds of call:

* ``host``     one frame through the synchronous per-plane host call, as a
               filter is asked for it (page-locked frames, copies included);
* ``planes``   a run of host frames through the pipelined multi-plane call;
* ``batch``    frames resident on the GPU through a prepared batch;
* ``rows``, ``columns``  a descale of one axis only, planes on the GPU;
* ``sweep``    one frame descaled to every candidate size, re-upscaled and
               scored.

Frames are a smoothed random field upscaled by the case's own operator plus
a little noise, quantised at limited range for integer formats.  Row pitches
are either tight or padded to 64 bytes, as frame pools allocate them.
"""
import functools
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PACKAGE = os.path.join(ROOT, "vapoursynth-descalemvc_gb300")
if PACKAGE not in sys.path:
    sys.path.insert(0, PACKAGE)

BASE = dict(kind="batch", width=1920, height=1080, out_width=1440, out_height=810, kernel="bicubic", taps=3,
            b=0.0, c=0.5, blur=1.0, border="symmetric", f64_mode=0, format="GRAYS", frames=1, pitch=64)
# The sweeps' kernels: the search tries each at every height.
SWEEP_KERNELS = (("bicubic", 3), ("bilinear", 3), ("lanczos", 3))


def _case(name, **fields):
    return dict(BASE, name=name, **fields)


def listed():
    return [
        # The smallest call of a filter: a reduced-size preview, one Float32 plane; latency is all of it.
        _case("host_360p", kind="host", width=640, height=360, out_width=480, out_height=270),
        # One frame of a 16-bit clip as a filter is asked for it, three planes of a call each.
        _case("host_1080p_yuv16", kind="host", kernel="lanczos", border="repeat", format="YUV420P16"),
        # A batch job over host frames: uploads, kernels and downloads overlapped.
        _case("planes_1080p_yuv16", kind="planes", kernel="lanczos", border="repeat", format="YUV420P16", frames=16),
        # A lone Float32 frame already on the GPU: too few rows to fill the chip.
        _case("frame_1080p", out_width=1280, out_height=720),
        # A clip's batch of 16-bit frames on the GPU, the usual bulk work.
        _case("clip_1080p_yuv16", kernel="lanczos", border="repeat", format="YUV420P16", frames=64),
        # 8-bit SD frames at a size that divides by nothing: odd vectors, short planes, unequal groups.
        _case("clip_480p_yuv8", kernel="spline36", width=720, height=480, out_width=598, out_height=398,
              format="YUV420P8", frames=24, pitch=0),
        # 4K Float32 frames with a blurred Mitchell kernel.
        _case("clip_4k", width=3840, height=2160, out_width=2560, out_height=1440, b=1 / 3, c=1 / 3, blur=1.1,
              frames=32),
        # The widest usual kernel at 4K: half-bandwidth 9, slowly decaying factors.
        _case("clip_4k_spline64", kernel="spline64", width=3840, height=2160, out_width=2560, out_height=1440,
              blur=1.1, frames=8),
        # The same solve in Float64, as the user forces it (the planner does for ill-conditioned sizes).
        _case("clip_4k_float64", kernel="spline64", width=3840, height=2160, out_width=2560, out_height=1440,
              blur=1.1, f64_mode=2, frames=4),
        # One axis only: anamorphic and field-based sources.
        _case("rows_1080p", kind="rows", kernel="lanczos", out_height=1080, frames=8),
        _case("columns_1080p", kind="columns", kernel="lanczos", out_width=1920, frames=8),
        # The native-resolution search: three kernels, every eighth height.
        _case("sweep_1080p", kind="sweep", out_width=0, out_height=0, first=500, last=1000, step=8, kernel="all"),
    ]


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    case = dict(BASE)
    kind = rng.choice(["host", "planes", "batch", "batch", "batch", "batch", "rows", "columns", "sweep"])
    width = _log_int(rng, 320, 3840 if kind in ("batch", "rows", "columns") else 1920)
    height = max(180, int(width * rng.uniform(0.42, 0.75)))
    name, taps, b, c = rng.choice([("bilinear", 3, 0.0, 0.5), ("bicubic", 3, 0.0, 0.5), ("bicubic", 3, 1 / 3, 1 / 3),
                                   ("lanczos", 2, 0.0, 0.5), ("lanczos", 3, 0.0, 0.5), ("lanczos", 4, 0.0, 0.5),
                                   ("spline16", 3, 0.0, 0.5), ("spline36", 3, 0.0, 0.5), ("spline64", 3, 0.0, 0.5)])
    fmt = rng.choice(["GRAYS", "GRAYS", "YUV420P16", "YUV420P8"])
    if kind in ("rows", "columns", "sweep"):
        fmt = "GRAYS"                                      # one axis and sweeps take Float32 planes
    if fmt != "GRAYS":
        width, height = width // 2 * 2, height // 2 * 2
    ratio = rng.uniform(0.5, 0.92)
    out_width, out_height = int(width * ratio), int(height * ratio)
    if fmt != "GRAYS":
        out_width, out_height = out_width // 2 * 2, out_height // 2 * 2
    f64 = 2 if kind in ("host", "batch") and rng.random() < 0.15 else 0
    pixels = {"host": 1, "planes": 16, "batch": 4 if f64 else 32, "rows": 8, "columns": 8, "sweep": 1}[kind]
    room = (1920 * 1080 if kind in ("planes", "sweep", "rows", "columns") else 3840 * 2160) * pixels
    most = max(1, min(64, room // (width * height)))
    frames = 1 if kind in ("host", "sweep") else _log_int(rng, 1, most)
    case.update(kind=kind, width=width, height=height, out_width=out_width, out_height=out_height, kernel=name,
                taps=taps, b=b, c=c, blur=rng.choice([1.0, 1.0, 1.0, 1.1]),
                border=rng.choice(["symmetric", "symmetric", "repeat", "zero"]), f64_mode=f64, format=fmt,
                frames=frames, pitch=rng.choice([64, 64, 0]))
    if kind == "rows":
        case["out_height"] = height
    elif kind == "columns":
        case["out_width"] = width
    elif kind == "sweep":
        first = int(height * rng.uniform(0.45, 0.55))
        last = int(height * rng.uniform(0.85, 0.93))
        case.update(out_width=0, out_height=0, kernel="all", blur=1.0, first=first, last=last,
                    step=max(1, (last - first) // rng.randint(8, 40)))
    return case


# ---- geometry ---------------------------------------------------------------

def _axes(case):
    """Per plane: (source w, source h, output w, output h, (active, shift) of the width, of the height)."""
    w, h, ow, oh = (case[k] for k in ("width", "height", "out_width", "out_height"))
    planes = [(w, h, ow, oh, (float(ow), 0.0), (float(oh), 0.0))]
    if case["format"] != "GRAYS":
        cw, ch = w // 2, h // 2
        planes += [(cw, ch, ow // 2, oh // 2, (ow * cw / w, 0.25 - 0.25 * ow / w), (oh * ch / h, 0.0))] * 2
    return planes


def _candidates(case):
    out = []
    for h in range(case["first"], case["last"], case["step"]):
        w = int(round(h * case["width"] / case["height"]))
        w += w & 1
        out += [(min(w, case["width"]), h, kernel, taps) for kernel, taps in SWEEP_KERNELS]
    return out


def _weight(kernel, taps, b, c, x):
    """Kernel values at distances x >= 0."""
    if kernel == "bilinear":
        return np.maximum(1 - x, 0)
    if kernel == "bicubic":
        near = ((12 - 9 * b - 6 * c) * x ** 3 + (-18 + 12 * b + 6 * c) * x ** 2 + (6 - 2 * b)) / 6
        far = ((-b - 6 * c) * x ** 3 + (6 * b + 30 * c) * x ** 2 + (-12 * b - 48 * c) * x + (8 * b + 24 * c)) / 6
        return np.where(x < 1, near, np.where(x < 2, far, 0.0))
    if kernel == "lanczos":
        return np.where(x < taps, np.sinc(x) * np.sinc(x / taps), 0.0)
    # Coefficients of (x - piece)^3, ^2, ^1, ^0 of each unit piece.
    pieces = {"spline16": [(1, -9 / 5, -1 / 5, 1), (-1 / 3, 4 / 5, -7 / 15, 0)],
              "spline36": [(13 / 11, -453 / 209, -3 / 209, 1), (-6 / 11, 270 / 209, -156 / 209, 0),
                           (1 / 11, -45 / 209, 26 / 209, 0)],
              "spline64": [(49 / 41, -6387 / 2911, -3 / 2911, 1), (-24 / 41, 4032 / 2911, -2328 / 2911, 0),
                           (6 / 41, -1008 / 2911, 582 / 2911, 0), (-1 / 41, 168 / 2911, -97 / 2911, 0)]}[kernel]
    out = np.zeros_like(x)
    for i, coefficients in enumerate(pieces):
        out = np.where((x >= i) & (x < i + 1), np.polyval(coefficients, x - i), out)
    return out


@functools.lru_cache(maxsize=32)
def _operator(src, dst, active, shift, kernel, taps, b, c, blur, border):
    """The upscaling operator of one axis (src x dst), Float64."""
    base = {"bilinear": 1, "bicubic": 2, "spline16": 2, "spline36": 3, "spline64": 4, "lanczos": taps}[kernel]
    support = math.ceil(base * blur)
    at = (np.arange(src) + 0.5) / (src / active) + shift
    begin = np.where(at - support < 0, np.floor(at - support + 0.5), np.floor(at - support + 0.49999999999999994)) + 0.5
    centre = begin[:, None] + np.arange(2 * support)[None, :]
    weight = _weight(kernel, taps, b, c, np.abs(centre - at[:, None]) / blur)
    weight = weight / weight.sum(1, keepdims=True)
    column = np.floor(centre).astype(np.int64)
    outside = (column < 0) | (column >= dst)
    if border == "repeat":
        column = np.clip(column, 0, dst - 1)
    elif border == "symmetric":
        column = column % (2 * dst)
        column = np.where(column < dst, column, 2 * dst - 1 - column)
    else:
        weight = np.where(outside, 0.0, weight)
        column = np.clip(column, 0, dst - 1)
    a = np.zeros((src, dst))
    np.add.at(a, (np.arange(src)[:, None].repeat(2 * support, 1), column), weight)
    return torch.from_numpy(a).cuda()


def _plane_operators(case, plane):
    sw, sh, ow, oh, (aw, shift_w), (ah, shift_h) = plane
    k = (case["kernel"], case["taps"], case["b"], case["c"], case["blur"], case["border"])
    return _operator(sw, ow, aw, shift_w, *k), _operator(sh, oh, ah, shift_h, *k)


# ---- inputs -----------------------------------------------------------------

def _field(rows, cols, gen):
    """A smoothed random field in [0, 1] (Gaussian, sigma 1.5)."""
    x = torch.rand((1, 1, rows, cols), generator=gen, device="cuda")
    t = torch.arange(-6, 7, device="cuda", dtype=torch.float32)
    g = torch.exp(-t * t / 4.5)
    g = g / g.sum()
    x = torch.nn.functional.pad(x, (6, 6, 6, 6), mode="reflect")
    x = torch.nn.functional.conv2d(x, g.view(1, 1, 1, -1))
    return torch.nn.functional.conv2d(x, g.view(1, 1, -1, 1))[0, 0]


SAMPLES = {"GRAYS": (torch.float32, 0, 32), "YUV420P16": (torch.int16, 2, 16), "YUV420P8": (torch.uint8, 1, 8)}


def _pitch(case, width, size):
    return -(-width * size // case["pitch"]) * case["pitch"] // size if case["pitch"] else width


def _planes(count, rows, cols, case, device="cuda"):
    """`count` planes of the case's pitch, 16-bit samples held as int16 bit patterns."""
    dtype = SAMPLES[case["format"]][0]
    size = torch.empty((), dtype=dtype).element_size()
    shape = (count, rows, _pitch(case, cols, size))
    if device == "cpu":
        return torch.zeros(shape, dtype=dtype, pin_memory=True)[:, :, :cols]
    return torch.zeros(shape, dtype=dtype, device=device)[:, :, :cols]


def _frames(case, seed):
    """Per plane of the format: the samples of every frame."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    dtype, _, bits = SAMPLES[case["format"]]
    out = []
    for index, plane in enumerate(_axes(case)):
        sw, sh, ow, oh = plane[:4]
        ah, av = (m.float() for m in _plane_operators(case, plane))
        data = _planes(case["frames"], sh, sw, case)
        for frame in data:
            x = _field(oh if case["kind"] != "rows" else sh, ow if case["kind"] != "columns" else sw, gen)
            if case["kind"] != "rows":
                x = av @ x
            if case["kind"] != "columns":
                x = x @ ah.T
            x = x + 1e-3 * torch.randn((sh, sw), generator=gen, device="cuda")
            if dtype != torch.float32:
                unit = 1 << (bits - 8)
                x = (x - 0.5) * 224 * unit + 128 * unit if index else x * 219 * unit + 16 * unit
                x = x.round().clamp(0, (1 << bits) - 1).to(torch.int32)
            frame.copy_(x)
        out.append(data)
    return out


# ---- the calls --------------------------------------------------------------

@functools.lru_cache(maxsize=1)
def _executor():
    import dsmvc_gb300 as gb
    return gb.Executor(torch.cuda.current_device())


def _plans(case, plane):
    import dsmvc_gb300 as gb
    sw, sh, ow, oh, (aw, shift_w), (ah, shift_h) = plane
    k = (case["kernel"], case["taps"], case["b"], case["c"], case["blur"], case["border"], case["f64_mode"])
    ex = _executor()
    plans = (gb.AxisPlan(gb.AxisRequest(sw, ow, aw, shift_w, *k)) if case["kind"] != "columns" else None,
             gb.AxisPlan(gb.AxisRequest(sh, oh, ah, shift_h, *k)) if case["kind"] != "rows" else None)
    for p in plans:
        if p is not None:
            ex.prepare(p)
    return plans


def _stream():
    return torch.cuda.current_stream().cuda_stream


def _sweep_frame(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    w, h = case["width"], case["height"]
    bw, bh = w * 28 // 45, h * 28 // 45                    # the hidden native size: 672 lines of 1080
    ah, av = (_operator(s, d, float(d), 0.0, "bicubic", 3, 0.0, 0.5, 1.0, case["border"]).float()
              for s, d in ((w, bw), (h, bh)))
    frame = av @ _field(bh, bw, gen) @ ah.T + 1e-3 * torch.randn((h, w), generator=gen, device="cuda")
    data = _planes(1, h, w, case)[0]
    data.copy_(frame)
    return data


def _sweep_state(case, seed):
    import dsmvc_gb300 as gb
    w, h = case["width"], case["height"]
    data = _sweep_frame(case, seed)
    requests = []
    for cw, ch, kernel, taps in _candidates(case):
        for s, d in ((w, cw), (h, ch)):
            requests.append(gb.AxisRequest(s, d, float(d), 0.0, kernel, taps, 0.0, 0.5, 1.0, case["border"], 0))
    plans = gb.build_plans(requests)
    ex = gb.Executor(torch.cuda.current_device())          # a search's plans go with it
    ex.prepare_many(plans)
    pairs = list(zip(plans[0::2], plans[1::2]))
    torch.cuda.synchronize()
    sweep = gb.Sweep(ex, pairs, data.data_ptr(), data.stride(0))
    return {"kind": "sweep", "sweep": sweep, "frame": data, "executor": ex}


def prepare(case, seed):
    import dsmvc_gb300 as gb
    if case["kind"] == "sweep":
        return _sweep_state(case, seed)
    ex = _executor()
    _, code, bits = SAMPLES[case["format"]]
    plans, conversions = {}, {}
    for index, plane in enumerate(_axes(case)):
        plans[plane[:2]] = _plans(case, plane)
        conversions[index > 0] = gb.integer_conversion(bits, index > 0, False) if code else None
    host = case["kind"] in ("host", "planes")
    outputs, kept, by_frame = [], _frames(case, seed), [[] for _ in range(case["frames"])]
    for index, (plane, data) in enumerate(zip(_axes(case), kept)):
        h, v = plans[plane[:2]]
        conversion = conversions[index > 0]
        rows, cols = plane[3] if v is not None else plane[1], plane[2] if h is not None else plane[0]
        out = _planes(case["frames"], rows, cols, case, "cpu" if host else "cuda")
        if host:
            pinned = _planes(*data.shape, case, "cpu")
            pinned.copy_(data)
            kept[index] = pinned
        for x, y, tasks in zip(kept[index], out, by_frame):
            if host:
                x, y = (t.numpy().view(np.uint16) if code == 2 else t.numpy() for t in (x, y))
                tasks.append((h, v, x, y, conversion))
            else:
                vectors = plane[1] if v is None else plane[0] if h is None else 0
                tasks.append(gb.PlaneTask(h, v, x.data_ptr(), x.stride(0), y.data_ptr(), y.stride(0), code, vectors,
                                          conversion))
        outputs.append(out)
    tasks = [t for frame in by_frame for t in frame]
    state = {"kind": case["kind"], "executor": ex, "outputs": outputs, "kept": kept, "tasks": tasks}
    torch.cuda.synchronize()
    if case["kind"] == "planes":
        state["planes"] = ex.host_planes(tasks)
    elif not host:
        state["batch"] = ex.prepare_batch(tasks)
    return state


def run(state):
    kind = state["kind"]
    if kind == "sweep":
        state["sweep"].run(_stream())
        return state["sweep"].scores(_stream())
    if kind == "host":
        for h, v, x, y, conversion in state["tasks"]:
            state["executor"].inverse_2d(h, v, x, conversion, y)
    elif kind == "planes":
        state["planes"].run()
    else:
        state["batch"].launch(_stream())
    return state["outputs"]


def work(case):
    size = torch.empty((), dtype=SAMPLES[case["format"]][0]).element_size()
    if case["kind"] == "sweep":
        w, h = case["width"], case["height"]
        flops = 0.0
        for cw, ch, kernel, taps in _candidates(case):
            support = {"bilinear": 1, "bicubic": 2}.get(kernel, taps)
            band = 2 * support - 1
            flops += h * w * 4 * support + h * cw * (4 * band + 2)             # rows of the frame
            flops += cw * h * 4 * support + cw * ch * (4 * band + 2)           # columns of the intermediate
            flops += ch * w * 4 * support + h * w * (4 * support + 2)          # upscaled again and compared
        return {"bytes": 4.0 * w * h + 4.0 * len(_candidates(case)), "flops": flops}
    moved, flops = 0, 0.0
    for sw, sh, ow, oh, _, _ in _axes(case):
        base = {"bilinear": 1, "bicubic": 2, "spline16": 2, "spline36": 3, "spline64": 4}
        support = math.ceil(base.get(case["kernel"], case["taps"]) * case["blur"])
        band = 2 * support - 1
        moved += (sw * sh + ow * oh) * size
        if case["kind"] != "columns":
            flops += sh * (4 * support * sw + ow * (4 * band + 2))
        if case["kind"] != "rows":
            flops += ow * (4 * support * sh + oh * (4 * band + 2))
    return {"bytes": float(moved * case["frames"]), "flops": float(flops * case["frames"])}


# ---- in 64 bits -------------------------------------------------------------

@functools.lru_cache(maxsize=8)
def _solver(*operator):
    """(A^T A)^-1 A^T of an operator."""
    a = _operator(*operator)
    return torch.cholesky_solve(a.T.contiguous(), torch.linalg.cholesky(a.T @ a))


def exact(case, seed):
    if case["kind"] == "sweep":
        frame = _sweep_frame(case, seed).double()
        scores = []
        for cw, ch, kernel, taps in _candidates(case):
            k = (kernel, taps, 0.0, 0.5, 1.0, case["border"])
            h = (case["width"], cw, float(cw), 0.0) + k
            v = (case["height"], ch, float(ch), 0.0) + k
            small = _solver(*v) @ frame @ _solver(*h).T
            scores.append((_operator(*v) @ small @ _operator(*h).T - frame).abs().mean())
        return torch.stack(scores).cpu().numpy()
    if case["format"] != "GRAYS":
        return None
    k = (case["kernel"], case["taps"], case["b"], case["c"], case["blur"], case["border"])
    (sw, sh, ow, oh, (aw, shift_w), (ah, shift_h)), = _axes(case)
    x, = _frames(case, seed)
    out = []
    for frame in x.double():
        if case["kind"] != "columns":
            frame = frame @ _solver(sw, ow, aw, shift_w, *k).T
        if case["kind"] != "rows":
            frame = _solver(sh, oh, ah, shift_h, *k) @ frame
        out.append(frame)
    out = torch.stack(out)
    return [out.cpu() if case["kind"] in ("host", "planes") else out]
