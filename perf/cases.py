"""The workloads this framework's speed is judged on, through its public entry points.

Three families cover what a user runs: engine streams (NLMeans, NLMeans-HQ and NL4D through
`build_engine` or `HostDenoiser`, a whole short clip per pass: reset, push every frame, emit what is
ready, drain the tail), the batched launch over clips of mixed size, and the differentiable passes
(`NlmWindow`, `Nl4dPass`, forward and backward). Sizes and options come from the presets, the
benchmark's workloads and the tests.
"""

from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

import av_denoise_b200_loader

avd = av_denoise_b200_loader.load()
from av_denoise_b200 import _abi  # noqa: E402
from av_denoise_b200.autograd import Nl4dPass, Nl4dPassConfig, NlmWindow  # noqa: E402

LAYOUTS = {"gray": avd.ChromaLayout.GRAY, "420": avd.ChromaLayout.YUV420, "422": avd.ChromaLayout.YUV422,
           "444": avd.ChromaLayout.YUV444}


# ---- the cases ----------------------------------------------------------------------------------


def _stream(name, algo, w, h, frames, depth, layout, planes, **options):
    case = dict(kind="stream", algo=algo, w=w, h=h, frames=frames, depth=depth, layout=layout, planes=planes, d=0,
                a=2, s=4, strength=0.0, hq=False, sigma=0.0, motion=False, escalate=False, prefilter="none", host=False,
                noise=8.0, pan=2)
    case.update(options)
    if name:
        case["name"] = name
    return case


def listed():
    return [
        # The smallest call: the veryfast preset on four thumbnail frames; launches and host time count.
        _stream("nlm_veryfast_320x180", "nlm", 320, 180, 4, 8, "gray", "luma", strength=1.2),
        # The repository's spatial workload: eight 640x360 luma frames, search radius 7, patch radius 3.
        _stream("nlm_spatial_640x360", "nlm", 640, 360, 8, 8, "gray", "luma", a=7, s=3, strength=12.0, noise=10.0),
        # The headline workload: 1080p 8-bit 4:2:0, luma over five frames and chroma spatially, two engines.
        _stream("nlm_temporal_1080p", "nlm_pair", 1920, 1080, 8, 8, "420", "both", d=2, a=5, s=2, strength=8.0, pan=4),
        # A user's host program: the base preset (HQ, automatic sigma) on 10-bit 1080p wire frames.
        _stream("hq_base_host_1080p", "nlm", 1920, 1080, 14, 10, "420", "both", d=2, hq=True, host=True),
        # The slow preset with motion compensation and search escalation, on an odd 10-bit size.
        _stream("hq_slow_motion_1279x719", "nlm", 1279, 719, 12, 10, "420", "both", d=4, a=4, hq=True, motion=True,
                escalate=True, pan=4),
        # Float planes with full chroma on an odd size, one step of a float pipeline.
        _stream("nlm_float_444_957x539", "nlm", 957, 539, 5, 32, "444", "both", d=1, a=3, s=4, strength=6.0),
        # Twenty-odd frames of clips of mixed size and window in one launch (HQ, pinned sigma).
        dict(name="batch_mixed_clips", kind="batch", clips="640x360x5r2 1280x720x6r4 1920x1080x4r1 853x479x7r3", a=4,
             s=2, noise=10.0),
        # Strength selection by gradient: one windowed frame forward and backward.
        dict(name="nlm_window_gradient_720p", kind="nlm_grad", w=1280, h=720, c=1, d=2, a=5, s=2, strength=8.0,
             noise=4.0),
        # NL4D on a small odd frame with a pinned sigma and direct motion.
        _stream("nl4d_479x271", "nl4d", 479, 271, 6, 8, "gray", "luma", d=1, sigma=10.0 / 255.0, noise=10.0),
        # NL4D with its default options (automatic sigma, pooled threshold) on 1080p 8-bit luma.
        _stream("nl4d_default_1080p", "nl4d", 1920, 1080, 12, 8, "420", "luma", d=2, noise=10.0),
        # The 4K NL4D workload: 10-bit 4:2:0, seven-frame window, search radius 16, automatic sigma.
        _stream("nl4d_4k_10bit", "nl4d", 3840, 2160, 12, 10, "420", "both", d=3, spatial_radius=16, lambda_ht=2.7,
                pooled=False, noise=5.0, pan=4),
        # The NL4D pass as a layer: forward and backward on a luma window.
        dict(name="nl4d_pass_gradient_720p", kind="nl4d_grad", w=1280, h=720, c=1, d=2, spatial_radius=9, wiener=False,
             pooled=False, noise=10.0),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _size(rng, lo, hi):
    w = _log(rng, lo, hi)
    h = max(16, int(w * rng.choice([0.5625, 0.5625, 0.75, 0.42]))) + rng.randint(0, 3)
    return w, h


def draw(rng):
    kind = rng.choice(["nlm", "nlm", "hq", "hq", "motion", "float", "batch", "nlm_grad", "nl4d", "nl4d", "nl4d_grad"])
    layout = rng.choice(["gray", "420", "420", "422", "444"])
    depth = rng.choice([8, 8, 10, 12])
    planes = "luma" if layout == "gray" else rng.choice(["luma", "chroma", "both"])
    noise = rng.uniform(4.0, 16.0)
    if kind == "nlm":
        w, h = _size(rng, 176, 1920)
        return _stream(None, "nlm", w, h, rng.randint(3, 8), depth, layout, planes, d=rng.randint(0, 3),
                       a=rng.randint(1, 7), s=rng.randint(0, 5), strength=rng.uniform(1.0, 12.0), noise=noise)
    if kind == "hq":
        w, h = _size(rng, 176, 1920)
        d = rng.randint(0, 4)
        return _stream(None, "nlm", w, h, rng.randint(3, 14), depth, layout, planes, d=d, a=rng.choice([2, 2, 4]),
                       s=rng.choice([2, 4, 4]), hq=True, sigma=rng.choice([0.0, noise / 255.0]),
                       prefilter=rng.choice(["none", "none", "bilateral", "nlm"]), host=rng.random() < 0.3, noise=noise)
    if kind == "motion":
        w, h = _size(rng, 176, 1280)
        return _stream(None, "nlm", w, h, rng.randint(4, 10), depth, layout, planes, d=rng.randint(1, 4),
                       a=rng.choice([2, 4]), s=rng.choice([2, 4]), strength=4.0, motion=True,
                       escalate=rng.random() < 0.5, noise=noise, pan=4)
    if kind == "float":
        w, h = _size(rng, 176, 960)
        return _stream(None, "nlm", w, h, rng.randint(2, 5), 32, layout, planes, d=rng.randint(0, 2),
                       a=rng.randint(1, 5), s=rng.randint(1, 5), strength=rng.uniform(3.0, 10.0), noise=noise)
    if kind == "batch":
        clips = []
        for _ in range(rng.randint(2, 4)):
            w, h = _size(rng, 176, 1920)
            clips.append(f"{w}x{h}x{rng.randint(2, 6)}r{rng.randint(0, 4)}")
        return dict(kind="batch", clips=" ".join(clips), a=rng.randint(2, 5), s=rng.randint(1, 3), noise=noise)
    if kind == "nlm_grad":
        w, h = _size(rng, 128, 1280)
        return dict(kind="nlm_grad", w=w, h=h, c=rng.choice([1, 1, 2]), d=rng.randint(0, 2), a=rng.randint(2, 5),
                    s=rng.randint(1, 3), strength=rng.uniform(5.0, 10.0), noise=noise)
    if kind == "nl4d":
        w, h = _size(rng, 176, 1920)
        return _stream(None, "nl4d", w, h, rng.randint(4, 12), depth, layout, planes, d=rng.randint(1, 3),
                       spatial_radius=rng.randint(5, 16), pooled=rng.random() < 0.7,
                       sigma=rng.choice([0.0, noise / 255.0]), noise=noise)
    w, h = _size(rng, 128, 1280)
    return dict(kind="nl4d_grad", w=w, h=h, c=rng.choice([1, 1, 2]), d=rng.randint(1, 2),
                spatial_radius=rng.randint(5, 12), wiener=rng.random() < 0.3, pooled=rng.random() < 0.5, noise=noise)


# ---- inputs -------------------------------------------------------------------------------------


def _base(gen, h, w):
    """Gratings over flat rectangles and blurred texture, in 8-bit codes, as the synthetic clips have."""
    dev = "cuda"

    def uni(lo, hi, n=1):
        return (torch.rand(n, generator=gen, device=dev, dtype=torch.float32) * (hi - lo) + lo).cpu().tolist()

    img = torch.full((h, w), 128.0, device=dev)
    u = [uni(0, 1, 40) for _ in range(5)]
    for i in range(40):
        rw, rh = max(2, int(w * (0.03 + 0.22 * u[0][i]))), max(2, int(h * (0.03 + 0.22 * u[1][i])))
        x0, y0 = int((w - rw) * u[2][i]), int((h - rh) * u[3][i])
        img[y0:y0 + rh, x0:x0 + rw] = 16.0 + 219.0 * u[4][i]
    y = torch.arange(h, device=dev, dtype=torch.float32)[:, None]
    x = torch.arange(w, device=dev, dtype=torch.float32)[None, :]
    f, th, amp, ph = uni(0.01, 0.3, 6), uni(0.0, math.pi, 6), uni(5.0, 30.0, 6), uni(0.0, 2 * math.pi, 6)
    for i in range(6):
        img += amp[i] * torch.sin(2 * math.pi * f[i] * (x * math.cos(th[i]) + y * math.sin(th[i])) + ph[i])
    tex = torch.rand((1, 1, h, w), generator=gen, device=dev) * 2 - 1
    k = torch.exp(-0.5 * (torch.arange(-6, 7, device=dev, dtype=torch.float32) / 1.5) ** 2)
    k = k / k.sum()
    tex = torch.nn.functional.conv2d(tex, k.view(1, 1, 13, 1), padding=(6, 0))
    tex = torch.nn.functional.conv2d(tex, k.view(1, 1, 1, 13), padding=(0, 6))[0, 0]
    img += tex * (12.0 / tex.abs().max())
    return img.clamp(16, 235)


def _series(gen, rng, w, h, frames, noise, pan, sx=1, sy=1):
    """`frames` noisy frames of one plane in 8-bit code units (f32), a panned base and a moving sprite."""
    off = [(0, 0)]
    for _ in range(frames - 1):
        off.append((off[-1][0] + int(rng.integers(-pan, pan + 1)), off[-1][1] + int(rng.integers(-pan, pan + 1))))
    m = pan * frames + 2
    base = _base(gen, h + 2 * m, w + 2 * m)
    size = max(4, min(w, h) // 6)
    sprite = _base(gen, size, size)
    px, py, vx, vy = int(w * 0.3), int(h * 0.3), int(rng.integers(-4, 5)), int(rng.integers(-4, 5))
    out = []
    for k in range(frames):
        ox, oy = off[k][0] // sx, off[k][1] // sy
        fr = base[m + oy:m + oy + h, m + ox:m + ox + w].clone()
        x0, y0 = min(max(px + k * vx, 0), w - size), min(max(py + k * vy, 0), h - size)
        fr[y0:y0 + size, x0:x0 + size] = sprite
        out.append(fr + noise * torch.randn((h, w), generator=gen, device="cuda"))
    return out


def _generators(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed)), np.random.default_rng(int(seed))


def _format(depth):
    return {8: avd.SampleFormat.u8(), 32: avd.SampleFormat.f32()}.get(depth) or avd.SampleFormat.u16(depth)


def _clip(case, geometry, seed):
    """Every frame's planes as device words of the case's sample format."""
    gen, rng = _generators(seed)
    depth = case["depth"]
    series = []
    for i in range(geometry.plane_count()):
        w, h = geometry.plane_dims(i)
        sx, sy = max(1, round(case["w"] / w)), max(1, round(case["h"] / h))
        noise = case["noise"] if i == 0 else 0.6 * case["noise"]
        planes = []
        for fr in _series(gen, rng, w, h, case["frames"], noise, case["pan"], sx, sy):
            if depth == 32:
                planes.append((fr.clamp(0, 255) / 255.0 - (0.5 if i else 0.0)).contiguous().reshape(-1))
                continue
            codes = (fr * float(1 << (depth - 8))).round().clamp(0, (1 << depth) - 1).reshape(-1)
            pad = (-codes.numel()) % (4 if depth == 8 else 2)
            codes = torch.nn.functional.pad(codes, (0, pad)).to(torch.uint8 if depth == 8 else torch.int16)
            planes.append(codes.view(torch.int32))
        series.append(planes)
    return [list(t) for t in zip(*series)]


# ---- engine streams -----------------------------------------------------------------------------


def _motion(case):
    if not case["motion"]:
        return avd.MotionCompensationMode()
    return avd.MotionCompensationMode(avd.MotionSearch(max_search_escalation=8 if case["escalate"] else 4))


def _nlm(case, temporal=True, strength=None):
    d = case["d"] if temporal else 0
    strength = strength or case["strength"]
    tuning = avd.NlmTuning(search_radius=case["a"], patch_radius=case["s"], strength=strength or None)
    pre = {"none": avd.PrefilterMode.none(), "bilateral": avd.PrefilterMode.bilateral(1.5, 0.08),
           "nlm": avd.PrefilterMode.nlm_spatial()}[case["prefilter"]]
    options = avd.NlmeansOptions(prefilter=pre, motion_compensation=_motion(case), tuning=tuning,
                                 mode=avd.DenoisingMode.temporal(d) if d else avd.DenoisingMode.spacial())
    if not case["hq"]:
        return avd.NlmeansAlgorithm.fast(options)
    return avd.NlmeansAlgorithm.hq_(avd.NlmeansHqOptions(options, avd.HqParams(sigma_override=case["sigma"] or None)))


def _nl4d(case):
    return avd.Nl4dOptions(temporal_radius=case["d"], sigma=case["sigma"] or None,
                           spatial_radius=case.get("spatial_radius", 9), lambda_ht=case.get("lambda_ht"),
                           pooled_threshold=case.get("pooled", True))


def _specs(case, geometry):
    luma, chroma = case["planes"] in ("luma", "both"), case["planes"] in ("chroma", "both")
    if case["algo"] == "nlm_pair":
        # One engine's window spans must agree, so the temporal luma and the spatial chroma run as two.
        return [avd.EngineSpec.nlmeans(_nlm(case), None, geometry),
                avd.EngineSpec.nlmeans(None, _nlm(case, temporal=False, strength=5.0), geometry)]
    make, spec = (_nl4d, avd.EngineSpec.nl4d) if case["algo"] == "nl4d" else (_nlm, avd.EngineSpec.nlmeans)
    return [spec(make(case) if luma else None, make(case) if chroma else None, geometry)]


def _geometry(case):
    fmt = _format(case["depth"])
    return avd.Geometry(case["w"], case["h"], LAYOUTS[case["layout"]], fmt, fmt)


def _prepare_stream(case, seed):
    geometry = _geometry(case)
    clip = _clip(case, geometry, seed)
    dims = [geometry.plane_dims(i) for i in range(geometry.plane_count())]
    state = dict(case=case, clip=clip, dims=dims, engines=[])
    if case["host"]:
        state["host"] = avd.HostDenoiser(_specs(case, geometry)[0])
        state["wire"] = [[p.cpu().numpy().tobytes()[:n] for p, n in zip(f, state["host"].plane_lengths)] for f in clip]
        state["out"] = [[bytearray(n) for n in state["host"].plane_lengths] for _ in clip]
        return state
    stream = torch.cuda.current_stream()
    state["planes"] = [[avd.DevicePlane.from_tensor(p, w, h) for p, (w, h) in zip(f, dims)] for f in clip]
    for spec in _specs(case, geometry):
        engine = avd.build_engine(spec)
        engine.set_stream(stream.cuda_stream)
        out = [[torch.zeros_like(p) for p in f] for f in clip]
        planes = [[avd.DevicePlane.from_tensor(p, w, h) for p, (w, h) in zip(f, dims)] for f in out]
        state["engines"].append((engine, out, planes))
    return state


def _run_stream(state):
    if "host" in state:
        host, out, n = state["host"], state["out"], 0
        host.reset_stream()
        for planes in state["wire"]:
            while True:
                try:
                    host.push(planes)
                    break
                except avd.QueueFull:
                    n += bool(host.recv_into(out[n]))
        while n < len(out) and host.recv_into(out[n]):
            n += 1
        tail = []
        host.flush(tail.append)
        frames = [[np.frombuffer(p, np.uint8) for p in f] for f in out[:n]]
        return frames + [[np.frombuffer(p, np.uint8) for p in f] for f in tail]
    for engine, _, _ in state["engines"]:
        engine.reset()
    done = [0] * len(state["engines"])
    for planes in state["planes"]:
        for i, (engine, _, out) in enumerate(state["engines"]):
            for _ in range(engine.push(planes)):
                engine.emit_into(out[done[i]])
                done[i] += 1
    for i, (engine, _, out) in enumerate(state["engines"]):
        for _ in range(engine.finish()):
            engine.emit_into(out[done[i]])
            done[i] += 1
    return [out for _, out, _ in state["engines"]]


# ---- the batched launch -------------------------------------------------------------------------


def _batch_clips(case):
    """(width, height, frames, temporal radius) of each clip, written as 640x360x5r2."""
    return [tuple(int(v) for v in c.replace("r", "x").split("x")) for c in case["clips"].split()]


def _batch_weights(case, radius):
    """A clip's strength and noise offset: the HQ defaults at the case's pinned sigma."""
    sigma = case["noise"] / 255.0
    strength = float(avd.hq_default_strength(1, radius)) * case["noise"]
    return strength, float(np.float32(6.0) * np.float32(sigma) ** 2 * np.float32((2 * case["s"] + 1) ** 2))


def _prepare_batch(case, seed):
    gen, rng = _generators(seed)
    clips = []
    for w, h, n, _ in _batch_clips(case):
        clips.append((torch.stack(_series(gen, rng, w, h, n, case["noise"], 2)).clamp(0, 255) / 255.0).contiguous())
    outs = [torch.zeros_like(c) for c in clips]
    jobs = []
    for clip, out, (_, _, _, radius) in zip(clips, outs, _batch_clips(case)):
        n, h, w = clip.shape
        strength, offset = _batch_weights(case, radius)
        for k in range(n):
            jobs.append(_abi.AvdBatchJob(clip.data_ptr(), out[k].data_ptr(), n, k, radius, w, h, strength, offset,
                                         offset))
    scratch = torch.zeros(_abi.load().avd_batch_scratch_bytes(len(jobs), case["a"]) // 4, dtype=torch.int32,
                          device="cuda")
    return dict(case=case, clips=clips, outs=outs, jobs=(_abi.AvdBatchJob * len(jobs))(*jobs), n=len(jobs),
                scratch=scratch)


def _run_batch(state):
    case, lib = state["case"], _abi.load()
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    if lib.avd_batch_submit(state["jobs"], state["n"], 1, case["a"], case["s"], 1.0, state["scratch"].data_ptr(),
                            stream):
        raise RuntimeError(lib.avd_last_error().decode())
    return state["outs"]


# ---- the differentiable passes ------------------------------------------------------------------


def _window(case, seed):
    gen, rng = _generators(seed)
    n = 2 * case["d"] + 1
    chans = [torch.stack(_series(gen, rng, case["w"], case["h"], n, case["noise"], 1)) for _ in range(case["c"])]
    win = (torch.stack(chans, dim=-1).clamp(0, 255) / 255.0).contiguous()
    grad = torch.randn(win.shape[1:], generator=gen, device="cuda")
    return win, grad


def _prepare_grad(case, seed):
    window, grad = _window(case, seed)
    if case["kind"] == "nlm_grad":
        return dict(case=case, window=window.requires_grad_(), grad=grad,
                    strength=torch.tensor(case["strength"], device="cuda", requires_grad=True))
    sigma = torch.full((case["c"],), case["noise"] / 255.0, device="cuda", requires_grad=True)
    config = Nl4dPassConfig(radius=case["d"], spatial_radius=case["spatial_radius"], wiener=case["wiener"],
                            pool_ratio=2.42 / 2.7 if case["pooled"] else None)
    return dict(case=case, window=window.requires_grad_(), grad=grad, sigma=sigma, config=config)


def _run_grad(state):
    case = state["case"]
    if case["kind"] == "nlm_grad":
        out = NlmWindow.apply(state["window"], state["strength"], case["d"], case["a"], case["s"])
        gw, gs = torch.autograd.grad(out, (state["window"], state["strength"]), state["grad"])
    else:
        out = Nl4dPass.apply(state["window"], state["sigma"], state["config"])
        gw, gs = torch.autograd.grad(out, (state["window"], state["sigma"]), state["grad"])
    return [out.detach(), gw, gs]


# ---- the interface ------------------------------------------------------------------------------


def prepare(case, seed):
    return {"stream": _prepare_stream, "batch": _prepare_batch}.get(case["kind"], _prepare_grad)(case, seed)


def run(state):
    return {"stream": _run_stream, "batch": _run_batch}.get(state["case"]["kind"], _run_grad)(state)


# Per (pixel, offset, channel): difference, square, two running box sums (four adds), and the weight's
# scale, exponential, sum and product.
def _nlm_flops(pixels, channels, d, a, frames):
    offsets = (2 * a + 1) ** 2 * (2 * d + 1) - 1
    return pixels * offsets * (2 * channels + 8) * frames


# Per reference patch (a step-4 grid): every centre candidate's and one refine rectangle per neighbour's
# 64 squared differences, and eight members' transforms both ways.
def _nl4d_flops(pixels, channels, d, radius, frames):
    candidates = (2 * radius + 1) ** 2 + 2 * 2 * d * 25
    return pixels / 16 * channels * (candidates * 192 + 24000) * frames


def work(case):
    if case["kind"] == "batch":
        clips = _batch_clips(case)
        return {"bytes": sum(8 * w * h * n for w, h, n, _ in clips),
                "flops": sum(_nlm_flops(w * h, 1, r, case["a"], n) for w, h, n, r in clips)}
    if case["kind"] != "stream":
        p, c, n = case["w"] * case["h"], case["c"], 2 * case["d"] + 1
        one = (_nlm_flops(p, c, case["d"], case["a"], 1) if case["kind"] == "nlm_grad" else
               _nl4d_flops(p, c, case["d"], case["spatial_radius"], 1))
        # window read twice, output written, upstream gradient read, window gradient written
        return {"bytes": 4 * p * c * (3 * n + 2), "flops": 3 * one}
    geometry = _geometry(case)
    sample = {8: 1, 32: 4}.get(case["depth"], 2)
    dims = [geometry.plane_dims(i) for i in range(geometry.plane_count())]
    engines = 2 if case["algo"] == "nlm_pair" else 1
    total = sum(w * h for w, h in dims) * sample * 2 * case["frames"] * engines
    flops = 0.0
    for group, channels in (("luma", 1), ("chroma", 2)):
        if case["planes"] not in (group, "both"):
            continue
        w, h = dims[0 if channels == 1 else 1]
        if case["algo"] == "nl4d":
            flops += _nl4d_flops(w * h, channels, case["d"], case.get("spatial_radius", 9), case["frames"])
        else:
            d = 0 if case["algo"] == "nlm_pair" and channels == 2 else case["d"]
            flops += _nlm_flops(w * h, channels, d, case["a"], case["frames"])
    return {"bytes": total, "flops": flops}


# ---- the 64-bit values --------------------------------------------------------------------------


def _box(v, s):
    """Sums of `v` (H+2s, W+2s) over every (2s+1)^2 patch."""
    k = 2 * s + 1
    h, w = v.shape[0] - 2 * s, v.shape[1] - 2 * s
    rows = sum(v[i:i + h] for i in range(k))
    return sum(rows[:, i:i + w] for i in range(k))


def _offsets(d, a):
    for f in range(2 * d + 1):
        for qy in range(-a, a + 1):
            for qx in range(-a, a + 1):
                if f != d or qy or qx:
                    yield f, qy, qx


def _nlm_exact(frames, a, s, strength, offset=0.0, grad=None):
    """One windowed NLMeans frame in float64 from frames (2d+1, H, W, C): the output, and with an upstream
    gradient also dL/d(frames) and dL/d(strength)."""
    x = frames.to(torch.float64)
    n, h, w, c = x.shape
    d, m = n // 2, a + s
    scale = 3.0 if c == 1 else 1.5
    h2 = 65025.0 / (3.0 * strength * strength * (2 * s + 1) ** 2)
    yi = torch.arange(-m, h + m, device=x.device).clamp(0, h - 1)
    xi = torch.arange(-m, w + m, device=x.device).clamp(0, w - 1)
    pad = x[:, yi][:, :, xi]
    centre = pad[d, a:a + h + 2 * s, a:a + w + 2 * s]
    num, wsum = torch.zeros_like(x[d]), torch.zeros_like(x[d, ..., 0])
    best = torch.zeros_like(wsum)

    def weigh(f, qy, qx):
        diff = centre - pad[f, a + qy:a + qy + h + 2 * s, a + qx:a + qx + w + 2 * s]
        excess = scale * _box((diff * diff).sum(-1), s) - offset
        return diff, excess.clamp(min=0.0), pad[f, m + qy:m + qy + h, m + qx:m + qx + w]

    for q in _offsets(d, a):
        _, excess, value = weigh(*q)
        wt = torch.exp(-excess * h2)
        num += wt[..., None] * value
        wsum += wt
        best = torch.maximum(best, wt)
    den = best + wsum
    live = den > 1e-30  # a pixel without any weight passes through, as the kernels' finish has it
    den = torch.where(live, den, torch.ones_like(den))
    out = torch.where(live[..., None], (x[d] * best[..., None] + num) / den[..., None], x[d])
    if grad is None:
        return out
    g = grad.to(torch.float64).reshape(out.shape)
    passed = g * ~live[..., None]
    g = g * live[..., None]
    gpad, taken = torch.zeros_like(pad), torch.zeros_like(best, dtype=torch.bool)
    gcentre = torch.zeros_like(centre)
    gx = torch.zeros_like(x)
    gx[d] = passed + g * (best / den)[..., None]
    gbest = (g * (x[d] - out)).sum(-1) / den
    gh2 = torch.zeros((), dtype=torch.float64, device=x.device)
    for f, qy, qx in _offsets(d, a):
        diff, excess, value = weigh(f, qy, qx)
        wt = torch.exp(-excess * h2)
        gw = (g * (value - out)).sum(-1) / den
        first = (wt == best) & ~taken
        taken |= first
        gw = gw + torch.where(first, gbest, torch.zeros_like(gbest))
        gh2 -= (gw * wt * excess).sum()
        gpad[f, m + qy:m + qy + h, m + qx:m + qx + w] += g * (wt / den)[..., None]
        gd = torch.nn.functional.pad(gw * wt * (-h2) * (excess > 0), (2 * s,) * 4)
        gdiff = 2.0 * scale * _box(gd, s)[..., None] * diff
        gcentre += gdiff
        gpad[f, a + qy:a + qy + h + 2 * s, a + qx:a + qx + w + 2 * s] -= gdiff
    gpad[d, a:a + h + 2 * s, a:a + w + 2 * s] += gcentre
    rows = torch.zeros((n, h, w + 2 * m, c), dtype=torch.float64, device=x.device).index_add_(1, yi, gpad)
    gx += torch.zeros_like(gx).index_add_(2, xi, rows)
    return out, gx, gh2 * (-2.0 * h2 / strength)


def exact(case, seed):
    if case["kind"] == "batch":
        state, outs = _prepare_batch(case, seed), []
        for clip, (_, _, _, radius) in zip(state["clips"], _batch_clips(case)):
            strength, offset = _batch_weights(case, radius)
            n = clip.shape[0]
            frames = []
            for k in range(n):
                idx = [min(max(k + j, 0), n - 1) for j in range(-radius, radius + 1)]
                frames.append(_nlm_exact(clip[idx][..., None], case["a"], case["s"], strength, offset)[..., 0])
            outs.append(torch.stack(frames))
        return outs
    if case["kind"] == "nlm_grad":
        window, grad = _window(case, seed)
        return list(_nlm_exact(window, case["a"], case["s"], case["strength"], grad=grad))
    # NL4D's groups and integer planes' codes are decisions and whole numbers; only float NLMeans planes
    # have a 64-bit value.
    if case["kind"] != "stream" or case["depth"] != 32 or case["algo"] != "nlm":
        return None
    geometry = _geometry(case)
    clip = _clip(case, geometry, seed)
    n, d = case["frames"], case["d"]
    outs = [[p.to(torch.float64) for p in f] for f in clip]
    for group, idx, bias in (("luma", [0], 0.0), ("chroma", [1, 2], 0.5)):
        if case["planes"] not in (group, "both"):
            continue
        w, h = geometry.plane_dims(idx[0])
        frames = [torch.stack([f[i].reshape(h, w) + bias for i in idx], dim=-1) for f in clip]
        for k in range(n):
            window = torch.stack([frames[min(max(k + j, 0), n - 1)] for j in range(-d, d + 1)])
            res = _nlm_exact(window, case["a"], case["s"], case["strength"]) - bias
            for j, i in enumerate(idx):
                outs[k][i] = res[..., j].reshape(-1)
    return [outs]
