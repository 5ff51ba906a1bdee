"""What a user of this library has it compute, as cases that can be timed.

A case is a dict of plain values; ``kind`` says which public calls a pass makes:

* ``steps``   one ``Grid.step(n)`` call on a grid that lives on the GPU;
* ``frame``   a renderer's frame: a brush stroke, ``step(n)``, the texture
  export with its mip pyramid;
* ``surface`` the renderer's per-texel outputs, the texture export and the
  total volume of a state;
* ``batch``   one ``Batch.step(n)`` over uneven grids;
* ``io``      host state in, ``step(n)``, host state out (page-locked arrays);
* ``serve``   a stream of requests through the serving loop.

Scenes are fractal value-noise terrain (0-40 m) under a lake whose surface is
disturbed, so that water moves everywhere, shores run dry and wet again, and
rain falls on disks.  All of it follows from the seed.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import terrainwatersim_gb300 as tws
from terrainwatersim_gb300 import serve

CLOSED, OPEN = tws.BOUNDARY_CLOSED, tws.BOUNDARY_OPEN


def listed():
    return [
        # The smallest call: an interactive program advances a small grid one
        # step per call; launch and call latency decide.
        dict(name="call_256", kind="steps", W=256, H=256, steps=1, flux="f32", bound="closed",
             disks=1, radius=16),
        # A small grid run for many steps in one call (a batch job on one
        # small scene): the benchmark's 256^2, 1000-step configuration.
        dict(name="run_256", kind="steps", W=256, H=256, steps=1000, flux="f32", bound="closed",
             disks=1, radius=16),
        # The application's own frame: its 1024^2 grid with its parameters and
        # open border, one brush stroke, one step, textures and mips.
        dict(name="frame_1024", kind="frame", W=1024, H=1024, steps=1, flux="f32", bound="open",
             levels=10),
        # A medium grid of odd sides, open border, rain and a standing brush.
        dict(name="run_1021x763", kind="steps", W=1021, H=763, steps=100, flux="f32",
             bound="open", disks=2, radius=24, brush=True),
        # An ordinary single grid.
        dict(name="run_2048", kind="steps", W=2048, H=2048, steps=100, flux="f32", bound="closed",
             disks=1, radius=64),
        # The headline configuration: 4096^2, one rain disk, 200 steps a call.
        dict(name="run_4096", kind="steps", W=4096, H=4096, steps=200, flux="f32", bound="closed",
             disks=1, radius=64),
        # The largest grid in both flux storages, eight rain disks.
        dict(name="run_16384", kind="steps", W=16384, H=16384, steps=24, flux="f32",
             bound="closed", disks=8, radius=128),
        dict(name="run_16384_f16", kind="steps", W=16384, H=16384, steps=24, flux="f16",
             bound="closed", disks=8, radius=128),
        # Many uneven grids advanced together.
        dict(name="batch_20", kind="batch", grids=20, lo=128, hi=2048, steps=32, flux="f32",
             bound="closed", radius=16),
        # What a renderer reads from a large state.
        dict(name="surface_4096", kind="surface", W=4096, H=4096, steps=0, flux="f32",
             bound="closed", levels=12),
        # A grid whose state comes from the host and goes back to it.
        dict(name="io_2048", kind="io", W=2048, H=2048, steps=50, flux="f32", bound="closed",
             disks=1, radius=64),
        # A burst of small and medium requests through the serving loop.
        dict(name="serve_24", kind="serve", requests=24, lo=64, hi=1024, least=100, most=800,
             flux="f16", bound="closed"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(["steps", "frame", "surface", "batch", "io", "serve"],
                       [12, 2, 2, 3, 2, 2])[0]
    flux = rng.choice(["f32", "f32", "f16"])
    bound = rng.choice(["closed", "closed", "open"])
    if kind == "batch":
        return dict(kind=kind, grids=rng.randint(3, 20), lo=64, hi=_log_int(rng, 256, 2048),
                    steps=rng.choice([1, 5, 16, 32, 50]), flux=flux, bound=bound,
                    radius=rng.randint(4, 40))
    if kind == "serve":
        return dict(kind=kind, requests=rng.randint(4, 24), lo=64, hi=_log_int(rng, 128, 1024),
                    least=50, most=_log_int(rng, 100, 800), flux=flux, bound="closed")
    side = _log_int(rng, 64, 11000 if kind == "steps" else 4096)
    W, H = side, max(48, int(side * rng.uniform(0.5, 1.3)))
    case = dict(kind=kind, W=W, H=H, flux=flux, bound=bound)
    if kind == "surface":
        case.update(steps=0, levels=rng.randint(0, int(math.log2(min(W, H)))))
    elif kind == "frame":
        case.update(steps=rng.randint(1, 10), levels=rng.randint(0, int(math.log2(min(W, H)))))
    else:
        most = max(1.0, min(1000.0, 2.5e9 / (W * H)))
        case.update(steps=_log_int(rng, 1, most), disks=rng.randint(0, 8),
                    radius=rng.randint(4, max(5, min(W, H) // 16)))
        if rng.random() < 0.2:
            case["brush"] = True
    return case


# ---- inputs -------------------------------------------------------------------
def _noise(gen, W, H, spacing, octaves):
    """Fractal value noise in [0, 1): bilinear octaves, halving in spacing and
    amplitude."""
    out = torch.zeros(H, W, device="cuda")
    amp, total = 1.0, 0.0
    for _ in range(octaves):
        lattice = torch.rand(1, 1, H // spacing + 2, W // spacing + 2, device="cuda",
                             generator=gen)
        out += amp * torch.nn.functional.interpolate(lattice, size=(H, W), mode="bilinear",
                                                     align_corners=True)[0, 0]
        total += amp
        amp *= 0.5
        spacing = max(1, spacing // 2)
    return out / total


def _scene(seed, W, H):
    """(terrain, depth) float32 on the GPU: the same for the same arguments."""
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    b = 40.0 * _noise(gen, W, H, 64, 6)
    d = torch.clamp(14.0 + 8.0 * _noise(gen, W, H, 24, 2) - b, min=0.0)
    return b, d


def _params(case):
    """The library's parameters and the same three constants as plain doubles
    of the floats that the step is defined with."""
    bound = CLOSED if case["bound"] == "closed" else OPEN
    if case["kind"] == "frame":  # the application's: 60 steps a second, 1 m cells
        p = tws.params_reference(60.0, 0.98, 10.0, 1024.0, 1024, bound)
        dt = float(np.float32(1.0 / 60.0))
        k = (0.98 ** dt, dt * 10.0, dt)
    else:
        p = tws.params_physical(0.02, 9.81, 1.0, 1.0, 0.998, bound)
        k = (0.998, 0.02 * 9.81, 0.02)
    return p, tuple(float(np.float32(x)) for x in k)


def _disks(case, seed, W, H, count, rate=0.01):
    """Rain disks at whole cells, from the seed."""
    r = min(case["radius"], (min(W, H) - 1) // 2)
    rng = np.random.default_rng(seed)
    return [(tws.SOURCE_DISK, float(rng.integers(r, W - r)), float(rng.integers(r, H - r)),
             float(r), rate) for _ in range(count)]


def _sources(case, seed):
    W, H = case["W"], case["H"]
    out = _disks(case, seed, W, H, case.get("disks", 0)) if case.get("disks") else []
    if case.get("brush"):
        out = out[:tws.MAX_SOURCES - 1] + [(tws.SOURCE_BRUSH, W * 0.6, H * 0.4, 400.0, 0.02)]
    return out


def _stroke(case, seed):
    rng = np.random.default_rng(seed)
    return (tws.SOURCE_BRUSH, float(rng.uniform(0.2, 0.8) * case["W"]),
            float(rng.uniform(0.2, 0.8) * case["H"]), 900.0, 0.5)


def _batch_sizes(case):
    """Sides log-uniform in [lo, hi], aspect 1 to 2, either orientation."""
    rng = np.random.default_rng(7)
    out = []
    for i in range(case["grids"]):
        side = int(round(math.exp(rng.uniform(math.log(case["lo"]), math.log(case["hi"])))))
        other = int(round(side * rng.uniform(1.0, 2.0)))
        out.append((side, other) if i % 2 == 0 else (other, side))
    return out


def _requests(case):
    """(width, height, steps, fill) of the requests of a stream."""
    rng = np.random.default_rng(11)
    out = []
    for i in range(case["requests"]):
        side = int(round(math.exp(rng.uniform(math.log(case["lo"]), math.log(case["hi"])))))
        other = int(round(side * rng.uniform(1.0, 2.0)))
        steps = int(round(math.exp(rng.uniform(math.log(case["least"]), math.log(case["most"])))))
        W, H = (side, other) if i % 2 == 0 else (other, side)
        out.append((W, H, steps, float(rng.uniform(8, 20))))
    return out


# ---- a program's state -----------------------------------------------------------
_the_stream = None


def _stream():
    """The program's one simulation stream (grids are advanced in turn)."""
    global _the_stream
    if _the_stream is None:
        _the_stream = torch.cuda.Stream()
    return _the_stream.cuda_stream


class _DeviceArray:
    """A strided view of a grid's device memory, for torch.as_tensor; the
    tensor keeps it, and it keeps the grid."""

    def __init__(self, grid, ptr, shape, strides, typestr):
        self.grid = grid
        self.__cuda_array_interface__ = dict(data=(ptr, False), shape=shape, strides=strides,
                                             typestr=typestr, version=3)


class _Views:
    """Tensors over a grid's buffers, as a program that draws from them keeps
    them: made once for each buffer that the grid steps between."""

    def __init__(self):
        self.known = {}

    def _of(self, g, ptr, shape, strides, typestr):
        t = self.known.get(ptr)
        if t is None:
            t = self.known[ptr] = torch.as_tensor(_DeviceArray(g, ptr, shape, strides, typestr),
                                                  device="cuda")
        return t

    def state(self, g):
        """(depth, flux, flow map) of the grid as it stands."""
        b = g.buffers()
        W, H, P = b.width, b.height, b.pitch
        e, ft = (2, "<f2") if b.flux_storage == tws.FLUX_F16 else (4, "<f4")
        return (self._of(g, b.depth, (H, W), (4 * P, 4), "<f4"),
                self._of(g, b.flux, (H, W, 4), (4 * e * P, 4 * e, e), ft),
                self._of(g, b.velocity, (H, W, 2), (8 * P, 8, 4), "<f4"))

    def depth(self, g):
        b = g.buffers()
        return self._of(g, b.depth, (b.height, b.width), (4 * b.pitch, 4), "<f4")


def _flux(case):
    return tws.FLUX_F16 if case["flux"] == "f16" else tws.FLUX_F32


def _make_grid(case, seed, W, H):
    b, d = _scene(seed, W, H)
    torch.cuda.synchronize()
    g = tws.Grid(W, H, _params(case)[0], _flux(case), stream=_stream())
    g.upload_device(b.data_ptr(), d.data_ptr())
    return g


def prepare(case, seed):
    kind = case["kind"]
    s = dict(kind=kind, steps=case.get("steps", 0), views=_Views())
    if kind == "batch":
        s["batch"] = tws.Batch(_flux(case), stream=_stream())
        for i, (W, H) in enumerate(_batch_sizes(case)):
            g = _make_grid(case, 100 * seed + i, W, H)
            g.set_sources(_disks(case, 100 * seed + i, W, H, 1))
            s["batch"].add(g)
        s["views"] = [_Views() for _ in s["batch"].grids]
        return s
    if kind == "serve":
        p = _params(case)[0]
        s["flux"] = _flux(case)
        s["requests"] = []
        for i, (W, H, steps, fill) in enumerate(_requests(case)):
            rain = _disks(dict(radius=max(4, min(W, H) // 32)), 100 * seed + i, W, H, 1)
            s["requests"].append(serve.make_request(i, W, H, 100 * seed + i, fill, p, rain, steps,
                                                    0.0))
        return s
    W, H = case["W"], case["H"]
    if kind == "io":
        b, d = _scene(seed, W, H)
        s["in"] = [x.cpu().pin_memory() for x in (b, d)]
        s["out"] = [torch.empty(H, W, *n, pin_memory=True) for n in ((), (4,), (2,))]
        s["np_in"] = [x.numpy() for x in s["in"]]
        s["np_out"] = [x.numpy() for x in s["out"]]
        s["grid"] = tws.Grid(W, H, _params(case)[0], _flux(case), stream=_stream())
        s["grid"].set_sources(_sources(case, seed))
        return s
    g = s["grid"] = _make_grid(case, seed, W, H)
    if kind == "steps":
        g.set_sources(_sources(case, seed))
        return s
    # frame and surface: the renderer's own buffers
    levels = s["levels"] = case["levels"]
    s["rgba"] = torch.empty(H, W, 4, device="cuda")
    s["flow"] = torch.empty(H, W, 2, device="cuda", dtype=torch.float16)
    texels = sum((W >> l) * (H >> l) for l in range(1, levels + 1))
    s["mips"] = torch.empty(max(1, texels), 4, device="cuda")
    if kind == "frame":
        s["stroke"] = _stroke(case, seed)
    else:
        g.step(3)  # a state with flow
        s["surface"] = {n: torch.empty(H, W, *shape, device="cuda", dtype=t) for n, shape, t in (
            ("height", (), torch.float32), ("render_height", (), torch.float32),
            ("normal", (3,), torch.float32), ("flow_speed", (), torch.float32),
            ("foam", (), torch.float32), ("dry", (), torch.uint8))}
        s["out"] = tws.SurfaceOut(**{n: t.data_ptr() for n, t in s["surface"].items()})
    return s


def _export(s):
    s["grid"].export_textures(s["rgba"].data_ptr(), s["flow"].data_ptr(), s["levels"],
                              s["mips"].data_ptr() if s["levels"] else None)
    out = [s["rgba"], s["flow"]]
    return out + [s["mips"]] if s["levels"] else out


def run(s):
    kind = s["kind"]
    if kind == "steps":
        s["grid"].step(s["steps"])
        return s["views"].state(s["grid"])
    if kind == "frame":
        g = s["grid"]
        g.apply_source(s["stroke"])
        g.step(s["steps"])
        return _export(s)
    if kind == "surface":
        s["grid"].surface(s["out"])
        return [s["surface"], _export(s), s["grid"].volume()]
    if kind == "batch":
        s["batch"].step(s["steps"])
        return [v.state(g) for v, g in zip(s["views"], s["batch"].grids)]
    if kind == "io":
        g = s["grid"]
        g.io_wait()  # the arrays of this grid's previous pass are free again
        g.upload_async(*s["np_in"])
        g.step(s["steps"])
        g.download_async(s["np_out"])
        return s["out"]
    # serve: the finished grids come back; a program drops the previous ones
    s["kept"] = None
    with serve.Server(flux_storage=s["flux"], keep_grids=True) as server:
        for r in s["requests"]:
            server.submit(r)
        server.close_submissions()
        server.run()
        results = sorted(server.results(), key=lambda r: r.id)
    s["kept"] = [r.grid for r in results]
    s["views"] = _Views()
    return [[s["views"].depth(r.grid) for r in results], [r.volume for r in results]]


def work(case):
    kind, f = case["kind"], 8 if case["flux"] == "f16" else 16
    # one step, per cell: 8 products and sums and 4 maxima of the outflows, 4
    # of the scaling test, 11 of the depth and 6 of the flow map
    per_step = 40.0
    step_bytes = 4 + 4 + f + 4 + f + 8  # b, d, f in; d, f, flow map out
    if kind == "batch":
        cells = sum(W * H for W, H in _batch_sizes(case))
        return dict(bytes=cells * step_bytes, flops=cells * case["steps"] * per_step)
    if kind == "serve":
        r = _requests(case)
        return dict(bytes=sum(W * H * step_bytes for W, H, _, _ in r),
                    flops=sum(W * H * n * per_step for W, H, n, _ in r))
    cells = case["W"] * case["H"]
    if kind == "steps":
        return dict(bytes=cells * step_bytes, flops=cells * case["steps"] * per_step)
    if kind == "io":  # host to device and back
        return dict(bytes=cells * (8 + 28), flops=cells * case["steps"] * per_step)
    mips = sum((case["W"] >> l) * (case["H"] >> l) for l in range(1, case["levels"] + 1))
    export = cells * (16 + 4) + mips * 16
    if kind == "frame":
        return dict(bytes=cells * step_bytes + export,
                    flops=cells * case["steps"] * per_step + mips * 16)
    # surface: b, d and the flow map in; six outputs; the export; the volume
    return dict(bytes=cells * (16 + 29) + export, flops=cells * 40.0 + mips * 16)


# ---- the same in 64 bits -------------------------------------------------------------
def _add_sources(d, sources):
    H, W = d.shape
    x = torch.arange(W, device="cuda", dtype=torch.float64)
    y = torch.arange(H, device="cuda", dtype=torch.float64)[:, None]
    for kind, cx, cy, radius, rate in sources:
        rate = float(np.float32(rate))
        cx, cy = float(np.float32(cx)), float(np.float32(cy))
        if kind == tws.SOURCE_DISK:
            r = int(radius)
            ys = slice(max(0, int(cy) - r), int(cy) + r + 1)
            xs = slice(max(0, int(cx) - r), int(cx) + r + 1)
            inside = (x[xs] - cx) ** 2 + (y[ys] - cy) ** 2 <= r * r
            d[ys, xs] += rate * inside
        else:
            q = ((x - cx) ** 2 + (y - cy) ** 2) / float(np.float32(radius))
            d += torch.clamp(1.0 - q, 0.0, 1.0) * rate


def _steps64(b, d, constants, closed, sources, steps):
    """The step's definition in float64: (depth, four outflows, flow map)."""
    kf, ka, c = constants
    H, W = b.shape
    f = [torch.zeros_like(d) for _ in range(4)]
    vx = vy = torch.zeros_like(d)
    hp = torch.zeros(H + 2, W + 2, device="cuda", dtype=torch.float64)
    fp = [torch.zeros_like(hp) for _ in range(4)]
    mid = (slice(1, -1), slice(1, -1))
    px, mx, py, my = ((slice(1, -1), slice(2, None)), (slice(1, -1), slice(0, -2)),
                      (slice(2, None), slice(1, -1)), (slice(0, -2), slice(1, -1)))
    for n in range(steps):
        _add_sources(d, sources)
        torch.add(d, b, out=hp[mid])
        h = hp[mid]
        for k, nb in enumerate((px, mx, py, my)):
            f[k].mul_(kf).add_(torch.sub(h, hp[nb]), alpha=ka).clamp_(min=0.0)
        if closed:
            f[0][:, -1] = 0.0
            f[1][:, 0] = 0.0
            f[2][-1] = 0.0
            f[3][0] = 0.0
        total = (f[0] + f[1]).add_(f[2]).add_(f[3]).mul_(c)
        scale = torch.where(total > d, d / total.clamp(min=1e-300), 1.0)
        del total
        for k in range(4):
            f[k].mul_(scale)
            fp[k][mid] = f[k]
        x1, x0, y1, y0 = fp[1][px], fp[0][mx], fp[3][py], fp[2][my]
        change = (x1 + x0).add_(y1).add_(y0)
        for k in range(4):
            change.sub_(f[k])
        d.add_(change, alpha=c).clamp_(min=0.0)
        del change, scale
        if n == steps - 1:
            vx = (x1 - f[0]).sub_(x0 - f[1])
            vy = (y1 - f[2]).sub_(y0 - f[3])
    return d, f, vx, vy


def _state64(case, seed, W, H, sources, steps, scene=None):
    b, d = scene if scene is not None else (x.double() for x in _scene(seed, W, H))
    _, constants = _params(case)
    d, f, vx, vy = _steps64(b, d, constants, case["bound"] == "closed", sources, steps)
    return b, d, f, vx, vy


def _stored_scale(case):
    """FP16 storage keeps flux times a power of two that puts the largest
    outflow of 32 m deep water at 2^12 to 2^13."""
    if case["flux"] != "f16":
        return 1.0
    return 2.0 ** math.floor(math.log2(8192.0 * _params(case)[1][2] / 32.0))


def _outputs64(case, state):
    _, d, f, vx, vy = state
    return [d, torch.stack(f, -1).mul_(_stored_scale(case)), torch.stack((vx, vy), -1)]


def _textures64(b, d, vx, vy, levels):
    rgba = torch.full((*b.shape, 4), 0.3, device="cuda", dtype=torch.float64)
    rgba[..., 0], rgba[..., 3] = b, d
    mips, m = [], rgba
    for _ in range(levels):
        h, w = m.shape[0] // 2 * 2, m.shape[1] // 2 * 2
        m = m[:h, :w].reshape(h // 2, 2, w // 2, 2, 4).mean((1, 3))
        mips.append(m.reshape(-1, 4))
    out = [rgba, torch.stack((vx, vy), -1)]
    return out + [torch.cat(mips)] if levels else out


def _pcg_stream(seed, sequence, count):
    """`count` outputs of O'Neill's PCG32 (XSH-RR 64/32) as 24-bit fractions."""
    mult, inc, mask = 6364136223846793005, (sequence << 1) | 1, (1 << 64) - 1
    state = ((inc + seed) * mult + inc) & mask
    # state k = mult^k state + inc (mult^(k-1) + ... + 1), modulo 2^64
    powers = np.full(count, mult, np.uint64)
    powers[0] = 1
    powers = np.multiply.accumulate(powers)
    sums = np.concatenate([np.zeros(1, np.uint64), np.add.accumulate(powers)[:-1]])
    old = powers * np.uint64(state) + sums * np.uint64(inc)
    xs = (((old >> np.uint64(18)) ^ old) >> np.uint64(27)).astype(np.uint32)
    rot = (old >> np.uint64(59)).astype(np.uint32)
    bits = (xs >> rot) | (xs << ((np.uint32(32) - rot) & np.uint32(31)))
    return (bits >> np.uint32(8)).astype(np.float64) / 16777216.0


def _generated_scene64(seed, W, H, fill):
    """tws_generate_scene's terrain (six octaves of PCG32 value noise,
    smoothstep-bilinear, 0-40 m) and lake, in 64 bits."""
    x, y = np.arange(W), np.arange(H)[:, None]
    acc = np.zeros((H, W))
    for o in range(6):
        s = 64 >> o
        lx, ly = W // s + 2, H // s + 2
        v = _pcg_stream(seed, o + 1, lx * ly).reshape(ly, lx)
        i, j = x // s, y // s
        tx, ty = (x % s) / s, (y % s) / s
        tx, ty = tx * tx * (3 - 2 * tx), ty * ty * (3 - 2 * ty)
        top = v[j, i] + (v[j, i + 1] - v[j, i]) * tx
        low = v[j + 1, i] + (v[j + 1, i + 1] - v[j + 1, i]) * tx
        acc += 0.5 ** o * (top + (low - top) * ty)
    b = torch.from_numpy(acc / 1.96875 * 40.0).cuda()
    return b, torch.clamp(float(np.float32(fill)) - b, min=0.0)


def exact(case, seed):
    kind, steps = case["kind"], case.get("steps", 0)
    if kind == "batch":
        return [_outputs64(case, _state64(case, 100 * seed + i, W, H,
                                          _disks(case, 100 * seed + i, W, H, 1), steps))
                for i, (W, H) in enumerate(_batch_sizes(case))]
    if kind == "serve":
        depths, volumes = [], []
        for i, (W, H, n, fill) in enumerate(_requests(case)):
            rain = _disks(dict(radius=max(4, min(W, H) // 32)), 100 * seed + i, W, H, 1)
            d = _state64(case, 0, W, H, rain, n, _generated_scene64(100 * seed + i, W, H, fill))[1]
            depths.append(d)
            volumes.append(float(d.sum()))
        return [depths, volumes]
    W, H = case["W"], case["H"]
    if kind in ("steps", "io"):
        out = _outputs64(case, _state64(case, seed, W, H, _sources(case, seed), steps))
        if kind == "io":  # flux comes back in metres, whatever its storage
            out[1].div_(_stored_scale(case))
        return out
    if kind == "frame":
        b, d = (x.double() for x in _scene(seed, W, H))
        _add_sources(d, [_stroke(case, seed)])
        b, d, _, vx, vy = _state64(case, seed, W, H, [], steps, (b, d))
        return _textures64(b, d, vx, vy, case["levels"])
    b, d, _, vx, vy = _state64(case, seed, W, H, [], 3)
    h = b + d
    dry = d < 0.1
    A = torch.roll(h, -1, 0) - torch.roll(h, 1, 0)  # neighbours wrap around
    B = torch.roll(h, -1, 1) - torch.roll(h, 1, 1)
    n = torch.stack((-B, torch.ones_like(h), -A), -1)
    speed2 = vx * vx + vy * vy
    surface = dict(height=h, render_height=torch.where(dry, h - 10.1, h - 0.1),
                   normal=n / n.norm(dim=-1, keepdim=True), flow_speed=speed2.sqrt(),
                   foam=torch.clamp(speed2 * 0.00004, 0.0, 1.0), dry=None)
    return [surface, _textures64(b, d, vx, vy, case["levels"]), float(d.sum())]
