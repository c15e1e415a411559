"""Workloads of the reconstruction framework, for timing and for comparing results.

Each case is one pass of a program that uses the public entry points: the
holograms, transfer functions and plans it has in hand are made in ``prepare``,
the calls it makes per frame are ``run``.  Holograms are inline holograms of
opaque discs (lambda = 0.6328 um, pitch 10 um), generated from the seed with
plain torch.  Floating results are compared with ``exact``, the same chain in
64 bits; labels and boxes are whole numbers and have to be equal.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

from __graft_entry__ import load_package

LAM, DX = 0.6328, 10.0                      # um
LENGTHS = [128, 192, 256, 384, 512, 768, 1024, 1536, 2048]   # transform lengths in use: 2^a and 3 * 2^a
DTYPES = {"f16": torch.float16, "f32": torch.float32, "c64": torch.complex64}


def listed():
    return [
        # a live preview of a binned camera: the smallest frame, where launches and latency count
        {"name": "proj-256x32", "kind": "proj", "nx": 256, "ny": 256, "slices": 32, "dz": 200.0, "lpf": False},
        # one Gabor hologram of an ordinary camera, projection over 256 slices
        {"name": "proj-1024x256", "kind": "proj", "nx": 1024, "ny": 1024, "slices": 256, "dz": 200.0, "lpf": False},
        # a rectangular sensor and a slice count that divides nothing
        {"name": "proj-2048x1536x157", "kind": "proj", "nx": 2048, "ny": 1536, "slices": 157, "dz": 317.0,
         "lpf": False},
        # the largest frame: 4096^2 over 1024 slices
        {"name": "proj-4096x1024", "kind": "proj", "nx": 4096, "ny": 4096, "slices": 1024, "dz": 190.0, "lpf": False},
        # the two-plane frame: 20 Gerchberg-Saxton iterations, then 512 slices
        {"name": "frame-2048x512", "kind": "frame", "n": 2048, "iters": 20, "slices": 512, "dz": 200.0},
        # phase retrieval alone, as for a recorded pair with 9 iterations
        {"name": "gs-1024x9", "kind": "gs", "n": 1024, "iters": 9},
        # the volume a particle search walks through, with its projection
        {"name": "vol-1024x250-f32", "kind": "vol", "nx": 1024, "ny": 1024, "slices": 250, "dz": 100.0,
         "dtype": "f32"},
        # the complex amplitude around a few particles of a small, not power-of-two frame
        {"name": "vol-768x65-c64", "kind": "vol", "nx": 768, "ny": 768, "slices": 65, "dz": 150.0, "dtype": "c64"},
        # one propagation by a new distance (its transfer function included): refocusing by hand
        {"name": "prop-2048", "kind": "prop", "n": 2048, "z": 80000.0},
        # labels and roots of one thresholded projection
        {"name": "label-2048", "kind": "label", "nx": 2048, "ny": 2048, "slices": 1, "blobs": 800, "noise": 1e-4},
        # per-slice labels and boxes of a thresholded volume: the 3-D particle search
        {"name": "detect-1024x100", "kind": "label", "nx": 1024, "ny": 1024, "slices": 100, "blobs": 300,
         "noise": 1e-5},
        # a mixed batch of recorded holograms of four sizes, planned once
        {"name": "batch-24", "kind": "batch", "items": 24, "plan": 1000},
    ]


def _log_int(rng: random.Random, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    kind = rng.choice(["proj", "proj", "frame", "gs", "vol", "vol", "prop", "label", "label", "batch"])
    if kind in ("proj", "vol"):
        nx, ny = rng.choice(LENGTHS), rng.choice(LENGTHS)
        if rng.random() < 0.5:
            ny = nx
        case = {"kind": kind, "nx": nx, "ny": ny, "dz": round(rng.uniform(50.0, 500.0), 1)}
        if kind == "proj":
            case["slices"] = _log_int(rng, 8, 512)
            case["lpf"] = rng.random() < 0.3
        else:
            case["dtype"] = rng.choice(["f32", "f32", "f16", "c64"])
            case["slices"] = _log_int(rng, 4, min(512, (1 << 29) // (nx * ny)))
        return case
    if kind == "frame":
        return {"kind": kind, "n": rng.choice(LENGTHS[2:]), "iters": rng.randint(2, 20),
                "slices": _log_int(rng, 16, 512), "dz": round(rng.uniform(50.0, 500.0), 1)}
    if kind == "gs":
        return {"kind": kind, "n": rng.choice(LENGTHS), "iters": rng.randint(1, 20)}
    if kind == "prop":
        return {"kind": kind, "n": rng.choice(LENGTHS), "z": round(rng.uniform(500.0, 200000.0), 1)}
    if kind == "label":
        nx, ny = _log_int(rng, 100, 2048), _log_int(rng, 100, 2048)   # any size: no transform is involved
        slices = 1 if rng.random() < 0.5 else _log_int(rng, 2, min(250, (1 << 28) // (nx * ny)))
        return {"kind": kind, "nx": nx, "ny": ny, "slices": slices, "blobs": _log_int(rng, 10, 1500),
                "noise": rng.choice([0.0, 1e-5, 1e-4, 1e-3])}
    return {"kind": "batch", "items": rng.randint(3, 24), "plan": rng.randint(1, 1 << 20)}


def _batch_items(case):
    """(nx, ny, slices, dz) of a mixed batch: a third 512^2, a third 1024^2, the rest 2048 x 1536 and 2048^2."""
    rng = random.Random(case["plan"])
    out = []
    for i in range(case["items"]):
        nx, ny = [(512, 512), (1024, 1024), (2048, 1536), (512, 512), (1024, 1024), (2048, 2048)][i % 6]
        out.append((nx, ny, rng.randint(32, 512), rng.uniform(100.0, 500.0)))
    return out


# ---------------------------------------------------------------- inputs

def _generator(seed: int) -> torch.Generator:
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _kernel(nx: int, ny: int, z: float, dtype=torch.float32) -> torch.Tensor:
    """exp(i 2 pi z sqrt(1/lambda^2 - fx^2 - fy^2)) in natural frequency order."""
    fx = torch.fft.fftfreq(nx, DX, dtype=torch.float64, device="cuda")
    fy = torch.fft.fftfreq(ny, DX, dtype=torch.float64, device="cuda")
    w = torch.sqrt((1.0 / LAM ** 2 - fy[:, None] ** 2 - fx[None, :] ** 2).clamp_min(0.0))
    return torch.polar(torch.ones_like(w), torch.remainder(w * z, 1.0) * (2 * math.pi)).to(torch.complex64)


def _holograms(nx: int, ny: int, g: torch.Generator, planes_at=(0.0,)):
    """Float32 inline holograms of one disc field, recorded at the given sensor positions."""
    planes, per = 4, max(2, nx * ny // (4 * 6000))          # about 700 discs at 2048^2
    x = (torch.arange(nx, device="cuda") + nx // 2) % nx - nx // 2
    y = (torch.arange(ny, device="cuda") + ny // 2) % ny - ny // 2
    r2 = (x[None, :] ** 2 + y[:, None] ** 2).float()
    fields = [torch.zeros((ny, nx), dtype=torch.complex64, device="cuda") for _ in planes_at]
    for p in range(planes):
        at = torch.randint(0, nx * ny, (per,), generator=g, device="cuda")
        points = torch.zeros(nx * ny, device="cuda")
        points[at] = 1.0
        radius = 0.6 + 0.8 * p                               # 12 .. 60 um across
        disc = torch.fft.fft2((r2 <= radius * radius).float())
        mask = torch.fft.ifft2(torch.fft.fft2(points.view(ny, nx)) * disc).real > 0.5
        spec = torch.fft.fft2(mask.to(torch.complex64))
        z = 5000.0 + 25000.0 * (p + torch.rand((), generator=g, device="cuda").item())
        for f, s in zip(fields, planes_at):
            f += torch.fft.ifft2(spec * _kernel(nx, ny, z + s))
    out = []
    for f in fields:
        i = (1.0 - f).abs().square()
        i = (i - i.min()) / (i.max() - i.min())
        i = i + 0.01 * torch.randn(i.shape, generator=g, device="cuda")
        out.append(i.clamp_min(0.0).contiguous())
    return out


def _field(n: int, g: torch.Generator) -> torch.Tensor:
    """A complex field: a hologram's amplitude with a smooth phase."""
    amp = torch.sqrt(_holograms(n, n, g)[0])
    t = torch.arange(n, device="cuda", dtype=torch.float32) * (2 * math.pi / n)
    return torch.polar(amp, 0.7 * torch.sin(3 * t)[:, None] + 0.5 * torch.cos(2 * t)[None, :]).contiguous()


def _binary(case, g: torch.Generator) -> torch.Tensor:
    """A thresholded volume: discs that widen away from their focus, and single noise pixels."""
    nx, ny, slices = case["nx"], case["ny"], case["slices"]
    vol = torch.rand((slices, ny, nx), generator=g, device="cuda") < case["noise"]
    u = torch.rand((case["blobs"], 4), generator=g, device="cuda").cpu().tolist()
    for cx, cy, cz, cr in u:
        x, y, z, r = cx * nx, cy * ny, cz * slices, 1.0 + 9.0 * cr * cr
        reach = 0 if slices == 1 else 6
        z0, z1 = max(0, int(z) - reach), min(slices, int(z) + reach + 1)
        h = int(r + reach) + 1
        x0, x1, y0, y1 = max(0, int(x) - h), min(nx, int(x) + h + 1), max(0, int(y) - h), min(ny, int(y) + h + 1)
        zz = torch.arange(z0, z1, device="cuda", dtype=torch.float32)[:, None, None]
        yy = torch.arange(y0, y1, device="cuda", dtype=torch.float32)[None, :, None]
        xx = torch.arange(x0, x1, device="cuda", dtype=torch.float32)[None, None, :]
        rad = r + 0.5 * (zz - int(z)).abs()
        vol[z0:z1, y0:y1, x0:x1] |= (xx - x) ** 2 + (yy - y) ** 2 <= rad * rad
    return vol


Z0, SEPARATION = 5000.0, 5000.0             # first slice, distance of the two recording planes


def _inputs(case, seed):
    """The arrays of the case, without this framework's code."""
    g = _generator(seed)
    kind = case["kind"]
    if kind in ("proj", "vol"):
        return {"holo": _holograms(case["nx"], case["ny"], g)[0]}
    if kind in ("gs", "frame"):
        h1, h2 = _holograms(case["n"], case["n"], g, (0.0, SEPARATION))
        return {"h1": h1, "h2": h2}
    if kind == "prop":
        return {"field": _field(case["n"], g)}
    if kind == "label":
        return {"vol": _binary(case, g)}
    return {"holos": [_holograms(nx, ny, g)[0] for nx, ny, _, _ in _batch_items(case)]}


def prepare(case, seed):
    ph = load_package()
    s = dict(_inputs(case, seed), case=case, ph=ph)
    kind = case["kind"]

    def optics(nx, ny, *distances):
        d = ph.cu_transfer_sqrt_arr(nx, LAM, DX, n_slow=ny)
        return [ph.cu_transfer(z, nx, LAM, d) for z in distances]

    if kind in ("proj", "vol"):
        s["front"], s["step"] = optics(case["nx"], case["ny"], -Z0, -case["dz"])
        if kind == "proj" and case["lpf"]:
            s["mask"] = _low_pass(case["nx"], case["ny"])
    if kind in ("gs", "frame"):
        s["there"], s["back"] = optics(case["n"], case["n"], SEPARATION, -SEPARATION)
    if kind == "frame":
        s["front"], s["step"] = optics(case["n"], case["n"], -Z0, -case["dz"])
    if kind == "prop":
        s["d_sqr"] = ph.cu_transfer_sqrt_arr(case["n"], LAM, DX)
        s["in"] = ph.CuWavefront(s["field"])
        s["out"] = ph.CuWavefront(torch.empty_like(s["field"]))
    if kind == "label":   # the program's table of components, with room for all that it expects
        rows = 1024 + 2 * (case["blobs"] * min(case["slices"], 13) + int(case["noise"] * s["vol"].numel()))
        s["table"] = np.zeros(rows if case["slices"] == 1 else (rows, 5), dtype=np.int64)
    if kind == "batch":
        items = []
        for holo, (nx, ny, slices, dz) in zip(s["holos"], _batch_items(case)):
            front, step = optics(nx, ny, -Z0, -dz)
            items.append({"hologram": holo, "transfer_front": front, "transfer_dz": step, "slices": slices})
        s["batch"] = ph.ReconBatch(items, lanes=4, return_argmin=False)
    return s


def _low_pass(nx: int, ny: int) -> torch.Tensor:
    """A smooth centred low-pass mask of any shape, as a program makes its own."""
    x = (torch.arange(nx, device="cuda", dtype=torch.float32) - nx // 2) / (0.35 * nx)
    y = (torch.arange(ny, device="cuda", dtype=torch.float32) - ny // 2) / (0.35 * ny)
    return torch.exp(-((x[None, :] ** 2 + y[:, None] ** 2) ** 3)).contiguous()


# ---------------------------------------------------------------- one pass

def run(state):
    ph, case = state["ph"], state["case"]
    kind = case["kind"]
    if kind == "proj":
        wave = ph.cu_gabor_wavefront(state["holo"])
        if case["lpf"]:
            return ph.cu_get_reconst_xyprojection_lpf(wave, state["front"], state["step"], state["mask"],
                                                      case["slices"])
        return ph.cu_get_reconst_xyprojection(wave, state["front"], state["step"], case["slices"])
    if kind in ("gs", "frame"):
        wave = ph.cu_phase_retrieval_holo(state["h1"], state["h2"], state["there"], state["back"], case["iters"],
                                          case["n"])
        if kind == "gs":
            return wave.data
        proj = ph.cu_get_reconst_xyprojection(wave, state["front"], state["step"], case["slices"])
        return {"field": wave.data, "proj": proj}
    if kind == "vol":
        wave = ph.cu_gabor_wavefront(state["holo"])
        if case["dtype"] == "c64":
            return ph.cu_get_reconst_complex_vol(wave, state["front"], state["step"], case["slices"])
        vol, proj = ph.cu_get_reconst_vol_and_xyprojection(wave, state["front"], state["step"], case["slices"],
                                                           DTYPES[case["dtype"]])
        return {"vol": vol, "proj": proj}
    if kind == "prop":
        ph.cu_asm_prop_(state["out"], state["in"], state["d_sqr"], case["z"], case["n"], LAM)
        return state["out"].data
    if kind == "label":
        vol = state["vol"]
        if case["slices"] == 1:
            labels = ph.cu_connected_component_labeling(vol[0], reference_grid=False)
            found = ph.cu_find_valid_labels(labels)
        else:
            labels = ph.cu_connected_component_labeling_batch(vol)
            found = ph.cu_bounding_rectangles(labels)
        table = state["table"]
        count = min(len(found), len(table))
        table[:count] = found[:count]
        table[count:] = 0
        return {"labels": labels.view(torch.int32), "components": table}
    return state["batch"].run()[0]


# ---------------------------------------------------------------- what a pass cannot do without

def _fft2_flops(nx, ny):
    return 5.0 * nx * ny * math.log2(nx * ny)


def _slices_work(nx, ny, slices, out_bytes):
    """A hologram or field and two transfers in, `out_bytes` per pixel out."""
    n = nx * ny
    return (4.0 + 16.0 + out_bytes) * n, (slices + 1) * _fft2_flops(nx, ny) + (6.0 + 3.0 + 1.0) * n * slices


def work(case):
    kind = case["kind"]
    if kind == "proj":
        b, f = _slices_work(case["nx"], case["ny"], case["slices"], 4.0 + (4.0 if case["lpf"] else 0.0))
    elif kind == "vol":
        size = {"f16": 2, "f32": 4, "c64": 8}[case["dtype"]]
        b, f = _slices_work(case["nx"], case["ny"], case["slices"],
                            size * case["slices"] + (0 if case["dtype"] == "c64" else 4))
    elif kind in ("gs", "frame"):
        n = case["n"] ** 2
        b = n * (2 * 4.0 + 2 * 8.0 + 8.0)
        f = case["iters"] * (4 * _fft2_flops(case["n"], case["n"]) + n * 2 * (6 + 8))
        if kind == "frame":
            b2, f2 = _slices_work(case["n"], case["n"], case["slices"], 4.0)
            b, f = b + b2 - 4.0 * n, f + f2
    elif kind == "prop":
        n = case["n"] ** 2
        b, f = n * (8.0 + 4.0 + 8.0), 2 * _fft2_flops(case["n"], case["n"]) + n * 10.0
    elif kind == "label":
        n = case["nx"] * case["ny"] * case["slices"]
        b, f = n * (1.0 + 4.0), n * 4.0
    else:
        b = f = 0.0
        for nx, ny, slices, _ in _batch_items(case):
            bi, fi = _slices_work(nx, ny, slices, 4.0)
            b, f = b + bi, f + fi
    return {"bytes": b, "flops": f}


# ---------------------------------------------------------------- the same in 64 bits

def _transfer(nx, ny, z):
    """The Float32 square-root term (formed in Float64), its phase in Float64, rounded to ComplexF32;
    centred order moved to natural order."""
    def term(n):
        i = torch.arange(1, n + 1, dtype=torch.float64, device="cuda")
        return ((i - n / 2.0 - 1.0) * LAM / n / DX) ** 2
    d = (1.0 - term(nx)[None, :] - term(ny)[:, None]).float()
    phase = (2.0 * math.pi * z / LAM) * torch.sqrt(d).double()
    h = torch.complex(torch.cos(phase).float(), torch.sin(phase).float())
    return torch.fft.ifftshift(h).to(torch.complex128)


def _slices64(field, nx, ny, dz, slices, mask=None):
    """The slices of a reconstruction, one complex128 array after the other."""
    x = torch.fft.fft2(field.to(torch.complex128)) * _transfer(nx, ny, -Z0)
    if mask is not None:
        x = x * torch.fft.ifftshift(mask).double()
    step = _transfer(nx, ny, -dz)
    for k in range(slices):
        if k:
            x = x * step
        yield torch.fft.ifft2(x)


def _proj64(field, nx, ny, dz, slices, mask=None):
    p = torch.full((ny, nx), math.inf, dtype=torch.float64, device="cuda")
    for u in _slices64(field, nx, ny, dz, slices, mask):
        p = torch.minimum(p, u.real.square() + u.imag.square())
    return p


def _gs64(h1, h2, n, iters):
    a1, a2 = torch.sqrt(h1).double(), torch.sqrt(h2).double()
    there, back = _transfer(n, n, SEPARATION), _transfer(n, n, -SEPARATION)
    u = a1.to(torch.complex128)
    for _ in range(iters):
        u = torch.fft.ifft2(torch.fft.fft2(u) * there)
        u = torch.polar(a2, torch.angle(u))
        u = torch.fft.ifft2(torch.fft.fft2(u) * back)
        u = torch.polar(a1, torch.angle(u))
    return u


def exact(case, seed):
    kind = case["kind"]
    if kind == "label":
        return None
    s = _inputs(case, seed)
    if kind == "proj":
        nx, ny = case["nx"], case["ny"]
        mask = _low_pass(nx, ny) if case["lpf"] else None
        return _proj64(torch.sqrt(s["holo"]), nx, ny, case["dz"], case["slices"], mask)
    if kind == "gs":
        return _gs64(s["h1"], s["h2"], case["n"], case["iters"])
    if kind == "frame":
        n = case["n"]
        u = _gs64(s["h1"], s["h2"], n, case["iters"])
        return {"field": u, "proj": _proj64(u, n, n, case["dz"], case["slices"])}
    if kind == "vol":
        nx, ny = case["nx"], case["ny"]
        slices = _slices64(torch.sqrt(s["holo"]), nx, ny, case["dz"], case["slices"])
        if case["dtype"] == "c64":
            return torch.stack(list(slices))
        vol = torch.stack([(u.real.square() + u.imag.square()).clamp(0.0, 1.0) for u in slices])
        return {"vol": vol, "proj": vol.amin(0)}
    if kind == "prop":
        n = case["n"]
        return torch.fft.ifft2(torch.fft.fft2(s["field"].to(torch.complex128)) * _transfer(n, n, case["z"]))
    return [_proj64(torch.sqrt(h), nx, ny, dz, slices)
            for h, (nx, ny, slices, dz) in zip(s["holos"], _batch_items(case))]
