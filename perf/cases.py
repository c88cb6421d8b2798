"""The work that users of this package have it do, as measured cases.

A case is one call (or one training step) through the package's public entry points:

  solve     native.solve: a JPEG file's levels on the host in, the binary64 picture, canvas,
            coefficients and records out -- the drop-in call. With record_every 10 (the default) a
            record is taken every ten iterations, with 0 only the last one.
  levels    native.solve_levels: the same, quantized on the GPU, 8-bit levels out
  batch     native.solve_batch: many pictures of uneven sizes at once
  samples   native.solve_samples: a PNG file's levels in, its picture out
  unrolled  unrolled.unrolled_tgv without gradients: a learned model's reconstruction
  train     unrolled.unrolled_tgv, a loss and its gradients: a training step of the parameters

Pictures are seeded: piecewise smooth (rectangles with ramps, Gaussian blobs) with Gaussian
noise of sigma 2, made into levels by the 8x8 DCT and the Annex K tables at a quality, as an
encoder makes them. The iterations are counted (tolerance 0), so that every side makes as many.
"""

from __future__ import annotations

import math
import os
import random
import sys

import numpy as np
import torch
import torch.utils.checkpoint

sys.path.insert(0, os.path.join(os.getcwd(), "jpeg-unround_b200"))

from unround import jpegio, native, unrolled  # noqa: E402

# T.81 Annex K, Tables K.1 and K.2, in natural order.
LUMA = [16, 11, 10, 16, 24, 40, 51, 61, 12, 12, 14, 19, 26, 58, 60, 55, 14, 13, 16, 24, 40, 57, 69, 56,
        14, 17, 22, 29, 51, 87, 80, 62, 18, 22, 37, 56, 68, 109, 103, 77, 24, 35, 55, 64, 81, 104, 113, 92,
        49, 64, 78, 87, 103, 121, 120, 101, 72, 92, 95, 98, 112, 100, 103, 99]
CHROMA = [17, 18, 24, 47, 99, 99, 99, 99, 18, 21, 26, 66, 99, 99, 99, 99, 24, 26, 56, 99, 99, 99, 99, 99,
          47, 66, 99, 99, 99, 99, 99, 99] + [99] * 32
CELLS = {"grey": (1, 1), "444": (1, 1), "422": (1, 2), "420": (2, 2)}  # luma samples a chroma sample covers
L2_BYTES = 126e6


def _case(name, kind, rows, columns, colour, method, quality, iterations, **more):
    """quality 0: a custom table of steps from 1 to 64."""
    case = {"kind": kind, "rows": rows, "columns": columns, "colour": colour, "method": method, "quality": quality,
            "iterations": iterations, "record_every": 0, "coupled": True, "pictures": 1, "checkpoint_every": 10}
    case.update(more)
    return {"name": name, **case} if name else case


def listed():
    return [
        # A thumbnail: the smallest call, all latency and launches.
        _case("thumb-tv-grey", "solve", 120, 160, "grey", "tv", 50, 100),
        # A small greyscale picture by TV (the package's first workload).
        _case("tv-grey-512", "solve", 512, 512, "grey", "tv", 30, 200),
        # A photograph of the size of the common test sets with the default settings: TGV, the
        # channels coupled, 4:2:0, a record every 10 iterations.
        _case("photo-tgv-420", "solve", 512, 768, "420", "tgv", 75, 300, record_every=10),
        # Sizes of partial blocks, 4:4:4, the channels apart, with records.
        _case("ragged-tgv-444-apart", "solve", 1001, 667, "444", "tgv", 90, 150, record_every=10, coupled=False),
        # A video frame's size to an 8-bit picture, TV, 4:2:2, partial blocks.
        _case("frame-tv-422-levels", "levels", 1083, 1919, "422", "tv", 60, 200),
        # A camera's 12-megapixel picture, TGV, 4:2:0 (the package's headline workload).
        _case("tgv-420-12mp", "solve", 3024, 4032, "420", "tgv", 75, 500),
        # A large greyscale scan, TGV, a custom table (the package's large workload at half its side).
        _case("scan-tgv-grey-4096", "solve", 4096, 4096, "grey", "tgv", 0, 100),
        # A service's batch: pictures of uneven sizes, grey and colour, TV and TGV.
        _case("batch-12", "batch", 1024, 1024, "mixed", "mixed", 0, 300, pictures=12),
        # A PNG file's picture, RGB of 8 bits, partial blocks of everything.
        _case("png-tgv-rgb", "samples", 901, 1203, "444", "tgv", 100, 200),
        # A learned model's reconstruction of a batch of patches, and a training step of it.
        _case("unrolled-16x512", "unrolled", 512, 512, "grey", "tgv", 30, 100, pictures=16),
        _case("train-16x512", "train", 512, 512, "grey", "tgv", 30, 100, pictures=16),
        # A training step on a few small pictures, ragged, checkpoints far apart.
        _case("train-3x200x264", "train", 195, 261, "grey", "tgv", 20, 40, pictures=3, checkpoint_every=20),
    ]


def draw(rng):
    def size(low, high):
        return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))

    kind = rng.choice(["solve", "solve", "solve", "levels", "batch", "samples", "unrolled", "train"])
    colour = rng.choice(["grey", "420", "420", "422", "444"])
    method = rng.choice(["tv", "tgv"])
    quality = rng.choice([0, rng.randint(10, 95)])
    if kind == "batch":
        side = size(256, 1024)
        return _case("", kind, side, side, "mixed", "mixed", 0, size(60, 300), pictures=rng.randint(3, 12))
    if kind in ("unrolled", "train"):
        pictures = rng.randint(1, 16)
        return _case("", kind, size(64, 512), size(64, 512), "grey", "tgv", rng.randint(10, 60), size(20, 100),
                     pictures=pictures, checkpoint_every=rng.choice([1, 7, 10, 20]))
    if kind == "samples":
        return _case("", kind, size(64, 1600), size(64, 1600), rng.choice(["grey", "444"]), method, 100, size(50, 200),
                     record_every=rng.choice([0, 10]), coupled=rng.random() < 0.75)
    return _case("", kind, size(64, 2400), size(64, 2400), colour, method, quality, size(60, 300),
                 record_every=rng.choice([0, 10]), coupled=rng.random() < 0.75)


# ---- Pictures and levels.


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _table(base, quality, rng):
    if quality == 0:
        return [rng.randint(1, 64) for _ in range(64)]
    scale = 5000 // quality if quality < 50 else 200 - 2 * quality
    return [min(max((b * scale + 50) // 100, 1), 255) for b in base]


def _picture(rows, columns, rng, device):
    y = torch.arange(rows, dtype=torch.float64, device=device)[:, None]
    x = torch.arange(columns, dtype=torch.float64, device=device)[None, :]
    out = rng.uniform(60, 190) + rng.uniform(-40, 40) * y / rows + rng.uniform(-40, 40) * x / columns
    for _ in range(12):
        y0, y1 = sorted(rng.randrange(rows) for _ in range(2))
        x0, x1 = sorted(rng.randrange(columns) for _ in range(2))
        y1, x1 = max(y1, y0 + 1), max(x1, x0 + 1)
        ramp = rng.uniform(-60, 60) / (y1 - y0) * (y[y0:y1] - y0) + rng.uniform(-60, 60) / (x1 - x0) * (x[:, x0:x1] - x0)
        out[y0:y1, x0:x1] = rng.uniform(20, 235) + ramp
    for _ in range(20):
        cy, cx, s = rng.uniform(0, rows), rng.uniform(0, columns), rng.uniform(5, 60)
        ya, yb = max(int(cy - 3 * s), 0), min(int(cy + 3 * s) + 1, rows)
        xa, xb = max(int(cx - 3 * s), 0), min(int(cx + 3 * s) + 1, columns)
        blob = torch.exp(-((y[ya:yb] - cy) ** 2 + (x[:, xa:xb] - cx) ** 2) / (2 * s * s))
        out[ya:yb, xa:xb] += rng.uniform(-60, 60) * blob
    noise = torch.Generator(device=device).manual_seed(rng.getrandbits(40))
    out = out + 2.0 * torch.randn(out.shape, dtype=torch.float64, device=device, generator=noise)
    return torch.round(torch.clamp(out, 0, 255))


def _dct(device):
    k = torch.arange(8, dtype=torch.float64, device=device)
    c = 0.5 * torch.cos(math.pi * (2 * k[None, :] + 1) * k[:, None] / 16)
    c[0] = math.sqrt(1 / 8)
    return c


def _padded(plane, rows, columns):
    down = torch.clamp(torch.arange(rows, device=plane.device), max=plane.shape[0] - 1)
    across = torch.clamp(torch.arange(columns, device=plane.device), max=plane.shape[1] - 1)
    return plane[down][:, across]


def _blocks(plane):
    """(..., 8 a, 8 b) as (..., a, b, 8, 8)."""
    *lead, rows, columns = plane.shape
    return plane.reshape(*lead, rows // 8, 8, columns // 8, 8).transpose(-3, -2)


def _canvas(blocks):
    *lead, a, b, _, _ = blocks.shape
    return blocks.transpose(-3, -2).reshape(*lead, 8 * a, 8 * b)


def _pooled(plane, cells):
    return torch.nn.functional.avg_pool2d(plane[None, None], cells)[0, 0] if cells != (1, 1) else plane


def _levels(plane, table, rows, columns):
    blocks = _blocks(_padded(plane, 8 * rows, 8 * columns) - 128.0)
    c = _dct(plane.device)
    steps = torch.tensor(table, dtype=torch.float64, device=plane.device).reshape(8, 8)
    return torch.round((c @ blocks @ c.T) / steps)


def _file(case, seed):
    """A picture's channels (C, rows, columns), and per component its levels (a, b, 8, 8), table, cells."""
    rng = random.Random(seed)
    device = _device()
    rows, columns, colour = case["rows"], case["columns"], case["colour"]
    if colour == "grey":
        samples = _picture(rows, columns, rng, device)[None]
        planes, parts = samples, [(LUMA, (1, 1))]
    else:
        samples = torch.stack([_picture(rows, columns, rng, device) for _ in range(3)])
        r, g, b = samples
        y = 0.299 * r + 0.587 * g + 0.114 * b
        planes = torch.round(torch.clamp(torch.stack([y, 128 + (b - y) / 1.772, 128 + (r - y) / 1.402]), 0, 255))
        parts = [(LUMA, (1, 1)), (CHROMA, CELLS[colour]), (CHROMA, CELLS[colour])]
    components = []
    tables = {id(base): _table(base, case["quality"], rng) for base in (LUMA, CHROMA)}
    for plane, (base, cells) in zip(planes, parts):
        a, b = -(-rows // (8 * cells[0])), -(-columns // (8 * cells[1]))
        whole = _padded(plane, 8 * a * cells[0], 8 * b * cells[1])
        components.append((_levels(torch.round(_pooled(whole, cells)), tables[id(base)], a, b), tables[id(base)], cells))
    return samples, components


def _image(case, components):
    grey = len(components) == 1
    most = CELLS[case["colour"]]
    parts = [(levels.to(torch.int16).cpu().numpy(), table, *((1, 1) if grey or c > 0 else (most[1], most[0])))
             for c, (levels, table, _) in enumerate(components)]
    space = jpegio.ColorSpace.GRAYSCALE if grey else jpegio.ColorSpace.YCBCR
    return jpegio.image_of(case["rows"], case["columns"], space, parts)


def _options(case):
    options = ["--method", case["method"], "--iterations", str(case["iterations"]), "--tolerance", "0",
               "--record-every", str(case["record_every"])]
    return options + ([] if case["coupled"] else ["--channels", "apart"])


def _parts(case, seed):
    """A batch's pictures as cases of their own (sizes and settings the case's, contents the
    seed's); an unrolled problem's pictures."""
    contents = random.Random(seed)
    parts = [case] * case["pictures"]
    if case["kind"] == "batch":
        side, rng = case["rows"], random.Random(f"{case['rows']} {case['pictures']}")
        parts = [_case("", "solve", rng.randint(side // 4, side), rng.randint(side // 4, side),
                       rng.choice(["grey", "420"]), rng.choice(["tv", "tgv"]), rng.randint(10, 90), case["iterations"])
                 for _ in range(case["pictures"])]
    return [(part, contents.getrandbits(30)) for part in parts]


# ---- The calls.


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        parts = _parts(case, seed)
        return {"kind": kind, "images": [_image(p, _file(p, s)[1]) for p, s in parts],
                "options": [_options(p) for p, _ in parts]}
    if kind == "samples":
        samples, _ = _file(case, seed)
        levels = samples.permute(1, 2, 0).to(torch.uint8).cpu().numpy()
        return {"kind": kind, "levels": levels[:, :, 0] if case["colour"] == "grey" else levels, "options": _options(case)}
    if kind in ("unrolled", "train"):
        files = [_file(p, s) for p, s in _parts(case, seed)]
        problem = unrolled.UnrolledProblem([_image(case, c) for _, c in files], ["--method", "tgv"],
                                           iterations=case["iterations"], checkpoint_every=case["checkpoint_every"])
        values = (2.0, 1.0, problem.tau, problem.sigma)
        leaves = [torch.full((case["pictures"],), v, dtype=torch.float32, device=problem.device,
                             requires_grad=kind == "train") for v in values]
        clean = torch.stack([s[0] for s, _ in files]).to(device=problem.device, dtype=torch.float32)
        return {"kind": kind, "problem": problem, "leaves": leaves, "clean": clean}
    return {"kind": kind, "image": _image(case, _file(case, seed)[1]), "options": _options(case)}


def _result(decoded):
    return {**_picture_of(decoded), "canvas": decoded.canvas, "coefficients": list(decoded.coefficients)}


def _picture_of(decoded):
    history = decoded.result.history
    return {"picture": decoded.picture, "primal": history.primal, "dual": history.dual}


def run(state):
    kind = state["kind"]
    if kind == "solve":
        return _result(native.solve(state["image"], state["options"]))
    if kind == "levels":
        return native.solve_levels(state["image"], state["options"])
    if kind == "batch":
        return [_picture_of(d) for d in native.solve_batch(state["images"], state["options"])[0]]
    if kind == "samples":
        return _picture_of(native.solve_samples(state["levels"], 8, state["options"]))
    if kind == "unrolled":
        with torch.no_grad():
            return unrolled.unrolled_tgv(state["problem"], *state["leaves"])
    x = unrolled.unrolled_tgv(state["problem"], *state["leaves"])
    clean = state["clean"]
    loss = torch.mean((x[:, : clean.shape[1], : clean.shape[2]] - clean) ** 2)
    return {"x": x.detach(), "loss": loss.detach(), "grads": list(torch.autograd.grad(loss, state["leaves"]))}


def work(case):
    """The levels in, the results out, and an iteration's arithmetic; the state's fields (TGV 8, TV 3
    a sample, 4 bytes each) read and written by every iteration where they exceed the L2, since
    they cannot stay there. A training step makes the forward's iterations and their adjoints."""
    if case["kind"] == "batch":
        side = case["rows"]
        samples, method = case["pictures"] * (0.625 * side) ** 2 * 2, "tgv"
        tgv = 0.5
    else:
        method = case["method"]
        samples = case["pictures"] * case["rows"] * case["columns"] * (1 if case["colour"] == "grey" else 3)
        tgv = 1.0 if method == "tgv" else 0.0
    fields = 3 + 5 * tgv
    kind, n = case["kind"], case["iterations"]
    ends = {"solve": 2 + 24, "batch": 2 + 24, "levels": 2 + 1, "samples": 1 + 8, "unrolled": 12 + 4, "train": 12 + 4}[kind]
    once = samples * ends
    state = samples * fields * 4
    moved = once + (n * 2 * state if state > L2_BYTES else 0)
    flops = samples * n * (55 + 25 + 60 * tgv)
    if kind == "train":
        moved += n * 3 * state if state > L2_BYTES else 0
        flops *= 3
    return {"bytes": moved, "flops": flops}


# ---- The same results in 64 bits, by plain torch.


def _dx(f):
    return torch.nn.functional.pad(f[..., 1:] - f[..., :-1], (0, 1))


def _dy(f):
    return torch.nn.functional.pad(f[..., 1:, :] - f[..., :-1, :], (0, 0, 0, 1))


def _bx(f):
    kept = torch.nn.functional.pad(f[..., :-1], (0, 1))
    return kept - torch.nn.functional.pad(f[..., :-1], (1, 0))


def _by(f):
    kept = torch.nn.functional.pad(f[..., :-1, :], (0, 0, 0, 1))
    return kept - torch.nn.functional.pad(f[..., :-1, :], (0, 0, 1, 0))


def _ball(square, radius):
    inside = square <= radius * radius
    return torch.where(inside, torch.ones_like(square), radius / torch.sqrt(torch.where(inside, torch.ones_like(square), square)))


def _total(square, coupled):
    return square.sum(0, keepdim=True) if coupled else square


def _dual(s, xt, tau, sigma, alpha1, alpha0, coupled, rho):
    """The dual step from s = (x, p1, p2 [, w1, w2, r11, r22, r12]) and x~: the relaxed state and the tilde point."""
    x, p1, p2, *rest = s
    bar = 2 * xt - x
    g1, g2 = _dx(bar), _dy(bar)
    tilde = [xt]
    if rest:
        w1, w2, r11, r22, r12 = rest
        t1 = w1 + tau * (p1 + _dx(r11) + _dy(r12))
        t2 = w2 + tau * (p2 + _dx(r12) + _dy(r22))
        b1, b2 = 2 * t1 - w1, 2 * t2 - w2
        q11, q22, q12 = r11 + sigma * _bx(b1), r22 + sigma * _by(b2), r12 + sigma * 0.5 * (_by(b1) + _bx(b2))
        k = _ball(_total(q11 * q11 + q22 * q22 + 2 * q12 * q12, coupled), alpha0)
        g1, g2 = g1 - b1, g2 - b2
    q1, q2 = p1 + sigma * g1, p2 + sigma * g2
    scale = _ball(_total(q1 * q1 + q2 * q2, coupled), alpha1)
    tilde += [q1 * scale, q2 * scale] + ([t1, t2, q11 * k, q22 * k, q12 * k] if rest else [])
    return [rho * a + (1 - rho) * b for a, b in zip(tilde, s)], tilde


class _Component:
    """A component's intervals, centres and weights (DC absolute), and its proximal map."""

    def __init__(self, levels, table, cells, chroma):
        self.cells = cells
        self.rows, self.columns = 8 * levels.shape[0] * cells[0], 8 * levels.shape[1] * cells[1]
        steps = torch.tensor(table, dtype=torch.float64, device=levels.device).reshape(8, 8)
        mu = 9.0 * (0.3 if chroma else 1.0) * (sum(table) / 64) ** 0.9
        shift = torch.zeros_like(steps)
        shift[0, 0] = 1024.0
        self.lower, self.upper = (levels - 0.5) * steps + shift, (levels + 0.5) * steps + shift
        self.centre = levels * steps + shift
        dc = levels[..., 0, 0]
        flat = (levels != 0).flatten(2).sum(-1) - (dc != 0).long() == 0
        for d in (0, 1):
            near = (dc.diff(dim=d).abs() <= 1).to(torch.uint8)
            edge = torch.ones_like(near.narrow(d, 0, 1)) if near.shape[d] else None
            if edge is not None:
                flat &= torch.cat([near, edge], d).bool() & torch.cat([edge, near], d).bool()
        self.weight = mu / steps**2 * torch.where(flat, 0.1, 1.0)[..., None, None]
        self.c = _dct(levels.device)

    def spread(self, small):
        return small.repeat_interleave(self.cells[0], 0).repeat_interleave(self.cells[1], 1)

    def to_canvas(self, zeta):
        return self.spread(_canvas(self.c.T @ zeta @ self.c))

    def prox(self, v, tau):
        own = v[: self.rows, : self.columns]
        mean = _pooled(own, self.cells)
        t = tau / (self.cells[0] * self.cells[1]) * self.weight
        e = self.c @ _blocks(mean) @ self.c.T
        zeta = torch.clamp((e + t * self.centre) / (1 + t), self.lower, self.upper)
        out = v.clone()
        out[: self.rows, : self.columns] = own + self.spread(_canvas(self.c.T @ zeta @ self.c) - mean)
        return out, zeta

    def value(self, zeta):
        return 0.5 * (self.weight * (zeta - self.centre) ** 2).sum()

    def conjugate(self, xi):
        own = xi[: self.rows, : self.columns]
        mean = _pooled(own, self.cells)
        total = 255.0 * (own - self.spread(mean)).abs().sum() if self.cells != (1, 1) else 0.0
        for beyond in (xi[self.rows :], xi[: self.rows, self.columns :]):
            total = total + 128.0 * beyond.sum() + 255.0 * beyond.abs().sum()
        s = self.c @ _blocks(mean * (self.cells[0] * self.cells[1])) @ self.c.T
        best = torch.clamp(self.centre + s / self.weight, self.lower, self.upper)
        return total + (s * best - 0.5 * self.weight * (best - self.centre) ** 2).sum()


def _steps(tgv, ratio):
    norm = (17 + math.sqrt(33)) / 2 if tgv else 8.0
    return math.sqrt(ratio * 0.99 / norm), math.sqrt(0.99 / (ratio * norm))


def _start(x, tgv):
    zero = torch.zeros_like(x)
    return [x, zero, zero] + ([_dx(x), _dy(x), zero, zero, zero] if tgv else [])


def _iterate(case, x, prox, value, conjugate, ratio):
    """The solve from the picture x: the last x~, what prox kept with it, the records."""
    tgv, coupled = case["method"] == "tgv", case["coupled"] and x.shape[0] > 1
    tau, sigma = _steps(tgv, ratio)
    s = _start(x, tgv)
    tilde, kept = s, None
    primal, dual = [], []

    def record():
        grads = _dx(tilde[0]), _dy(tilde[0])
        if tgv:
            grads = [g - w for g, w in zip(grads, tilde[3:5])]
        first = _total(sum(g * g for g in grads), coupled).sqrt().sum()
        if not tgv:
            primal.append(float(first + value(kept)))
            dual.append(-float(conjugate(_bx(tilde[1]) + _by(tilde[2]))))
            return
        w1, w2, r11, r22, r12 = tilde[3:]
        second = _total(_bx(w1) ** 2 + _by(w2) ** 2 + 0.5 * (_by(w1) + _bx(w2)) ** 2, coupled).sqrt().sum()
        d1, d2 = _dx(r11) + _dy(r12), _dx(r12) + _dy(r22)
        theta = min(1.0, 1.0 / max(float(_total(d1 * d1 + d2 * d2, coupled).max().sqrt()), 1e-300))
        primal.append(float(first + 2.0 * second + value(kept)))
        dual.append(-float(conjugate(-theta * (_bx(d1) + _by(d2)))))

    every, last = case["record_every"], case["iterations"]
    if every > 0:
        record()
    for k in range(1, last + 1):
        xt, kept = prox(s[0] + tau * (_bx(s[1]) + _by(s[2])), tau)
        s, tilde = _dual(s, xt, tau, sigma, 1.0, 2.0, coupled, 1.9)
        if (every > 0 and k % every == 0) or k == last:
            record()
    return tilde[0], kept, np.array(primal), np.array(dual)


def _exact_file(case, seed):
    _, components = _file(case, seed)
    grey = len(components) == 1
    parts = [_Component(*c, chroma=n > 0) for n, c in enumerate(components)]
    rows, columns = max(p.rows for p in parts), max(p.columns for p in parts)
    x = torch.full((len(parts), rows, columns), 128.0, dtype=torch.float64, device=_device())
    for plane, p in zip(x, parts):
        plane[: p.rows, : p.columns] = p.to_canvas(p.centre)

    def prox(v, tau):
        made = [p.prox(plane, tau) for p, plane in zip(parts, v)]
        return torch.stack([m[0] for m in made]), [m[1] for m in made]

    def value(kept):
        return sum(p.value(z) for p, z in zip(parts, kept)) if kept is not None else 0.0

    def conjugate(xi):
        return sum(p.conjugate(plane) for p, plane in zip(parts, xi))

    canvas, zeta, primal, dual = _iterate(case, x, prox, value, conjugate, 3.0 if case["method"] == "tgv" else 10.0)
    own = canvas[:, : case["rows"], : case["columns"]]
    if grey:
        picture = own[0]
    else:
        y, cb, cr = own[0], own[1] - 128, own[2] - 128
        picture = torch.stack([y + 1.402 * cr, y - 0.114 * 1.772 / 0.587 * cb - 0.299 * 1.402 / 0.587 * cr,
                               y + 1.772 * cb], -1)
    return {"picture": picture.cpu().numpy(), "canvas": canvas.cpu().numpy(),
            "coefficients": [z.cpu().numpy() for z in zeta], "primal": primal, "dual": dual}


def _exact_samples(case, seed):
    samples, _ = _file(case, seed)
    lower, upper = torch.clamp(samples - 0.5, min=0), torch.clamp(samples + 0.5, max=255)

    def conjugate(xi):
        return torch.maximum(xi * lower, xi * upper).sum()

    picture, _, primal, dual = _iterate(case, samples, lambda v, tau: (torch.clamp(v, lower, upper), None),
                                        lambda kept: 0.0, conjugate, 0.3 if case["method"] == "tgv" else 10.0)
    picture = picture[0] if case["colour"] == "grey" else picture.permute(1, 2, 0)
    return {"picture": picture.cpu().numpy(), "primal": primal, "dual": dual}


def _exact_unrolled(case, seed):
    files = [_file(p, s) for p, s in _parts(case, seed)]
    parts = [_Component(*c[0], chroma=False) for _, c in files]
    c = parts[0].c
    lower, upper, centre, weight = (torch.stack([getattr(p, a) for p in parts]) for a in
                                    ("lower", "upper", "centre", "weight"))
    train = case["kind"] == "train"
    count = case["pictures"]
    # The parameters as the call has them, in 32 bits.
    leaves = [torch.full((count,), float(np.float32(v)), dtype=torch.float64, device=c.device, requires_grad=train)
              for v in (2.0, 1.0, *_steps(True, 3.0))]
    alpha0, alpha1, tau, sigma = (v[:, None, None] for v in leaves)

    def prox(s):
        t = tau[..., None, None] * weight
        e = c @ _blocks(s[0] + tau * (_bx(s[1]) + _by(s[2]))) @ c.T
        return _canvas(c.T @ torch.clamp((e + t * centre) / (1 + t), lower, upper) @ c)

    def several(n, *s):
        for _ in range(n):
            s = _dual(s, prox(s), tau, sigma, alpha1, alpha0, False, 1.9)[0]
        return tuple(s)

    with torch.set_grad_enabled(train):
        s = tuple(_start(_canvas(c.T @ centre @ c), True))
        left = case["iterations"] - 1
        while left > 0:
            n = min(5, left)
            s = torch.utils.checkpoint.checkpoint(several, n, *s, use_reentrant=False) if train else several(n, *s)
            left -= n
        x = prox(s)
        if not train:
            return x
        clean = torch.stack([samples[0] for samples, _ in files])
        loss = torch.mean((x[:, : clean.shape[1], : clean.shape[2]] - clean) ** 2)
        grads = torch.autograd.grad(loss, leaves)
    return {"x": x.detach(), "loss": loss.detach(), "grads": list(grads)}


def exact(case, seed):
    kind = case["kind"]
    if kind == "levels":
        return None  # whole numbers
    if kind == "batch":
        made = [_exact_file(p, s) for p, s in _parts(case, seed)]
        return [{name: e[name] for name in ("picture", "primal", "dual")} for e in made]
    if kind == "samples":
        return _exact_samples(case, seed)
    if kind in ("unrolled", "train"):
        return _exact_unrolled(case, seed)
    return _exact_file(case, seed)
