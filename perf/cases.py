"""Performance cases of the gradient-domain Poisson framework.

Each case is one call (or the few calls) that a program built on this package
makes through its public entry points, with inputs of the kind that call meets:
cloning a small patch, a served one-megapixel integration, the three-channel
tone-mapping integration, a rectangle with fixed borders, a masked composite, an
uneven batch, an all-FP64 solve, the exact DCT solve on power-of-two and on
video-sized grids, a whole tone mapping, the red-black smoother and the
reference-exact multigrid.

``listed()`` are the fixed cases, ``draw(rng)`` gives others of the same ranges,
``prepare`` / ``run`` are what a program has in hand and what it then calls,
``work`` is the least data and arithmetic of a pass, ``tolerance`` how far
another correct implementation may be, and ``exact`` the same answer in plain
64-bit torch without this package's code.
"""

from __future__ import annotations

import math

import numpy as np
import torch

import gradient_domain_b200 as gd
from gradient_domain_b200.hdr import tone_map_device
from gradient_domain_b200.solvers import DctPlan

F64 = torch.float64


def listed():
    return [
        # pasting a small patch into a photograph: a call of a few milliseconds made of
        # launches and small copies (seamless_clone from and to NumPy arrays)
        {"name": "clone_patch", "path": "clone", "height": 240, "width": 320, "patch_height": 96,
         "patch_width": 130, "mode": "mixed", "domain": "mask"},
        # one served megapixel: a single Neumann integration on a resident plan
        {"name": "neumann_1mp", "path": "solve", "boundary": "neumann", "height": 1024,
         "width": 1024, "channels": 1, "precision": "mixed", "sweeps": 0, "tolerance": 1e-8},
        # the headline: tone-mapping-style integration of three 16 MP channels, with the
        # three sweeps that the autotuner chooses for it
        {"name": "tonemap_16mp_x3", "path": "solve", "boundary": "neumann", "height": 4096,
         "width": 4096, "channels": 3, "precision": "mixed", "sweeps": 3, "tolerance": 1e-8},
        # rectangle with a fixed ring (solve_dirichlet's system), odd sides
        {"name": "dirichlet_odd", "path": "solve", "boundary": "dirichlet", "height": 1022,
         "width": 1533, "channels": 3, "precision": "mixed", "sweeps": 0, "tolerance": 1e-8},
        # compositing inside a star-shaped selection, to the direct-solver level that
        # seamless_clone asks for; every composite brings its own mask
        {"name": "composite_2048", "path": "solve", "boundary": "masked", "height": 1411,
         "width": 1387, "channels": 3, "precision": "mixed", "sweeps": 0, "tolerance": 1e-12},
        # an uneven batch of integrations, composites and rectangles in one plan
        {"name": "batch_ragged", "path": "batch", "count": 16, "low": 64, "high": 1024,
         "layout": 5},
        # all-FP64 solve to the level that replaces a factorisation (methods "direct", "mgcg_fp64")
        {"name": "direct_fp64", "path": "solve", "boundary": "dirichlet", "height": 1000,
         "width": 1500, "channels": 1, "precision": "fp64", "sweeps": 0, "tolerance": 1e-13},
        # exact Neumann solve by the cosine transform, three 16 MP channels
        {"name": "dct_16mp_x3", "path": "dct", "height": 4096, "width": 4096, "channels": 3},
        # the same on a video frame, sides with factors 3 and 5
        {"name": "dct_video", "path": "dct", "height": 1080, "width": 1920, "channels": 3},
        # HDR tone mapping of one photograph on the device, as the server runs it
        {"name": "tone_map_photo", "path": "tone_map", "height": 1440, "width": 2160,
         "levels": 8},
        # stand-alone red-black smoother, two sweeps on 16 MP
        {"name": "smooth_fp32", "path": "smooth", "height": 4096, "width": 4096,
         "dtype": "float32", "sweeps": 2},
        # the reference's own multigrid, cycle for cycle, from and to NumPy arrays
        {"name": "multigrid_reference", "path": "multigrid", "height": 1023, "width": 1023,
         "tolerance": 1e-8},
    ]


def _log_size(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    path = rng.choice(["clone", "solve", "solve", "solve", "solve", "batch", "dct", "dct",
                       "tone_map", "smooth", "smooth", "multigrid"])
    if path == "clone":
        h, w = _log_size(rng, 120, 1024), _log_size(rng, 120, 1024)
        return {"path": path, "height": h, "width": w, "patch_height": rng.randint(40, h - 4),
                "patch_width": rng.randint(40, w - 4),
                "mode": rng.choice(["import", "mixed", "average"]),
                "domain": rng.choice(["mask", "mask", "rectangle"])}
    if path == "solve":
        boundary = rng.choice(["neumann", "dirichlet", "masked"])
        precision = rng.choice(["mixed", "mixed", "fp64"])
        top = 1600 if boundary == "masked" else 3000
        h, w = _log_size(rng, 64, top), _log_size(rng, 64, top)
        tolerance = {"masked": rng.choice([1e-8, 1e-12]), "dirichlet": 1e-8,
                     "neumann": 1e-8}[boundary]
        if precision == "fp64":
            tolerance = rng.choice([1e-8, 1e-12])
        return {"path": path, "boundary": boundary, "height": h, "width": w,
                "channels": rng.choice([1, 3]), "precision": precision,
                "sweeps": rng.choice([0, 0, 1, 2, 3]), "tolerance": tolerance}
    if path == "batch":
        return {"path": path, "count": rng.randint(3, 16), "low": 64,
                "high": _log_size(rng, 200, 1024), "layout": rng.randint(0, 10 ** 6)}
    if path == "dct":
        if rng.random() < 0.4:
            h, w = 2 ** rng.randint(6, 12), 2 ** rng.randint(6, 12)
        else:
            h, w = _log_size(rng, 50, 2500), _log_size(rng, 50, 2500)
        return {"path": path, "height": h, "width": w, "channels": rng.choice([1, 3])}
    if path == "tone_map":
        return {"path": path, "height": _log_size(rng, 100, 2000),
                "width": _log_size(rng, 100, 3000), "levels": rng.choice([1, 4, 8])}
    if path == "smooth":
        return {"path": path, "height": _log_size(rng, 60, 4096),
                "width": _log_size(rng, 60, 4096), "dtype": rng.choice(["float32", "float64"]),
                "sweeps": rng.randint(1, 6)}
    return {"path": path, "height": _log_size(rng, 40, 1100), "width": _log_size(rng, 40, 1100),
            "tolerance": 1e-8}


# ---------------------------------------------------------------------------
# inputs


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) & 0x7fffffffffff)
    return g


def _uniform(g, shape, low=0.0, high=1.0):
    return low + (high - low) * torch.rand(shape, generator=g, dtype=F64, device="cuda")


def _blobs(g, h, w, count=32, noise=0.05):
    """Sum of Gaussian blobs plus uniform noise: the stand-in for an image channel."""
    m = min(h, w)
    cy, cx = _uniform(g, (1, count), 0, h), _uniform(g, (1, count), 0, w)
    s = _uniform(g, (1, count), 0.01 * m + 1.0, 0.12 * m + 1.0)
    a = _uniform(g, (1, count))
    y = torch.arange(h, dtype=F64, device="cuda")[:, None]
    x = torch.arange(w, dtype=F64, device="cuda")[:, None]
    img = (torch.exp(-(y - cy) ** 2 / (2 * s * s)) * a) @ torch.exp(-(x - cx) ** 2 / (2 * s * s)).T
    return img + noise * torch.rand((h, w), generator=g, dtype=F64, device="cuda")


def _forward(u):
    gx, gy = torch.zeros_like(u), torch.zeros_like(u)
    gx[..., :, :-1] = u[..., :, 1:] - u[..., :, :-1]
    gy[..., :-1, :] = u[..., 1:, :] - u[..., :-1, :]
    return gx, gy


def _backward(gx, gy):
    out = torch.zeros_like(gx)
    out[..., :, :-1] += gx[..., :, :-1]
    out[..., :, 1:] -= gx[..., :, :-1]
    out[..., :-1, :] += gy[..., :-1, :]
    out[..., 1:, :] -= gy[..., :-1, :]
    return out


def _tonemap_rhs(g, h, w):
    """Divergence of an attenuated log-radiance gradient field (one pyramid level)."""
    log_r = 2.5 * torch.randn((h, w), generator=g, dtype=F64, device="cuda")
    log_r += torch.log(0.05 + _blobs(g, h, w, 64, 0.0))
    gx, gy = _forward(log_r)
    m = torch.sqrt(gx * gx + gy * gy)
    scale = 0.1 * m.mean()
    m = m.clamp_min(1e-4)
    f = (scale / m) * (m / scale) ** 0.85
    return _backward(gx * f, gy * f)


def _star(g, h, w):
    """A star-shaped selection around the centre that leaves the border free."""
    y = torch.arange(h, dtype=F64, device="cuda")[:, None] + 0.5 - h / 2
    x = torch.arange(w, dtype=F64, device="cuda")[None, :] + 0.5 - w / 2
    t = torch.atan2(y / h, x / w)
    r = torch.full_like(t, 0.34)
    for k in (2, 5, 9):
        p = _uniform(g, (2,))
        r = r + 0.04 * p[0] * torch.cos(k * t + 2 * math.pi * p[1])
    inside = torch.sqrt((y / h) ** 2 + (x / w) ** 2) < r
    inside[0, :] = inside[-1, :] = False
    inside[:, 0] = inside[:, -1] = False
    return inside


def _neighbours(u):
    out = torch.zeros_like(u)
    out[..., 1:, :] += u[..., :-1, :]
    out[..., :-1, :] += u[..., 1:, :]
    out[..., :, 1:] += u[..., :, :-1]
    out[..., :, :-1] += u[..., :, 1:]
    return out


def _masked_rhs(source, target, inside):
    """Right-hand side of importing source's gradients into target: A x = f, A positive."""
    sx, sy = _forward(source)
    tx, ty = _forward(target)
    div = _backward(torch.where(inside, sx, tx), torch.where(inside, sy, ty))
    known = _neighbours(torch.where(inside, torch.zeros_like(target), target))
    return torch.where(inside, known - div, torch.zeros_like(div))


def _system(g, boundary, h, w, like_tonemap=False):
    """(right-hand side, mask or None, scale) of one channel; the plan solves A x = scale f."""
    if boundary == "masked":
        inside = _star(g, h, w)
        return _masked_rhs(_blobs(g, h, w), _blobs(g, h, w), inside), inside, 1.0
    if like_tonemap:
        return _tonemap_rhs(g, h, w), None, -1.0
    img = _blobs(g, h, w)
    if boundary == "neumann":
        return _backward(*_forward(img)), None, -1.0
    return _neighbours(img) - 4.0 * img, None, -1.0


def _solve_inputs(case, seed):
    g = _generator(seed)
    h, w, c = case["height"], case["width"], case["channels"]
    if case["boundary"] == "masked":
        inside = _star(g, h, w)
        f = [_masked_rhs(_blobs(g, h, w), _blobs(g, h, w), inside) for _ in range(c)]
        return f, [inside] * c, [1.0] * c
    tone = case["boundary"] == "neumann" and c == 3
    got = [_system(g, case["boundary"], h, w, tone) for _ in range(c)]
    return [t[0] for t in got], [None] * c, [t[2] for t in got]


def _batch_layout(case):
    """Boundary and shape of every instance, from the case alone (a plan is kept by them)."""
    r = np.random.default_rng(case["layout"])
    out = []
    for k in range(case["count"]):
        s = math.exp(r.uniform(math.log(case["low"]), math.log(case["high"])))
        aspect = r.uniform(0.5, 2.0)
        h = max(16, int(round(s * math.sqrt(aspect))))
        w = max(16, int(round(s / math.sqrt(aspect))))
        boundary = ("neumann", "masked", "dirichlet")[k % 3]
        out += [(boundary, h, w)] * (1 if r.random() < 0.5 else 3)
    return out


def _batch_inputs(case, seed):
    g = _generator(seed)
    return [_system(g, b, h, w) for b, h, w in _batch_layout(case)]


def _clone_inputs(case, seed):
    g = _generator(seed)
    h, w, ph, pw = (case[k] for k in ("height", "width", "patch_height", "patch_width"))

    def image(hh, ww):
        img = torch.stack([_blobs(g, hh, ww) for _ in range(3)], dim=2)
        img = img - img.min()
        return (img / img.max()).cpu().numpy()

    source, target = image(ph, pw), image(h, w)
    return source, target, _star(g, ph, pw).cpu().numpy(), ((h - ph) // 2, (w - pw) // 2)


def _radiance(case, seed):
    """A log-normal radiance with blob-shaped light, as an HDR photograph has."""
    g = _generator(seed)
    h, w = case["height"], case["width"]
    light = 0.05 + _blobs(g, h, w, 64, 0.0)
    noise = torch.randn((h, w, 3), generator=g, dtype=F64, device="cuda")
    return torch.exp(0.6 * noise) * (light ** 3)[:, :, None]


def _smooth_inputs(case, seed):
    g = _generator(seed)
    shape, dtype = (case["height"], case["width"]), getattr(torch, case["dtype"])
    return (torch.randn(shape, generator=g, dtype=F64, device="cuda").to(dtype),
            torch.randn(shape, generator=g, dtype=F64, device="cuda").to(dtype))


def _multigrid_inputs(case, seed):
    return _system(_generator(seed), "dirichlet", case["height"], case["width"])[0]


def prepare(case, seed):
    path = case["path"]
    if path == "solve":
        f, masks, scale = _solve_inputs(case, seed)
        zero_mean = case["boundary"] == "neumann"
        plan = gd.cached_plan(
            tuple(gd.Instance(*t.shape, case["boundary"], zero_mean) for t in f),
            gd.SolveParams(precision=case["precision"], sweeps=case["sweeps"] or None,
                           tolerance=case["tolerance"], zero_start=True))
        return {"case": case, "plan": plan, "f": f, "x": [torch.empty_like(t) for t in f],
                "scale": scale,
                "masks": [None if m is None else m.to(torch.uint8) for m in masks]}
    if path == "batch":
        got = _batch_inputs(case, seed)
        plan = gd.cached_plan(tuple(gd.Instance(h, w, b, b == "neumann")
                                    for b, h, w in _batch_layout(case)),
                              gd.SolveParams(tolerance=1e-8, zero_start=True))
        return {"case": case, "plan": plan, "f": [t[0] for t in got],
                "x": [torch.empty_like(t[0]) for t in got], "scale": [t[2] for t in got],
                "masks": [None if t[1] is None else t[1].to(torch.uint8) for t in got]}
    if path == "dct":
        g = _generator(seed)
        h, w = case["height"], case["width"]
        b = torch.stack([_tonemap_rhs(g, h, w) for _ in range(case["channels"])])
        return {"case": case, "plan": DctPlan(h, w), "b": b, "u": torch.empty_like(b)}
    if path == "tone_map":
        return {"case": case, "radiance": _radiance(case, seed),
                "config": gd.ToneMapConfig(levels=case["levels"])}
    if path == "smooth":
        u, b = _smooth_inputs(case, seed)
        return {"case": case, "u": u, "b": b}
    if path == "multigrid":
        return {"case": case, "b": _multigrid_inputs(case, seed).cpu().numpy(),
                "options": gd.MultigridOptions(tolerance=case["tolerance"])}
    source, target, mask, offset = _clone_inputs(case, seed)
    return {"case": case, "source": source, "target": target, "mask": mask, "offset": offset}


def run(state):
    case = state["case"]
    path = case["path"]
    if path in ("solve", "batch"):
        for k, mask in enumerate(state["masks"]):
            if mask is not None:
                state["plan"].set_mask(k, mask)
        state["plan"].solve(state["f"], state["x"], state["scale"])
        return state["x"]
    if path == "dct":
        for b, u in zip(state["b"], state["u"]):
            state["plan"].solve(b, u)
        return state["u"]
    if path == "tone_map":
        return tone_map_device(state["radiance"], state["config"])
    if path == "smooth":
        return gd.smooth(state["u"], state["b"], sweeps=case["sweeps"])
    if path == "multigrid":
        u, report = gd.solve(state["b"], options=state["options"])
        return u, report.cycles
    return gd.seamless_clone(state["source"], state["target"], state["mask"], state["offset"],
                             mode=case["mode"], domain=case["domain"])[0]


# ---------------------------------------------------------------------------
# the least work of a pass


def _transform_flops(h, w):
    """Cosine or sine transform and back of an h x w grid: 2.5 n log2 n per line of n."""
    return 2 * h * w * 2.5 * (math.log2(h) + math.log2(w))


def work(case):
    path = case["path"]
    if path == "batch":
        cells = sum(h * w for _, h, w in _batch_layout(case))
        masked = sum(h * w for b, h, w in _batch_layout(case) if b == "masked")
        return {"bytes": 16 * cells + masked, "flops": 100 * cells}
    cells = case["height"] * case["width"]
    if path == "solve":
        masked = cells if case["boundary"] == "masked" else 0
        # one multigrid cycle's arithmetic, about 100 operations a cell
        return {"bytes": 16 * cells * case["channels"] + masked,
                "flops": 100 * cells * case["channels"]}
    if path == "dct":
        return {"bytes": 16 * cells * case["channels"],
                "flops": _transform_flops(case["height"], case["width"]) * case["channels"]}
    if path == "tone_map":
        # radiance in, image and factor out; the transform and some 60 element-wise operations
        return {"bytes": 56 * cells,
                "flops": _transform_flops(case["height"], case["width"]) + 60 * cells}
    if path == "smooth":
        return {"bytes": 3 * cells * (4 if case["dtype"] == "float32" else 8),
                "flops": 6 * cells * case["sweeps"]}
    if path == "multigrid":
        return {"bytes": 16 * cells, "flops": 100 * cells}
    patch = case["patch_height"] * case["patch_width"]
    return {"bytes": 48 * cells + 25 * patch, "flops": 300 * patch}


def tolerance(case):
    """About four times the distance from ``exact`` that was measured over listed and drawn cases."""
    path = case["path"]
    if path in ("solve", "batch"):
        # the solver stops on its residual: two answers differ by the error that is left then
        # (measured up to 1.4e-7 at 1e-8, 1.4e-10 at 1e-12)
        return {"rel": 6e-7 if case.get("tolerance", 1e-8) > 1e-10 else 6e-10}
    if path == "dct":
        return {"rel": 4e-11}  # 9e-12: the eigenvalues of the smoothest modes cancel
    if path == "tone_map":
        return {"rel": 2e-11}  # 3e-12
    if path == "smooth":
        return {"rel": 3e-7 if case["dtype"] == "float32" else 2e-15}  # 5.5e-8, 2e-16
    if path == "multigrid":
        # the same cycles from the same start: rounding only, times the condition of a few cycles
        return {"rel": 1e-11}
    return {"rel": 1e-10 if case["domain"] == "mask" else 6e-7}


# ---------------------------------------------------------------------------
# the same answers in plain 64-bit torch


def _cosines(n):
    """Orthonormal cosine matrix (rows are modes) and the eigenvalues of -second difference."""
    k = torch.arange(n, dtype=F64, device="cuda")
    c = torch.cos(math.pi * k[:, None] * (2 * k[None, :] + 1) / (2 * n)) * math.sqrt(2 / n)
    c[0] /= math.sqrt(2.0)
    return c, 4 * torch.sin(math.pi * k / (2 * n)) ** 2


def _sines(n):
    k = torch.arange(1, n + 1, dtype=F64, device="cuda")
    s = torch.sin(math.pi * k[:, None] * k[None, :] / (n + 1)) * math.sqrt(2 / (n + 1))
    return s, 4 * torch.sin(math.pi * k / (2 * (n + 1))) ** 2


def _exact_neumann(f):
    """Zero-mean u with A u = f, A the positive Neumann operator."""
    (cy, ey), (cx, ex) = _cosines(f.shape[0]), _cosines(f.shape[1])
    t = cy @ f @ cx.T
    lam = ey[:, None] + ex[None, :]
    lam[0, 0] = 1.0
    t = t / lam
    t[0, 0] = 0.0
    return cy.T @ t @ cx


def _exact_dirichlet(f):
    (sy, ey), (sx, ex) = _sines(f.shape[0]), _sines(f.shape[1])
    return sy @ ((sy @ f @ sx) / (ey[:, None] + ex[None, :])) @ sx


def _exact_masked(f, inside):
    """Conjugate gradients on A u = f over the cells of ``inside`` (f (c, h, w))."""
    on = inside.to(F64)

    def apply(v):
        return on * (4.0 * v - _neighbours(v))

    x = torch.zeros_like(f)
    r = f * on
    p = r.clone()
    rr = (r * r).sum(dim=(1, 2))
    stop = 1e-28 * rr
    for it in range(1, 40001):
        q = apply(p)
        alpha = rr / (p * q).sum(dim=(1, 2)).clamp_min(1e-300)
        x += alpha[:, None, None] * p
        r -= alpha[:, None, None] * q
        new = (r * r).sum(dim=(1, 2))
        p = r + (new / rr.clamp_min(1e-300))[:, None, None] * p
        rr = new
        if it % 100 == 0 and bool((rr <= stop).all()):
            break
    return x


def _exact_system(boundary, f, inside, scale):
    if boundary == "neumann":
        return _exact_neumann(scale * f)
    if boundary == "dirichlet":
        return _exact_dirichlet(scale * f)
    return _exact_masked(f[None], inside)[0]


def _blur_half(a):
    """Binomial 1 4 6 4 1 blur with replicated edges, every other sample."""
    k = [1 / 16, 4 / 16, 6 / 16, 4 / 16, 1 / 16]
    for dim in (1, 0):
        n = a.shape[dim]
        i = torch.arange(n, device=a.device)
        a = sum(c * a.index_select(dim, (i + d).clamp(0, n - 1)) for c, d in zip(k, range(-2, 3)))
    return a[::2, ::2]


def _resize(a, h, w):
    """Bilinear resampling with the corners of both grids aligned."""
    for dim, n in ((0, h), (1, w)):
        m = a.shape[dim]
        t = torch.linspace(0, m - 1, n, dtype=F64, device=a.device)
        lo = t.floor().long()
        f = (t - lo).reshape((-1, 1) if dim == 0 else (1, -1))
        hi = (lo + 1).clamp_max(m - 1)
        a = a.index_select(dim, lo) * (1 - f) + a.index_select(dim, hi) * f
    return a


def _exact_tone_map(rad, config):
    lum = (rad * torch.tensor([0.2126, 0.7152, 0.0722], dtype=F64, device="cuda")).sum(dim=2)
    lum = lum.clamp_min(2.2250738585072014e-308)
    log_l = torch.log(lum)
    levels = [log_l]
    while len(levels) < config.levels and min(levels[-1].shape) > 16:
        levels.append(_blur_half(levels[-1]))
    factor = None
    for k in reversed(range(len(levels))):
        a = levels[k]
        p = torch.nn.functional.pad(a[None, None], (1, 1, 1, 1), mode="replicate")[0, 0]
        gx = (p[1:-1, 2:] - p[1:-1, :-2]) / (2.0 * 2.0 ** k)
        gy = (p[2:, 1:-1] - p[:-2, 1:-1]) / (2.0 * 2.0 ** k)
        m = torch.sqrt(gx * gx + gy * gy)
        scale = config.alpha * max(float(m.mean()), config.epsilon)
        m = m.clamp_min(config.epsilon)
        local = (scale / m) * (m / scale) ** config.beta
        factor = local if factor is None else _resize(factor, *a.shape) * local
    gx, gy = _forward(log_l)
    u = _exact_neumann(-_backward(gx * factor, gy * factor))
    image = (rad / lum[:, :, None]) ** config.saturation * torch.exp(u - u.max())[:, :, None]
    v = image.reshape(-1).sort().values
    at = 0.995 * (v.numel() - 1)
    lo = int(at)
    peak = v[lo] + (v[min(lo + 1, v.numel() - 1)] - v[lo]) * (at - lo)
    return (image / peak.clamp_min(1e-12)).clamp(0, 1), factor


def _exact_smooth(u, b, sweeps):
    u, b = u.to(F64).clone(), b.to(F64)
    i = torch.arange(u.shape[0], device="cuda")[:, None]
    j = torch.arange(u.shape[1], device="cuda")[None, :]
    for k in range(2 * sweeps):
        u = torch.where((i + j) % 2 == k % 2, 0.25 * (_neighbours(u) - b), u)
    return u


def _exact_clone(case, seed):
    source, target, mask, (row, col) = _clone_inputs(case, seed)
    h, w = target.shape[:2]
    canvas = np.zeros_like(target)
    canvas[row:row + source.shape[0], col:col + source.shape[1]] = source
    placed = np.zeros((h, w), dtype=bool)
    placed[row:row + source.shape[0], col:col + source.shape[1]] = mask
    t = torch.from_numpy(target).cuda().permute(2, 0, 1)
    s = torch.from_numpy(canvas).cuda().permute(2, 0, 1)
    m = torch.from_numpy(placed).cuda()
    (tx, ty), (sx, sy) = _forward(t), _forward(s)
    if case["mode"] == "mixed":
        sx, sy = torch.where(sx.abs() >= tx.abs(), sx, tx), torch.where(sy.abs() >= ty.abs(), sy, ty)
    elif case["mode"] == "average":
        sx, sy = 0.5 * (sx + tx), 0.5 * (sy + ty)
    div = _backward(torch.where(m, sx, tx), torch.where(m, sy, ty))
    unknown = torch.zeros_like(m)
    if case["domain"] == "mask":
        unknown[1:-1, 1:-1] = m[1:-1, 1:-1]
    else:  # the selection's bounding box plus the margin, without its ring
        ys, xs = torch.nonzero(m.any(dim=1))[:, 0], torch.nonzero(m.any(dim=0))[:, 0]
        top, bottom = max(int(ys[0]) - 24, 0), min(int(ys[-1]) + 25, h)
        left, right = max(int(xs[0]) - 24, 0), min(int(xs[-1]) + 25, w)
        unknown[top + 1:bottom - 1, left + 1:right - 1] = True
    known = _neighbours(torch.where(unknown, torch.zeros_like(t), t))
    x = _exact_masked(torch.where(unknown, known - div, torch.zeros_like(div)), unknown)
    return torch.where(unknown, x, t).permute(1, 2, 0).contiguous()


def exact(case, seed):
    path = case["path"]
    if path == "solve":
        f, masks, scale = _solve_inputs(case, seed)
        if case["boundary"] == "masked":
            return list(_exact_masked(torch.stack(f), masks[0]))
        return [_exact_system(case["boundary"], a, None, s) for a, s in zip(f, scale)]
    if path == "batch":
        return [_exact_system(b, f, inside, scale) for (b, _, _), (f, inside, scale)
                in zip(_batch_layout(case), _batch_inputs(case, seed))]
    if path == "dct":
        g = _generator(seed)
        return torch.stack([_exact_neumann(-_tonemap_rhs(g, case["height"], case["width"]))
                            for _ in range(case["channels"])])
    if path == "tone_map":
        return _exact_tone_map(_radiance(case, seed), gd.ToneMapConfig(levels=case["levels"]))
    if path == "smooth":
        return _exact_smooth(*_smooth_inputs(case, seed), case["sweeps"])
    if path == "multigrid":
        return _exact_dirichlet(-_multigrid_inputs(case, seed)), None
    return _exact_clone(case, seed)
