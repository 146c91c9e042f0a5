"""The work that users of this framework have it do, as cases that can be timed.

Kinds of case (``kind``), each through an entry point a user's program calls:

  op          ``ops.PoissonBlend`` / ``ops.ScreenedPoisson`` on host images: one plan node
  solve_host  ``Context.solve`` on host images
  solve       ``pt_poisson_solve`` on images in device memory (SOR or multigrid-CG)
  batch       ``pt_poisson_solve_batch`` on uneven images in device memory
  dataset     ``warmstart.solve_batch_device``: equal single-channel images, as the
              warm start's training data are solved
  train       ``UNet.features`` + ``UNet.grad_record``: one replica's part of a training step
  guess       ``warmstart.guess_image``: the network's warm start of one problem
  mask        ``masks.polygon`` / ``masks.ellipse`` into device memory

Images are sums of random sinusoids plus noise, masks ellipses or star
polygons, as in :mod:`paintop_b200.synth`; they are made on the GPU.
"""
import ctypes as C
import math
import os

import numpy as np
import torch

from paintop_b200 import _lib, masks, ops, warmstart

DEV = "cuda"
MULTIGRID, AUTO, DEVICE = _lib.PT_FLAG_MULTIGRID, _lib.PT_FLAG_OMEGA_AUTO, _lib.PT_FLAG_DEVICE_POINTERS


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # a small clone inside an edit: one plan node on a thumbnail, where latency counts
        dict(name="op_clone_97x71", kind="op", width=97, height=71, channels=3, lam=0.0),
        # a plan node on an ordinary photograph-sized layer of ragged extent
        dict(name="op_screened_1531x1023", kind="op", width=1531, height=1023, channels=4, lam=0.01),
        # the 512 x 512 seamless-clone configuration on host buffers
        dict(name="clone_512_host", kind="solve_host", width=512, height=512, channels=3, lam=0.0, omega=1.9, tol=1e-5),
        # the headline: a screened 2048 x 2048 RGBA solve, images resident on the GPU
        dict(name="screened_2048", kind="solve", method="sor", width=2048, height=2048, channels=4, lam=0.01,
             omega=1.8, tol=1e-6, shape="star"),
        # a service's queue of uneven jobs solved in one call
        dict(name="batch_uneven_48", kind="batch", method="sor", count=48, low=64, high=1024, tol=1e-6),
        # solving the warm start's training instances
        dict(name="dataset_128x256", kind="dataset", count=128, size=256, tol=1e-7),
        # a small ragged image by multigrid: many short launches
        dict(name="multigrid_237x181", kind="solve", method="multigrid", width=237, height=181, channels=3, lam=0.0,
             omega=1.8, tol=1e-6, shape="ellipse"),
        # eight regions of a 4096 x 4096 RGB image by multigrid, the largest solve
        dict(name="multigrid_4096", kind="solve", method="multigrid", width=4096, height=4096, channels=3, lam=0.0,
             omega=1.8, tol=1e-6, shape="regions"),
        # the uneven queue by multigrid
        dict(name="batch_uneven_48_multigrid", kind="batch", method="multigrid", count=48, low=64, high=1024, tol=1e-6),
        # one training step's gradient at the training configuration
        dict(name="train_64x256", kind="train", count=64, height=256, width=256),
        # the network's guess for a large image (inference)
        dict(name="guess_2000x1500", kind="guess", width=2000, height=1500, channels=3, scale=6),
        # rasterising a large star polygon where the solve will read it
        dict(name="polygon_4096", kind="mask", shape="polygon", width=4096, height=4096, vertices=12),
    ]


def _log(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["op", "solve_host", "solve", "solve", "solve", "batch", "dataset", "train", "guess", "mask"])
    if kind == "op":
        lam = rng.choice([0.0, 0.005, 0.01, 0.1])
        high = 120 if lam == 0.0 else 1400
        return dict(kind=kind, width=_log(rng, 33, high), height=_log(rng, 33, high), channels=rng.choice([1, 3, 4]),
                    lam=lam)
    if kind == "solve_host":
        return dict(kind=kind, width=_log(rng, 64, 700), height=_log(rng, 64, 700), channels=rng.choice([1, 3, 4]),
                    lam=0.0, omega=1.9, tol=1e-5)
    if kind == "solve":
        method = rng.choice(["sor", "sor", "multigrid"])
        lam = rng.choice([0.0, 0.01, 0.05])
        high = 900 if method == "sor" and lam == 0.0 else 2048 if method == "sor" else 4096
        return dict(kind=kind, method=method, width=_log(rng, 61, high), height=_log(rng, 61, high),
                    channels=rng.choice([1, 2, 3, 4]) if high < 4096 else rng.choice([1, 3]), lam=lam,
                    omega=0.0 if method == "sor" and lam == 0.0 else 1.8, tol=rng.choice([1e-5, 1e-6, 1e-7]),
                    shape=rng.choice(["ellipse", "star", "regions"]))
    if kind == "batch":
        return dict(kind=kind, method=rng.choice(["sor", "multigrid"]), count=rng.randint(2, 40),
                    low=64, high=rng.choice([256, 512, 800]), tol=1e-6)
    if kind == "dataset":
        return dict(kind=kind, count=_log(rng, 2, 128), size=rng.choice([96, 128, 200, 256]), tol=1e-7)
    if kind == "train":
        return dict(kind=kind, count=_log(rng, 1, 48), height=8 * rng.randint(6, 32), width=8 * rng.randint(6, 32))
    if kind == "guess":
        return dict(kind=kind, width=_log(rng, 150, 2000), height=_log(rng, 150, 1500), channels=rng.choice([1, 3, 4]),
                    scale=rng.randint(3, 8))
    return dict(kind=kind, shape=rng.choice(["polygon", "ellipse"]), width=_log(rng, 64, 4096),
                height=_log(rng, 64, 4096), vertices=_log(rng, 3, 400))


def _sizes(case):
    """The (width, height) of a batch's images: log-uniform sides, aspects in [0.5, 2]. The sizes
    are the case's and not a seed's, so that every seed's batch is the same amount of work."""
    r = np.random.default_rng(1000 * case["count"] + case["high"])
    out = []
    for _ in range(case["count"]):
        s = math.exp(r.uniform(math.log(case["low"]), math.log(case["high"])))
        a = r.uniform(0.5, 2.0)
        out.append((max(8, round(s * math.sqrt(a))), max(8, round(s / math.sqrt(a)))))
    return out


def work(case):
    """Each input read once and each output written once; of the arithmetic, one residual's for a
    solve and the convolutions' for the network."""
    kind = case["kind"]
    if kind == "batch":
        px = sum(w * h for w, h in _sizes(case))
        return {"bytes": 4.0 * px * (3 * 3 + 1), "flops": 10.0 * px * 3}
    if kind == "dataset":
        px = case["count"] * case["size"] ** 2
        return {"bytes": 4.0 * px * 4, "flops": 10.0 * px}
    if kind == "train":
        px = case["count"] * case["height"] * case["width"]
        return {"bytes": 4.0 * px * (3 + 1 + 1) + 8.0 * _NPARAM, "flops": 3.0 * px * _conv_flops() - px * 2 * 9 * 4 * 16}
    px = case["width"] * case["height"]
    if kind == "guess":
        cells = case["channels"] * (px / case["scale"] ** 2)
        return {"bytes": 4.0 * px * (3 * case["channels"] + 1), "flops": cells * _conv_flops()}
    if kind == "mask":
        return {"bytes": 4.0 * px, "flops": 1.0 * px}
    return {"bytes": 4.0 * px * (3 * case["channels"] + 1), "flops": 10.0 * px * case["channels"]}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _waves(rng, gen, w, h, c, amplitude=1.0, highest=16.0):
    """(h, w, c) float32: 0.5 + 8 sinusoids + noise, clamped to [0, 1]."""
    x = (torch.arange(w, device=DEV, dtype=torch.float32) + 0.5) / w
    y = (torch.arange(h, device=DEV, dtype=torch.float32) + 0.5) / h
    f, th = rng.uniform(1.0, highest, (c, 8)), rng.uniform(0, 2 * math.pi, (c, 8))
    ph, am = rng.uniform(0, 2 * math.pi, (c, 8)), amplitude * rng.uniform(0.05, 0.2, (c, 8))
    put = lambda v: torch.tensor(v, device=DEV, dtype=torch.float32)[..., None]  # noqa: E731
    a = put(2 * math.pi * f * np.cos(th)) * x + put(ph)
    b = put(2 * math.pi * f * np.sin(th)) * y
    am = put(am)
    img = torch.einsum("ckh,ckw->hwc", torch.cos(b), am * torch.sin(a))
    img += torch.einsum("ckh,ckw->hwc", torch.sin(b), am * torch.cos(a))
    img += 0.5 + 0.02 * torch.randn(img.shape, generator=gen, device=DEV)
    return img.clamp_(0.0, 1.0).contiguous()


def _star(rng, w, h, n=12, area=0.30):
    """Vertices of a star with alternating radii that covers `area` of a w x h image."""
    ratio = rng.uniform(0.5, 0.8)
    turn = rng.uniform(0.0, math.pi / 6)
    r = math.sqrt(area / (0.5 * n * math.sin(2 * math.pi / n) * ratio)) if n % 2 == 0 else 0.4
    return [(w / 2 + w * r * (ratio if k % 2 else 1.0) * math.cos(turn + 2 * math.pi * k / n),
             h / 2 + h * r * (ratio if k % 2 else 1.0) * math.sin(turn + 2 * math.pi * k / n)) for k in range(n)]


def _polygon(w, h, pts, sub):
    """Coverage (h, w) float64 of a polygon under the nonzero rule, `sub` x `sub` samples a pixel:
    per sample row, +-1 at each crossing's first column not left of it, summed from the right."""
    p = np.asarray(pts, np.float64)
    q = np.roll(p, -1, 0)
    out = torch.zeros(h, w, dtype=torch.float64, device=DEV)
    step = max(1, (1 << 24) // (w * sub))
    for y0 in range(0, h, step):
        rows = min(step, h - y0)
        yy = (torch.arange(rows * sub, device=DEV, dtype=torch.float64) + 0.5) / sub + y0
        d = torch.zeros(rows * sub, w * sub + 1, dtype=torch.int32, device=DEV)
        for (ax, ay), (bx, by) in zip(p, q):
            if ay == by:
                continue
            hit = (ay <= yy) != (by <= yy)
            c = ax + (yy - ay) / (by - ay) * (bx - ax)
            col = torch.ceil(sub * c - 0.5).clamp(0, w * sub).long()
            d.scatter_add_(1, col[:, None], torch.where(hit, 1 if by > ay else -1, 0).int()[:, None])
        # a sample's winding: the crossings whose column count is beyond it
        wind = d.flip(1).cumsum(1).flip(1)[:, 1:]
        out[y0:y0 + rows] = (wind != 0).double().view(rows, sub, w, sub).sum((1, 3)) / (sub * sub)
    return out


def _ellipse(w, h, cx, cy, rx, ry, angle=0.0, half=0.0):
    """Coverage (h, w) float64 of an ellipse at pixel centres, feathered by `half` pixels."""
    x = torch.arange(w, device=DEV, dtype=torch.float64)[None, :] + 0.5 - cx
    y = torch.arange(h, device=DEV, dtype=torch.float64)[:, None] + 0.5 - cy
    u, v = math.cos(angle) * x + math.sin(angle) * y, math.cos(angle) * y - math.sin(angle) * x
    f = torch.sqrt((u / rx) ** 2 + (v / ry) ** 2)
    if half <= 0.0:
        return (f <= 1.0).double()
    grad = torch.hypot(u / rx ** 2, v / ry ** 2)
    sd = torch.where(grad > 0, (f - 1.0) * f / grad, torch.full_like(f, -1e9))
    t = ((sd + half) / (2 * half)).clamp(0.0, 1.0)
    return 1.0 - t * t * (3.0 - 2.0 * t)


def _mask(rng, w, h, shape):
    """A hard (h, w) float32 mask."""
    if shape == "star":
        return _polygon(w, h, _star(rng, w, h), 1).float()
    if shape == "regions":
        m = torch.zeros(h, w, dtype=torch.float64, device=DEV)
        for k in range(8):
            cx, cy, n = (k % 4 + 0.5) * w / 4, (k // 4 + 0.5) * h / 2, int(rng.integers(7, 14))
            t = np.sort(rng.uniform(0, 2 * math.pi, n))
            r = rng.uniform(0.6, 0.95, n)
            pts = [(cx + 0.125 * w * a * math.cos(b), cy + 0.25 * h * a * math.sin(b)) for a, b in zip(r, t)]
            m = torch.maximum(m, _polygon(w, h, pts, 1))
        return m.float()
    k = math.sqrt(4.0 * rng.uniform(0.2, 0.6) / math.pi)
    rx, ry = 0.5 * w * k, 0.5 * h * k
    cx = w / 2 + rng.uniform(-1, 1) * max(0.0, w / 2 - rx - 1)
    cy = h / 2 + rng.uniform(-1, 1) * max(0.0, h / 2 - ry - 1)
    return _ellipse(w, h, cx, cy, rx, ry).float()


def _images(rng, gen, w, h, c, shape):
    return _waves(rng, gen, w, h, c), _waves(rng, gen, w, h, c), _mask(rng, w, h, shape)


def _rngs(seed):
    return np.random.default_rng(seed), torch.Generator(DEV).manual_seed(seed)


def _geometry(case, seed):
    """What a mask case draws: a polygon's vertices, or an ellipse."""
    rng, w, h = np.random.default_rng(seed), case["width"], case["height"]
    if case["shape"] == "ellipse":
        return dict(center=(w * rng.uniform(0.4, 0.6), h * rng.uniform(0.4, 0.6)),
                    radii=(w * rng.uniform(0.15, 0.45), h * rng.uniform(0.15, 0.45)),
                    angle_rad=rng.uniform(0, math.pi), half_width_px=float(rng.choice([0.0, 1.0, 12.5])))
    return _star(rng, w, h, case["vertices"]) if case["vertices"] < 40 else [
        (w / 2 + 0.45 * w * r * math.cos(t), h / 2 + 0.45 * h * r * math.sin(t))
        for t, r in zip(2 * math.pi * np.arange(case["vertices"]) / case["vertices"],
                        rng.uniform(0.6, 1.0, case["vertices"]))]


# The network: the layout of its parameters is that of pt_unet_param_count's documentation.
_LAYERS = [(16, 16), (16, 16), (32, 16), (32, 32), (64, 32), (64, 64), (128, 64), (128, 128), (64, 192), (64, 64),
           (32, 96), (32, 32), (16, 48), (16, 16)]
_LEVELS = [0, 0, 1, 1, 2, 2, 3, 3, 2, 2, 1, 1, 0, 0]
_NPARAM = sum(o * 9 * i + o for o, i in _LAYERS) + 17
_nets = {}


def _conv_flops():
    return sum(2.0 * 9 * o * (4 if k == 0 else i) / 4 ** lev for k, ((o, i), lev) in enumerate(zip(_LAYERS, _LEVELS)))


def _weights(kind):
    """The network's flat parameters: freshly initialised to train, the trained file's to infer."""
    if kind == "guess":
        path = os.path.join(os.path.dirname(os.path.abspath(warmstart.__file__)), "weights", "warmstart_unet_256.params")
        return np.fromfile(path, dtype="<f4", offset=16)
    rng, parts = np.random.default_rng(7), []
    for k, (o, i) in enumerate(_LAYERS):
        w = rng.normal(0.0, math.sqrt(2.0 / (9 * (4 if k == 0 else i))), (o, 9, i))
        if k == 0:
            w[:, :, 4:] = 0.0
        parts += [w.ravel(), np.zeros(o)]
    return np.concatenate(parts + [rng.normal(0.0, 0.25, 16), np.zeros(1)]).astype(np.float32)


def _net(kind):
    """The one network that a program keeps for the purpose."""
    if kind not in _nets:
        net = warmstart.UNet(ops.context())
        net.set_params(_weights(kind))
        _nets[kind] = net
    return _nets[kind]


def _problems(case, seed):
    """The solves of a case: (source, target, mask) each, on the device."""
    rng, gen = _rngs(seed)
    if case["kind"] == "batch":
        return [_images(rng, gen, w, h, 3, "ellipse") for w, h in _sizes(case)]
    shape = case.get("shape", "ellipse")
    return [_images(rng, gen, case["width"], case["height"], case["channels"], shape)]


def _training(case, seed):
    """(guidance, anchor, mask, target, loss mask), each (B, H, W) on the device."""
    rng, gen = _rngs(seed)
    b, h, w = case["count"], case["height"], case["width"]
    planes = lambda **k: _waves(rng, gen, w, h, b, **k).permute(2, 0, 1).contiguous()  # noqa: E731
    g, a = planes(), planes()
    target = (planes(highest=3.0) - 0.5) * 0.5
    m = torch.stack([_mask(rng, w, h, "ellipse") for _ in range(b)])
    return g, a, m, target, warmstart.interior_mask(m.clone())


def prepare(case, seed):
    kind, ctx = case["kind"], ops.context()
    if kind == "train":
        g, a, m, target, lm = _training(case, seed)
        net = _net(kind)
        return dict(case, net=net, g=g, a=a, m=m, target=target, lm=lm,
                    record=torch.empty(net.param_count + 1, dtype=torch.float32, device=DEV))
    if kind == "mask":
        return dict(case, ctx=ctx, geometry=_geometry(case, seed))
    if kind == "dataset":
        rng, gen = _rngs(seed)
        n, s = case["count"], case["size"]
        g, a = (_waves(rng, gen, s, s, n).permute(2, 0, 1).contiguous() for _ in range(2))
        return dict(case, ctx=ctx, g=g, a=a, m=torch.stack([_mask(rng, s, s, "ellipse") for _ in range(n)]))
    problems = _problems(case, seed)
    if kind == "guess":
        g, a, m = problems[0]
        return dict(case, net=_net(kind), g=g, a=a, m=m)
    if kind in ("op", "solve_host"):
        src, tgt, m = (t.cpu().numpy() for t in problems[0])
        if kind == "solve_host":
            return dict(case, ctx=ctx, src=src, tgt=tgt, m=m)
        w, h, c = case["width"], case["height"], case["channels"]
        first, second = ("source", "target") if case["lam"] == 0.0 else ("guidance", "anchor")
        return dict(case, op=ops.PoissonBlend() if case["lam"] == 0.0 else ops.ScreenedPoisson(),
                    params={} if case["lam"] == 0.0 else {"lambda": case["lam"]},
                    inputs={first: ops.image_value(w, h, c, src), second: ops.image_value(w, h, c, tgt),
                            "mask": ops.mask_value(w, h, m)})
    flags = DEVICE | (MULTIGRID if case["method"] == "multigrid" else 0)
    omega, lam = case.get("omega", 0.0), case.get("lam", 0.0)
    if omega == 0.0:
        flags |= AUTO
    n = len(problems)
    s = dict(case, ctx=ctx, keep=problems, n=n, outs=[torch.empty_like(p[1]) for p in problems],
             reports=[(_lib.PtReport * (p[0].shape[2] + 1))() for p in problems])
    s["problems"] = (_lib.PtProblem * n)(*[
        ctx.make_problem(p[0].data_ptr(), p[1].data_ptr(), p[2].data_ptr(), p[0].shape[1], p[0].shape[0],
                         p[0].shape[2], lam, 100000, case["tol"], omega or 1.8, flags) for p in problems])
    s["out_ptrs"] = (C.c_void_p * n)(*[o.data_ptr() for o in s["outs"]])
    s["report_ptrs"] = (C.POINTER(_lib.PtReport) * n)(*[C.cast(r, C.POINTER(_lib.PtReport)) for r in s["reports"]])
    return s


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(s):
    kind = s["kind"]
    if kind == "op":
        got = s["op"].compute(s["inputs"], s["params"])
        return got["candidate"].samples, got["report"].report.solver.iterations
    if kind == "solve_host":
        out, per, _ = s["ctx"].solve(s["src"], s["tgt"], s["m"], s["width"], s["height"], s["channels"], lam=s["lam"],
                                     tolerance=s["tol"], omega=s["omega"], max_iterations=5000)
        return out, [r["iterations"] for r in per]
    if kind in ("solve", "batch"):
        L, ctx = _lib.lib(), s["ctx"]
        if kind == "solve":
            st = L.pt_poisson_solve(ctx.h, C.byref(s["problems"][0]), s["outs"][0].data_ptr(), s["reports"][0], None)
        else:
            st = L.pt_poisson_solve_batch(ctx.h, s["problems"], s["n"], s["out_ptrs"], s["report_ptrs"], None)
        if st != _lib.PT_OK:
            raise _lib.CudaError(st, ctx.last_error())
        return s["outs"], np.array([r.iterations for reps in s["reports"] for r in reps[:len(reps) - 1]], np.int64)
    if kind == "dataset":
        out, reports = warmstart.solve_batch_device(s["ctx"], s["g"], s["a"], s["m"], tol=s["tol"])
        return out, np.array([r["iterations"] for r in reports], np.int64)
    if kind == "train":
        f = s["net"].features(s["g"], s["a"], s["m"])
        return s["net"].grad_record(f, s["target"], s["lm"], out=s["record"])
    if kind == "guess":
        return warmstart.guess_image(s["net"], s["g"], s["a"], s["m"], s["scale"])
    if s["shape"] == "ellipse":
        return masks.ellipse(s["ctx"], s["width"], s["height"], **s["geometry"])
    return masks.polygon(s["ctx"], s["width"], s["height"], s["geometry"])


# ---------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------
def _interior(m):
    """mask > 0.5 away from the border, over the last two dimensions."""
    z = (m > 0.5).clone()
    z[..., 0, :] = z[..., -1, :] = False
    z[..., :, 0] = z[..., :, -1] = False
    return z


def _neighbours(u):
    """Sum of the four neighbours, (n, h, w); outside the image counts 0."""
    s = torch.zeros_like(u)
    s[:, 1:, :] += u[:, :-1, :]
    s[:, :-1, :] += u[:, 1:, :]
    s[:, :, 1:] += u[:, :, :-1]
    s[:, :, :-1] += u[:, :, 1:]
    return s


def _solution(src, tgt, m, lam, rel=1e-10, most=20000):
    """Conjugate gradients in 64 bits on planes (n, h, w): (4 + lam) u - neighbours(u) =
    lam a - laplacian(g) at interior cells, u = a elsewhere. `m`: (h, w) or (n, h, w)."""
    inside = _interior(m).expand_as(tgt)
    hit = inside.any(0)
    if not bool(hit.any()):
        return tgt.double()
    ys, xs = hit.any(1).nonzero(), hit.any(0).nonzero()
    box = (slice(None), slice(int(ys[0]) - 1, int(ys[-1]) + 2), slice(int(xs[0]) - 1, int(xs[-1]) + 2))
    g, a, k = src[box].double(), tgt[box].double(), inside[box].double()
    u = a.clone()
    r = k * ((lam * a - (_neighbours(g) - 4.0 * g)) - ((4.0 + lam) * u - _neighbours(u)))
    p, rr = r.clone(), (r * r).sum((1, 2), keepdim=True)
    first = rr.clone()
    for it in range(most):
        q = k * ((4.0 + lam) * p - _neighbours(p))
        pq = (p * q).sum((1, 2), keepdim=True)
        alpha = torch.where(pq > 0, rr / pq, torch.zeros_like(pq))
        u += alpha * p
        r -= alpha * q
        new = (r * r).sum((1, 2), keepdim=True)
        beta = torch.where(rr > 0, new / rr, torch.zeros_like(rr))
        p = r + beta * p
        rr = new
        if it % 50 == 49 and bool((rr <= rel * rel * first).all()):
            break
    out = tgt.double()
    out[box] = torch.where(k > 0, u, a)
    return out


def _solved_image(src, tgt, m, lam, rel=1e-10):
    planes = lambda t: t.permute(2, 0, 1)  # noqa: E731
    return _solution(planes(src), planes(tgt), m, lam, rel).permute(1, 2, 0).contiguous()


def _features(g, a, m):
    """(B, H, W, 4) in 64 bits."""
    inside = _interior(m)
    k = inside.double()
    lap = (_neighbours(g) - 4.0 * g) * k
    dist = torch.full_like(g, 32.0)
    pad = torch.nn.functional.pad(k, (32, 32, 32, 32))
    h, w = g.shape[1:]
    for d in range(31, 0, -1):
        for dy, dx in ((d, 0), (-d, 0), (0, d), (0, -d)):
            dist = torch.where(pad[:, 32 + dy:32 + dy + h, 32 + dx:32 + dx + w] == 0, torch.full_like(dist, float(d)), dist)
    return torch.stack([lap, (a - g) * (1.0 - k), k, dist / 32.0 * k], dim=-1)


def _network(p, f):
    """The prediction (B, H, W) of parameters `p` (flat, 64 bits) for features `f`."""
    F, at, convs = torch.nn.functional, 0, []
    for o, i in _LAYERS:
        w = p[at:at + o * 9 * i].view(o, 3, 3, i).permute(0, 3, 1, 2)
        at += o * 9 * i
        convs.append((w, p[at:at + o]))
        at += o
    conv = lambda x, k: F.relu(F.conv2d(x, convs[k][0], convs[k][1], padding=1))  # noqa: E731
    up = lambda x: F.interpolate(x, scale_factor=2, mode="bilinear", align_corners=False)  # noqa: E731
    x = F.pad(f.permute(0, 3, 1, 2), (0, 0, 0, 0, 0, 12))
    e0 = conv(conv(x, 0), 1)
    e1 = conv(conv(F.avg_pool2d(e0, 2), 2), 3)
    e2 = conv(conv(F.avg_pool2d(e1, 2), 4), 5)
    x = conv(conv(F.avg_pool2d(e2, 2), 6), 7)
    x = conv(conv(torch.cat([up(x), e2], 1), 8), 9)
    x = conv(conv(torch.cat([up(x), e1], 1), 10), 11)
    x = conv(conv(torch.cat([up(x), e0], 1), 12), 13)
    return torch.einsum("bchw,c->bhw", x, p[at:at + 16]) + p[at + 16]


def _exact_gradient(case, seed):
    g, a, m, target, lm = _training(case, seed)
    p = torch.tensor(_weights("train"), device=DEV, dtype=torch.float64, requires_grad=True)
    count, loss, part = float(lm.sum()), 0.0, 4
    for b in range(0, case["count"], part):
        f = _features(g[b:b + part].double(), a[b:b + part].double(), m[b:b + part])
        e = ((_network(p, f) - target[b:b + part].double()) ** 2 * (lm[b:b + part] > 0.5)).sum() / max(1.0, count)
        e.backward()
        loss += float(e)
    return loss, torch.cat([p.grad, torch.tensor([count], device=DEV, dtype=torch.float64)])


def _exact_guess(case, seed):
    g, a, m = (t.double() for t in _problems(case, seed)[0])
    w, h, c, s = case["width"], case["height"], case["channels"], case["scale"]
    hv, wv = -(-h // s), -(-w // s)
    hc, wc = (max(hv, 8) + 7) // 8 * 8, (max(wv, 8) + 7) // 8 * 8

    def pool(t):  # the mean of each block's pixels inside the image
        t = torch.nn.functional.pad(t, (0, wc * s - w, 0, hc * s - h))
        return t.view(-1, hc, s, wc, s).sum((2, 4))

    n = pool(torch.ones(1, h, w, dtype=torch.float64, device=DEV)).clamp(min=1.0)
    cg, ca = (pool(t.permute(2, 0, 1).contiguous()) / n for t in (g, a))
    cm = (pool(m[None]) / n).expand(c, -1, -1)
    p = torch.tensor(_weights("guess"), device=DEV, dtype=torch.float64)
    with torch.no_grad():
        corr = torch.cat([_network(p, _features(cg[k:k + 1], ca[k:k + 1], cm[k:k + 1])) for k in range(c)])[:, :hv, :wv]
    at = lambda size, n: (((torch.arange(size, device=DEV, dtype=torch.float64) + 0.5) / s) - 0.5).clamp(0.0, n - 1.0)  # noqa: E731
    fy, fx = at(h, hv), at(w, wv)
    iy, ix = fy.long(), fx.long()
    wy, wx = (fy - iy)[None, :, None], (fx - ix)[None, None, :]
    jy, jx = (iy + 1).clamp(max=hv - 1), (ix + 1).clamp(max=wv - 1)
    row = lambda i: corr[:, i][:, :, ix] * (1 - wx) + corr[:, i][:, :, jx] * wx  # noqa: E731
    return g + (row(iy) * (1 - wy) + row(jy) * wy).permute(1, 2, 0)


def exact(case, seed):
    kind = case["kind"]
    if kind == "train":
        return _exact_gradient(case, seed)
    if kind == "guess":
        return _exact_guess(case, seed)
    if kind == "mask":
        geometry = _geometry(case, seed)
        if case["shape"] == "ellipse":
            (cx, cy), (rx, ry) = geometry["center"], geometry["radii"]
            return _ellipse(case["width"], case["height"], cx, cy, rx, ry, geometry["angle_rad"],
                            geometry["half_width_px"])
        return _polygon(case["width"], case["height"], geometry, 4)
    if kind == "dataset":
        s = prepare(case, seed)
        return _solution(s["g"], s["a"], s["m"], 0.0), None
    solved = [_solved_image(*p, case.get("lam", 0.0), 1e-9 if case.get("width", 0) > 2048 else 1e-10)
              for p in _problems(case, seed)]
    if kind in ("op", "solve_host"):
        return solved[0].reshape(-1), None
    return solved, None
