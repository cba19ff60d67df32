"""Workloads of the fixed-trajectory NUFFT CG-SENSE path, as programs run them.

A program packs its trajectory once into a plan and then calls the plan's operators and
solvers for every frame, slice or training step that was measured on that trajectory.  A case
is therefore one call on new data: the plan of a trajectory is made on its first use and kept
(as such a program keeps it), images, coil maps and k-space are made anew from the seed.

Sizes come from the configurations of the benchmark and the tests (64^2 to 256^2 images on
two-fold grids, 4 to 16 coils, golden-angle radial, variable-density spiral and 3D
golden-means trajectories, kernel width 6 for images and 4 for volumes), and, for `draw`,
from the ranges around them: every grid size that the transforms are built for, image sizes
beside half the grid, ragged sample counts.

`exact` restates each call in 64 bits with plain torch: Kaiser-Bessel gridding with the
coefficients unrounded, torch.fft, conjugate gradients and torch's own autograd.  Outputs of
the plans are off it by the FP16 rounding of the coefficients (about 1e-4).
"""

from __future__ import annotations

import functools
import math

import numpy as np
import torch

from trajsparsenufft_b200 import autograd as tad
from trajsparsenufft_b200 import synth
from trajsparsenufft_b200.operator import Batch, Plan

LAM = 1e-4
DEV = "cuda"


def listed() -> list[dict]:
    return [
        # The smallest call: one low-resolution frame to k-space (a scout or a navigator, the
        # size of the smoke run). Latency and launches count.
        _case("forward_64", "forward", n=64, g=128, coils=4, traj="radial", shots=32, readout=128),
        # A small gridding reconstruction: k-space of 4 coils to a combined 128^2 image.
        _case("adjoint_128", "adjoint", n=128, g=256, coils=4, traj="radial", shots=96, readout=256),
        # The operator pair of the headline configuration, as a caller's own solver applies it.
        _case("forward_256", "forward", n=256, g=512, coils=8, traj="radial", shots=256, readout=512),
        _case("adjoint_256", "adjoint", n=256, g=512, coils=8, traj="radial", shots=256, readout=512),
        # A pack in the reference's layout (complex coefficients), 16 coils, no maps: coil
        # images out, on a 3 * 128 grid, from a spiral with an odd sample count.
        _case("coil_images_192", "adjoint", n=192, g=384, coils=16, traj="spiral", shots=16, readout=2049,
              layout="reference", maps=False),
        # The density-weighted normal operator of a caller's own iteration: 12 coils, 5 * 128
        # grid, spiral; the coil images and Re <p, q> come back as well.
        _case("normal_320", "normal", n=320, g=640, coils=12, traj="spiral", shots=24, readout=3001, density=True),
        # The FP32-class operator (coefficients as FP16 high + low parts).
        _case("forward_exact_256", "forward", n=256, g=512, coils=8, traj="radial", shots=128, readout=512,
              layout="fp32"),
        # A small iterative reconstruction with ramp density, called plainly: the program waits
        # for the image, its residual history and the status.
        _case("cg_128", "cg", n=128, g=256, coils=4, traj="radial", shots=96, readout=256, density=True, wait=True),
        # The headline reconstruction: ten CG iterations, queued frame after frame.
        _case("cg_256", "cg", n=256, g=512, coils=8, traj="radial", shots=256, readout=512),
        # One differentiable reconstruction of a training step on 4x undersampled data:
        # forward, loss and backward, gradients of the k-space and the coil maps.
        _case("grad_256", "grad", n=256, g=512, coils=8, traj="radial", shots=128, readout=512),
        # Independent slices of uneven sizes solved together.
        {"name": "batch_8", "op": "batch", "count": 8, "mix": synth.BASE_SEED, "iters": 10},
        # The largest: the normal operator of a 128^3 volume, 8 coils, 3D golden-means spokes.
        _case("normal_128x3", "normal", dims=3, n=128, g=256, coils=8, traj="koosh", shots=2048, readout=256,
              width=4),
    ]


def _case(name, op, *, n, g, coils, traj, shots, readout, dims=2, width=6, layout="centred", maps=True,
          density=False, iters=10, wait=False) -> dict:
    c = {"op": op, "dims": dims, "n": n, "g": g, "coils": coils, "traj": traj, "shots": shots,
         "readout": readout, "width": width, "layout": layout, "maps": maps, "density": density}
    if op in ("cg", "grad"):
        c["iters"] = iters
    if op == "cg":
        c["wait"] = wait
    return {"name": name, **c} if name else c


def draw(rng) -> dict:
    """One more case of the ranges above; volumes one time in six."""
    if rng.random() < 0.08:
        return {"op": "batch", "count": rng.randint(2, 8), "mix": rng.randrange(1 << 20), "iters": rng.randint(4, 10)}
    if rng.random() < 1 / 6:
        # volumes up to the listed one's grid, samples spread over their logarithm
        g = rng.choice([128, 128, 256])
        n = 4 * rng.randint(g // 10, g // 8)
        readout = rng.randint(g // 2, g)
        shots = int(_log_uniform(rng, 64, (1 << 16 if g == 128 else 1 << 18) // readout))
        return _case("", rng.choice(["forward", "adjoint", "normal", "cg"]), dims=3, n=n, g=g,
                     coils=rng.choice([4, 8]), traj="koosh", shots=shots, readout=readout, width=4,
                     density=rng.random() < 0.3, iters=rng.randint(3, 10) if g == 128 else 1)
    op = rng.choice(["forward", "adjoint", "normal", "cg", "cg", "grad"])
    g = rng.choice([128, 256, 384, 512, 640] + ([1024] if op in ("forward", "adjoint", "normal") else []))
    n = 4 * rng.randint(g // 10, g // 8)
    coils = rng.choice([4, 8, 12, 16])
    if rng.random() < 0.5:
        traj, shots, readout = "radial", int(_log_uniform(rng, 16, 300)), rng.randint(g // 2, g)
    else:
        traj, shots, readout = "spiral", rng.randint(4, 32), int(_log_uniform(rng, 512, 4096))
    layout = rng.choice(["centred"] * 4 + ["reference", "fp32"])
    if layout == "fp32" and op not in ("forward", "adjoint"):
        layout = "centred"
    return _case("", op, n=n, g=g, coils=coils, traj=traj, shots=shots, readout=readout,
                 width=6 if rng.random() < 0.8 else 4, layout=layout,
                 maps=op not in ("forward", "adjoint") or rng.random() < 0.7,
                 density=op in ("normal", "cg") and rng.random() < 0.5, iters=rng.randint(3, 12),
                 wait=rng.random() < 0.3)


def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(max(hi, lo + 1))))


# ---- what a program has in hand ----------------------------------------------------------
def _trajectory(case) -> np.ndarray:
    make = {"radial": synth.golden_radial, "spiral": synth.vd_spiral, "koosh": synth.kooshball}
    return make[case["traj"]](case["shots"], case["readout"])


def _parts(case) -> list[dict]:
    """The single reconstructions of a batch as cases of their own."""
    out = []
    for spec in synth.uneven_batch(case["count"], case["mix"]):
        kind, size = spec["kind"].split()
        shots, readout = (int(v) for v in size.split("x"))
        out.append(_case("", "cg", n=spec["n"], g=spec["g"], coils=spec["c"], traj=kind, shots=shots,
                         readout=readout, iters=case["iters"]))
    return out


def _geometry(case) -> tuple:
    return tuple(case[k] for k in ("dims", "n", "g", "coils", "traj", "shots", "readout", "width", "layout"))


@functools.lru_cache(maxsize=32)
def _plan_of(dims, n, g, coils, traj, shots, readout, width, layout) -> Plan:
    return Plan.from_trajectory(_trajectory({"traj": traj, "shots": shots, "readout": readout}), im_size=n,
                                grid_size=g, coils=coils, width=width, device=0,
                                reference_layout=layout == "reference", reference_steps=layout == "fp32")


@functools.lru_cache(maxsize=4)
def _batch_of(geometries) -> Batch:
    return Batch([_plan_of(*geo) for geo in geometries], streams=4)


def _density(case):
    if not case["density"]:
        return None
    return torch.from_numpy(synth.ramp_density(_trajectory(case), case["readout"])).to(DEV)


def _axes(case):
    t = (torch.arange(case["n"], dtype=torch.float64, device=DEV) - case["n"] // 2) / case["n"]
    return torch.meshgrid(*([t] * case["dims"]), indexing="ij")


def _image(case, rng) -> torch.Tensor:
    """Ellipses (ellipsoids) of different sizes and magnitudes under a smooth phase."""
    ax = _axes(case)
    img = torch.zeros_like(ax[0])
    for _ in range(10):
        r2 = sum(((a - c) / h) ** 2 for a, c, h in zip(ax, rng.uniform(-0.25, 0.25, 3), rng.uniform(0.05, 0.3, 3)))
        img += rng.uniform(0.1, 1.0) * (r2 <= 1.0)
    ph = sum(float(s) * a for a, s in zip(ax, rng.uniform(-math.pi, math.pi, 3)))
    return torch.polar(img, ph).to(torch.complex64)


def _maps(case, rng) -> torch.Tensor:
    """Gaussian coil sensitivities around the field of view, root sum of squares one."""
    ax = _axes(case)
    maps = torch.empty((case["coils"], *ax[0].shape), dtype=torch.complex64, device=DEV)
    rss = torch.zeros_like(ax[0])
    for c in range(case["coils"]):
        ang = 2.0 * math.pi * (c + rng.uniform(0, 0.2)) / case["coils"]
        centre = (0.7 * math.sin(ang), 0.7 * math.cos(ang), 0.35 * math.cos(2 * ang))
        mag = torch.exp(-sum((a - q) ** 2 for a, q in zip(ax, centre)) / (2.0 * 0.4 ** 2))
        ph = sum(float(s) * a for a, s in zip(ax, rng.uniform(-math.pi, math.pi, 3)))
        maps[c] = torch.polar(mag, ph).to(torch.complex64)
        rss += mag * mag
    return maps.div_(rss.sqrt_().to(torch.float32))


def _inputs(case, seed) -> dict:
    """Images, maps, density and (where the call starts from measurements) noisy k-space."""
    rng = np.random.default_rng([seed, 2])
    x, s = _image(case, rng), _maps(case, rng)
    d = {"x": x, "maps": s, "density": _density(case)}
    if case["op"] in ("adjoint", "cg", "grad"):
        y = _kb_of(*_geometry(case)[:-1]).forward(x.to(torch.complex128), s)
        gen = torch.Generator(device=DEV).manual_seed(seed)
        noise = torch.randn((*y.shape, 2), generator=gen, device=DEV, dtype=torch.float32)
        rms = torch.linalg.vector_norm(y) / math.sqrt(y.numel())
        d["y"] = (y + (1e-3 / math.sqrt(2.0)) * rms * torch.view_as_complex(noise)).to(torch.complex64)
    if case["op"] == "forward" and not case["maps"]:
        d["x"] = (s * x).contiguous()
    return d


def prepare(case, seed):
    if case["op"] == "batch":
        parts = _parts(case)
        ins = [_inputs(p, 64 * seed + i) for i, p in enumerate(parts)]
        return {"case": case, "batch": _batch_of(tuple(_geometry(p) for p in parts)), "ys": [d["y"] for d in ins],
                "maps": [d["maps"] for d in ins], "outs": [torch.empty_like(d["x"]) for d in ins]}
    state = _inputs(case, seed)
    if case["op"] == "grad":
        state["ops"] = tad.PlanOps(_plan_of(*_geometry(case)))
    return {"case": case, "plan": _plan_of(*_geometry(case)), **state}


def run(state):
    case = state["case"]
    if case["op"] == "batch":
        outs, _ = state["batch"].cg_sense(state["ys"], state["maps"], lam=LAM, iters=case["iters"],
                                          outs=state["outs"], sync=False)
        return outs
    plan, maps = state["plan"], state["maps"] if case["maps"] else None
    fp32 = case["layout"] == "fp32"
    if case["op"] == "forward":
        return plan.forward(state["x"], maps, reference=fp32)
    if case["op"] == "adjoint":
        return plan.adjoint(state["y"], maps, reference=fp32)
    if case["op"] == "normal":
        q, coils, pq = plan.normal(state["x"], maps, density=state["density"], lam=LAM, coils=True, pq=True)
        return {"q": q, "coils": coils, "pq": pq}
    if case["op"] == "cg":
        x, hist, _ = plan.cg_sense(state["y"], maps, density=state["density"], lam=LAM, iters=case["iters"],
                                   sync=case["wait"])
        return {"x": x, "hist": hist} if case["wait"] else x
    y = state["y"].detach().requires_grad_(True)
    s = maps.detach().requires_grad_(True)
    xk = tad.cg_sense(y, s, state["ops"], lam=LAM, iters=case["iters"], checkpoint=2)
    (xk - state["x"]).abs().pow(2).sum().backward()
    return {"x": xk.detach(), "y_grad": y.grad, "maps_grad": s.grad}


# ---- what a call cannot do without ----------------------------------------------------------
def work(case) -> dict:
    """Bytes: the call's inputs once, its outputs once and the trajectory (from which every
    coefficient follows).  Operations: the interpolation's multiply-adds and the transforms of
    the oversampled grid at 5 G^d log2(G^d), for as many operator applications as there are."""
    if case["op"] == "batch":
        each = [work(p) for p in _parts(case)]
        return {k: sum(w[k] for w in each) for k in ("bytes", "flops")}
    d, c, m = case["dims"], case["coils"], case["shots"] * case["readout"]
    pix, cells = case["n"] ** d, case["g"] ** d
    one = 4.0 * c * m * case["width"] ** d + 5.0 * c * cells * math.log2(cells)
    img, coil, smp, plan = 8.0 * pix, 8.0 * pix * c, 8.0 * m * c, 4.0 * d * m + (4.0 * m if case["density"] else 0.0)
    op = case["op"]
    if op in ("forward", "adjoint"):
        return {"bytes": plan + smp + (img + coil if case["maps"] else coil), "flops": one}
    if op == "normal":
        return {"bytes": plan + 2 * img + 2 * coil, "flops": 2 * one}
    if op == "cg":
        return {"bytes": plan + smp + coil + img, "flops": (1 + 2 * case["iters"]) * one}
    # gradient: data and map cotangents beside the inputs, the reverse step applies the
    # operator pair once more per iteration
    return {"bytes": plan + 2 * smp + 2 * coil + 3 * img, "flops": (2 + 4 * case["iters"]) * one}


def tolerance(case) -> dict:
    """Four times the distance from `exact` that was measured: 7e-5 for the operators (the FP16
    coefficients), 2.6e-7 with FP16 high + low coefficients, 6e-5 for radial solves, up to 5e-3
    for solves of strongly undersampled spirals (badly conditioned: the coefficients' rounding
    grows over the iterations) and 4e-4 for gradients."""
    if case["op"] == "batch" or (case["op"] in ("cg", "grad") and case["traj"] == "spiral"):
        return {"rel": 2e-2}
    if case["op"] == "grad":
        return {"rel": 1.5e-3}
    return {"rel": 1e-6 if case["layout"] == "fp32" else 3e-4}


# ---- the same in 64 bits ------------------------------------------------------------------------
def _kb_fourier(t, g, width, beta):
    """Continuous Fourier transform of the Kaiser-Bessel kernel at t / g."""
    z2 = beta ** 2 - (math.pi * width * t / g) ** 2
    z = z2.abs().sqrt().clamp_min(1e-30)
    return width * torch.where(z2 >= 0, torch.sinh(z) / z, torch.sin(z) / z) / torch.special.i0(beta)


class _Kb:
    """Kaiser-Bessel NUFFT in FP64: image centred on the grid, real separable weights."""

    def __init__(self, dims, n, g, coils, traj, shots, readout, width):
        self.d, self.n, self.g, self.c = dims, n, g, coils
        k = torch.from_numpy(_trajectory({"traj": traj, "shots": shots, "readout": readout})).to(DEV, torch.float64)
        ratio = g / n
        beta = torch.tensor(math.pi * math.sqrt((width / ratio * (ratio - 0.5)) ** 2 - 0.8), dtype=torch.float64,
                            device=DEV)
        u = k * g
        q = torch.floor(u - width / 2).long()[:, :, None] + 1 + torch.arange(width, device=DEV)
        z = 1.0 - (2.0 * (u[:, :, None] - q) / width) ** 2
        w = torch.where(z > 0, torch.special.i0(beta * z.clamp_min(0).sqrt()) / torch.special.i0(beta), 0.0)
        q = q % g
        self.idx, self.w = q[:, 0], w[:, 0]
        for a in range(1, dims):
            self.idx = (self.idx[:, :, None] * g + q[:, a, None, :]).flatten(1)
            self.w = (self.w[:, :, None] * w[:, a, None, :]).flatten(1)
        t = torch.arange(n, dtype=torch.float64, device=DEV) - n // 2
        inv = 1.0 / _kb_fourier(t, g, width, beta)
        self.deapod = functools.reduce(lambda a, b: a[..., None] * b, [inv] * dims)
        self.pos = t.long() % g
        self.step = max(1, (1 << 26) // (self.w.shape[1] * 2 * coils))

    def _axis_index(self):
        return (slice(None), *torch.meshgrid(*([self.pos] * self.d), indexing="ij"))

    def coils_to_samples(self, u):
        grid = torch.zeros((self.c, *([self.g] * self.d)), dtype=torch.complex128, device=DEV)
        grid[self._axis_index()] = u * self.deapod
        grid = torch.fft.fftn(grid, dim=tuple(range(1, self.d + 1))).reshape(self.c, -1).T.contiguous()
        return torch.cat([(grid[i] * w[:, :, None]).sum(1) for i, w in zip(self.idx.split(self.step),
                                                                           self.w.split(self.step))]).T.contiguous()

    def samples_to_coils(self, y):
        grid = torch.zeros((self.g ** self.d, 2 * self.c), dtype=torch.float64, device=DEV)
        rows = torch.view_as_real(y.T.contiguous()).flatten(1)
        for i, w, v in zip(self.idx.split(self.step), self.w.split(self.step), rows.split(self.step)):
            grid.index_add_(0, i.flatten(), (w[:, :, None] * v[:, None, :]).flatten(0, 1))
        grid = torch.view_as_complex(grid.reshape(-1, self.c, 2)).T.reshape(self.c, *([self.g] * self.d))
        img = torch.fft.ifftn(grid, dim=tuple(range(1, self.d + 1)), norm="forward")
        return img[self._axis_index()] * self.deapod

    def forward(self, x, maps):
        return self.coils_to_samples(maps.to(torch.complex128) * x)

    def adjoint(self, y, maps):
        return (maps.conj().to(torch.complex128) * self.samples_to_coils(y)).sum(0)


@functools.lru_cache(maxsize=12)
def _kb_of(*geometry) -> _Kb:
    return _Kb(*geometry)


class _ToSamples(torch.autograd.Function):
    @staticmethod
    def forward(ctx, u, kb):
        ctx.kb = kb
        return kb.coils_to_samples(u)

    @staticmethod
    def backward(ctx, gy):
        return _ToCoils.apply(gy, ctx.kb), None


class _ToCoils(torch.autograd.Function):
    @staticmethod
    def forward(ctx, y, kb):
        ctx.kb = kb
        return kb.samples_to_coils(y)

    @staticmethod
    def backward(ctx, gu):
        return _ToSamples.apply(gu, ctx.kb), None


def _cg(kb, y, s, w, iters):
    """Conjugate gradients on (A^H W A + lam) x = A^H W y from zero: x and the residual norms."""
    weigh = (lambda v: v) if w is None else (lambda v: v * w)
    r = (s.conj() * _ToCoils.apply(weigh(y), kb)).sum(0)
    x, p = torch.zeros_like(r), r
    rho = (r.real ** 2 + r.imag ** 2).sum()
    hist = [rho]
    for _ in range(iters):
        q = (s.conj() * _ToCoils.apply(weigh(_ToSamples.apply(s * p, kb)), kb)).sum(0) + LAM * p
        alpha = rho / (p.real * q.real + p.imag * q.imag).sum()
        x, r = x + alpha * p, r - alpha * q
        new = (r.real ** 2 + r.imag ** 2).sum()
        p = r + (new / rho) * p
        rho = new
        hist.append(rho)
    return x, torch.stack(hist).sqrt()


def exact(case, seed):
    if case["op"] == "batch":
        return [_exact_one(p, _inputs(p, 64 * seed + i)) for i, p in enumerate(_parts(case))]
    return _exact_one(case, _inputs(case, seed))


def _exact_one(case, d):
    kb, op = _kb_of(*_geometry(case)[:-1]), case["op"]
    s = d["maps"].to(torch.complex128)
    w = None if d["density"] is None else d["density"].to(torch.float64)
    if op == "forward":
        return kb.forward(d["x"].to(torch.complex128), s) if case["maps"] else kb.coils_to_samples(
            d["x"].to(torch.complex128))
    if op == "adjoint":
        y = d["y"].to(torch.complex128)
        return kb.adjoint(y, s) if case["maps"] else kb.samples_to_coils(y)
    if op == "normal":
        p = d["x"].to(torch.complex128)
        y = kb.forward(p, s)
        coils = kb.samples_to_coils(y if w is None else y * w)
        q = (s.conj() * coils).sum(0) + LAM * p
        return {"q": q, "coils": coils, "pq": (p.conj() * q).real.sum()}
    if op == "cg":
        with torch.no_grad():
            x, hist = _cg(kb, d["y"].to(torch.complex128), s, w, case["iters"])
        return {"x": x, "hist": hist} if case["wait"] else x
    y = d["y"].to(torch.complex128).requires_grad_(True)
    s = s.requires_grad_(True)
    x, _ = _cg(kb, y, s, None, case["iters"])
    (x - d["x"]).abs().pow(2).sum().backward()
    return {"x": x.detach(), "y_grad": y.grad, "maps_grad": s.grad}
