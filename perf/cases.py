"""Performance cases of the framework: what its users have it compute, through its
public entry points, over the range of sizes, types and options it is used with.

``listed()`` names the standing cases and ``draw(rng)`` gives more of the same
ranges.  ``prepare`` makes what a program holds before the call (inputs on the
GPU, the solver, network or labeller object it keeps), ``run`` is one call as a
program makes it, ``work`` the bytes and operations the call cannot do without,
and ``exact`` the same results in 64 bits with plain torch.

Kinds of case:

* ``solve2d``  one 2-D solve through ``FDTDSolver2D.forward``, with or without the
  gradient of a monitor figure of merit;
* ``solve3d``  one 3-D solve through ``FDTDSolver3D.forward``, likewise;
* ``lens``     one evaluation (figure of merit and its gradient) of the metalens
  design problem, ``Metalens3D.evaluate``;
* ``batch2d``  many 2-D grids of different sizes at once, forward and gradient,
  ``FDTDBatch2D.forward``;
* ``labels``   training labels of the surrogate, ``FDTDLabeler.label``;
* ``fno``      a training step or a prediction of the neural operator, ``FNO2d``;
* ``density``  the design layer, density to permittivity with robust variants.

A monitor's DFT comes back as complex128 whatever the solve's type; of an FP32
solve it holds FP32 field values, and a program keeps it as complex64.
"""

from __future__ import annotations

import math
from dataclasses import replace

import numpy as np
import torch
import torch.nn.functional as F
from torch.utils.checkpoint import checkpoint

F64 = torch.float64
EPS_SIO2, EPS_SI = 2.085, 12.1
WAVELENGTHS = [1500.0, 1550.0, 1600.0]


def listed():
    return [
        # the solver as its constructor's defaults make it: the smallest solve
        dict(name="tm2d default 100", kind="solve2d", pol="TM", h=100, w=100, steps=1000, pml=10,
             dtype="f32", monitors=0, grad=False),
        # a verification solve of one 256^2 TMz design with its monitor line (the
        # workload of the 2-D benchmark and of every surrogate correction)
        dict(name="tm2d 256 monitor", kind="solve2d", pol="TM", h=256, w=256, steps=2000, pml=20,
             dtype="f32", monitors=1, grad=False),
        # the large 2-D grid of the benchmark
        dict(name="tm2d 1024 monitor", kind="solve2d", pol="TM", h=1024, w=1024, steps=1000,
             pml=20, dtype="f32", monitors=1, grad=False),
        # FP64 is the validation type; the TE update of the solver's equations grows
        # without bound, so TE runs are short and in FP64; a ragged grid
        dict(name="te2d 333x270 f64", kind="solve2d", pol="TE", h=333, w=270, steps=250, pml=12,
             dtype="f64", monitors=1, grad=False),
        # one iteration of 2-D inverse design on a ragged grid: figure of merit and gradient
        dict(name="tm2d 300x413 gradient", kind="solve2d", pol="TM", h=300, w=413, steps=600,
             pml=12, dtype="f32", monitors=1, grad=True),
        # a robust-design study: ragged instances of several sizes and step counts, their
        # gradients in one backward call
        dict(name="batch2d 12 gradient", kind="batch2d", n=12, side_lo=100, side_hi=512,
             steps_lo=300, steps_hi=900, pml=20, sizes=7),
        # a chunk of training labels for the surrogate (256^2 grids, 2000 steps)
        dict(name="labels 96", kind="labels", n=96, steps=2000),
        # a small 3-D solve, line source, no monitor
        dict(name="fd3d 90 cube", kind="solve3d", d=90, h=90, w=90, steps=300, pml=8, dl=20.0,
             axes="reference", source="line", dtype="f32", monitors=0, grad=False),
        # the 3-D benchmark grid: slab and design block, plane source, monitor plane
        dict(name="fd3d 256 cube", kind="solve3d", d=256, h=256, w=256, steps=200, pml=12,
             dl=25.0, axes="reference", source="plane", dtype="f32", monitors=1, grad=False),
        # one iteration of the metalens design loop's proposing model (the coarse grid)
        dict(name="lens 96x192x192 gradient", kind="lens", d=96, h=192, w=192, steps=300, pml=6),
        # one optimiser step of the surrogate's training
        dict(name="fno train 128", kind="fno", batch=128, side=128, train=True),
        # the design layer on a full 3-D density, with eroded and dilated variants
        dict(name="density 40x256x256", kind="density", layers=40, h=256, w=256, radius=4.0,
             beta=8.0),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solve2d", "solve2d", "solve2d", "solve3d", "solve3d", "batch2d", "labels",
                       "lens", "fno", "density"])
    if kind == "solve2d":
        pol = "TE" if rng.random() < 0.2 else "TM"
        h, w = _log(rng, 64, 1400), _log(rng, 64, 1400)
        grad = rng.random() < 0.35
        if pol == "TE":
            h, w, steps, dtype = min(h, 512), min(w, 512), rng.randint(100, 300), "f64"
        else:
            dtype = "f64" if rng.random() < 0.15 else "f32"
            steps = _log(rng, 300, 2000)
            room = 2.5e8 if grad or dtype == "f64" else 1.0e9  # cell-steps
            steps = max(200, min(steps, int(room / (h * w))))
        return dict(kind=kind, pol=pol, h=h, w=w, steps=steps, pml=rng.randint(8, 20), dtype=dtype,
                    monitors=1 if grad else rng.randint(0, 1), grad=grad)
    if kind == "solve3d":
        grad = rng.random() < 0.4
        dtype = "f64" if rng.random() < 0.15 else "f32"
        axes = rng.choice(["reference", "physical"])
        hi = 144 if grad or dtype == "f64" else 224
        d, h, w = (_log(rng, 40, hi) for _ in range(3))
        if axes == "reference":
            h = w = d
        room = 1.5e8 if grad or dtype == "f64" else 1.5e9
        steps = max(60, min(_log(rng, 100, 600), int(room / (d * h * w))))
        return dict(kind=kind, d=d, h=h, w=w, steps=steps, pml=min(rng.randint(5, 12), d // 8),
                    dl=rng.choice([20.0, 25.0]), axes=axes, source=rng.choice(["line", "plane"]),
                    dtype=dtype, monitors=1 if grad else rng.randint(0, 1), grad=grad)
    if kind == "batch2d":
        lo = _log(rng, 80, 200)
        return dict(kind=kind, n=rng.randint(4, 14), side_lo=lo, side_hi=_log(rng, lo + 40, 512),
                    steps_lo=rng.randint(150, 400), steps_hi=rng.randint(400, 900), pml=20,
                    sizes=rng.randint(2, 7))
    if kind == "labels":
        return dict(kind=kind, n=_log(rng, 8, 96), steps=_log(rng, 1200, 2000))
    if kind == "lens":
        return dict(kind=kind, d=2 * rng.randint(36, 56), h=4 * rng.randint(24, 56),
                    w=4 * rng.randint(24, 56), steps=rng.randint(220, 300), pml=rng.randint(4, 8))
    if kind == "fno":
        return dict(kind=kind, batch=_log(rng, 2, 128), side=128, train=rng.random() < 0.5)
    return dict(kind="density", layers=_log(rng, 1, 40), h=_log(rng, 40, 400),
                w=_log(rng, 40, 400), radius=0.5 * rng.randint(2, 12),
                beta=float(_log(rng, 1, 32)))


# ---------------------------------------------------------------------------
# inputs, made from the seed alone
# ---------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _smooth(shape, cell, gen):
    """Smooth noise: a coarse N(0,1) map, one value per ``cell`` cells, interpolated."""
    n, h, w = shape
    c = torch.randn(n, 1, h // cell + 2, w // cell + 2, generator=gen, device="cuda")
    return F.interpolate(c, size=(h, w), mode="bilinear", align_corners=True)[:, 0]


def _blobs(n, h, w, gen):
    """0/1 Si/SiO2 design maps with features of about eight cells."""
    return (_smooth((n, h, w), 8, gen) > 0).to(torch.float32)


def _eps2d(h, w, pml, gen):
    """SiO2 with a block of Si blobs between the source and the monitor rows."""
    eps = torch.full((h, w), EPS_SIO2, device="cuda")
    a, b = pml + 12, h - pml - 6
    c, d = pml + 2, w - pml - 2
    eps[a:b, c:d] += (EPS_SI - EPS_SIO2) * _blobs(1, b - a, d - c, gen)[0]
    return eps


def _pulse(center=1550.0, width=200.0):
    spread = center ** 2 / (2.0 * math.pi * width)
    return {"type": "gaussian_pulse", "spread": spread, "t0": 3.0 * spread, "amplitude": 1.0}


def _source2d(c):
    return dict(_pulse(), row=c["pml"] + 5)


def _monitor_row(h, pml, steps):
    """The far side of the grid, or as far as the pulse is sure to come (a tenth of a
    cell per step, its speed in silicon)."""
    return min(h - pml - 3, pml + 5 + steps // 10)


def _monitor2d(c):
    return {"row": _monitor_row(c["h"], c["pml"], c["steps"]), "wavelengths_nm": WAVELENGTHS}


def _eps3d(c, gen):
    """Substrate, slab and air, with a design block of intermediate permittivities in the slab."""
    d, h, w = c["d"], c["h"], c["w"]
    eps = torch.ones(d, h, w, device="cuda")
    z, t = 3 * d // 8, max(4, d // 8)
    eps[:z] = EPS_SIO2
    eps[z:z + t] = EPS_SI
    y, x = h // 4, w // 4
    u = torch.sigmoid(3.0 * _smooth((t, h - 2 * y, w - 2 * x), 6, gen))
    eps[z:z + t, y:h - y, x:w - x] = EPS_SIO2 + (EPS_SI - EPS_SIO2) * u
    return eps


def _source3d(c):
    if c["source"] == "line":  # the solver's default source: the mid line in Ez
        return dict(_pulse())
    return dict(_pulse(), plane="xy", z=3 * c["d"] // 8 - 6, component="Ex")


def _monitor3d(c):
    """A plane inside the design block, a few cells from the source, so that a short
    solve's pulse reaches it."""
    d, h, w = c["d"], c["h"], c["w"]
    comp, z = ("Ez", 3 * d // 8 + max(4, d // 8) - 3) if c["source"] == "line" else (
        "Ex", 3 * d // 8 + 2)
    return {"component": comp, "plane": "xy", "z": z,
            "extent": [[h // 4, h - h // 4], [w // 4, w - w // 4]], "wavelengths_nm": [1550.0]}


def _batch_shapes(c):
    """Sides, step counts and wavelengths of the batch's instances."""
    n, out = c["n"], []
    for b in range(n):
        f = (b % c["sizes"]) / max(1, c["sizes"] - 1)
        side = int(round(c["side_lo"] + f * (c["side_hi"] - c["side_lo"])))
        steps = int(round(c["steps_lo"] + f * (c["steps_hi"] - c["steps_lo"])))
        out.append((side, max(side - 8 * (b % 3), 60), steps, 1450.0 + 25.0 * (b % 8)))
    return out


def _lens_setup(c):
    from diffnano_b200.design.metalens import MetalensSetup

    d, h, w = c["d"], c["h"], c["w"]
    m = min(h, w)
    return replace(MetalensSetup(), shape=(d, h, w), dl=50.0, pml=c["pml"], n_steps=c["steps"],
                   design_z=(d // 5, 2 * d // 5), design_xy=(m // 6, m - m // 6),
                   src_z=d // 5 - 5, focus_z=2 * d // 5 + 5, radius=2.0)


def _lens_rho(c, gen):
    d, m = c["d"], min(c["h"], c["w"])
    return torch.sigmoid(2.0 * _smooth((1, 2 * d // 5 - d // 5, m - m // 6 - m // 6), 6, gen))[0]


def _fno_inputs(c, seed):
    from diffnano_b200.surrogate.fno import FNOConfig

    g, n = _gen(seed), c["side"]
    cfg = FNOConfig(H=n, W=n)
    eps = EPS_SIO2 + (EPS_SI - EPS_SIO2) * _blobs(c["batch"], n, n, g)
    target = torch.randn(c["batch"], n, cfg.n_out, generator=g, device="cuda")
    C, M = cfg.width, cfg.n_modes

    def uniform(*shape, bound):
        return (2 * torch.rand(*shape, generator=g, device="cuda") - 1) * bound

    p = {"P": uniform(C, 8, bound=0.577), "p": uniform(C, bound=0.577)}
    p["P"][:, 3:] = 0
    for l in range(cfg.layers):
        p[f"wre{l}"] = uniform(M, C, C, bound=2.0 / C)
        p[f"wim{l}"] = uniform(M, C, C, bound=2.0 / C)
        p[f"W{l}"], p[f"b{l}"] = uniform(C, C, bound=C ** -0.5), uniform(C, bound=C ** -0.5)
    p["r"] = 1.0 / n + uniform(n, C, bound=0.5 / n)
    p["Q1"], p["q1"] = uniform(cfg.hidden, C, bound=C ** -0.5), uniform(cfg.hidden, bound=0.125)
    p["Q2"] = uniform(8, cfg.hidden, bound=cfg.hidden ** -0.5)
    p["Q2"][cfg.n_out:] = 0
    p["q2"] = torch.zeros(8, device="cuda")
    return cfg, eps, target, p


def _density_inputs(c, seed):
    g = _gen(seed)
    shape = (c["layers"], c["h"], c["w"])
    rho = torch.sigmoid(2.0 * _smooth(shape, 6, g) + 0.2 * torch.randn(shape, generator=g,
                                                                      device="cuda"))
    return rho, [torch.randn(shape, generator=g, device="cuda") for _ in range(3)]


# ---------------------------------------------------------------------------
# what a program has in hand, and its call
# ---------------------------------------------------------------------------
def prepare(case, seed):
    c, kind = case, case["kind"]
    s = {"case": c}
    if kind == "solve2d":
        from diffnano_b200 import FDTDSolver2D

        dt = torch.float32 if c["dtype"] == "f32" else F64
        s["solver"] = FDTDSolver2D(grid_shape=(c["h"], c["w"]), dl=20.0, wavelength_nm=1550.0,
                                   polarization=c["pol"], pml_layers=c["pml"], n_steps=c["steps"],
                                   courant=0.5, device="cuda", dtype=dt,
                                   monitors=[_monitor2d(c)] if c["monitors"] else None)
        s["eps"] = _eps2d(c["h"], c["w"], c["pml"], _gen(seed)).to(dt).requires_grad_(c["grad"])
        s["source"] = _source2d(c)
    elif kind == "solve3d":
        from diffnano_b200 import FDTDSolver3D

        dt = torch.float32 if c["dtype"] == "f32" else F64
        s["solver"] = FDTDSolver3D(grid_shape=(c["d"], c["h"], c["w"]), dl=c["dl"],
                                   wavelength_nm=1550.0, pml_layers=c["pml"], n_steps=c["steps"],
                                   courant=0.4, device="cuda", dtype=dt, cpml_axes=c["axes"],
                                   monitors=[_monitor3d(c)] if c["monitors"] else None)
        s["eps"] = _eps3d(c, _gen(seed)).to(dt).requires_grad_(c["grad"])
        s["source"] = _source3d(c)
    elif kind == "lens":
        from diffnano_b200.design.metalens import Metalens3D

        s["model"] = Metalens3D(_lens_setup(c), "cuda")
        s["rho"] = _lens_rho(c, _gen(seed))
    elif kind == "batch2d":
        from diffnano_b200.solvers.batch2d import BatchInstance, FDTDBatch2D

        g, specs, eps = _gen(seed), [], []
        for h, w, steps, wl in _batch_shapes(c):
            specs.append(BatchInstance(grid_shape=(h, w), n_steps=steps, dl=20.0, wavelength_nm=wl,
                                       pml_layers=c["pml"], courant=0.5,
                                       source=dict(_pulse(wl), row=c["pml"] + 5),
                                       monitor={"row": _monitor_row(h, c["pml"], steps),
                                                "wavelengths_nm": [wl]}))
            eps.append(_eps2d(h, w, c["pml"], g).requires_grad_(True))
        s["batch"], s["eps"] = FDTDBatch2D(specs, "TM", torch.float32, "cuda"), eps
    elif kind == "labels":
        from diffnano_b200.surrogate.data import FDTDLabeler, TMzSetup

        s["labeler"] = FDTDLabeler(replace(TMzSetup(), n_steps=c["steps"]), device="cuda")
        s["eps"] = EPS_SIO2 + (EPS_SI - EPS_SIO2) * _blobs(c["n"], 128, 128, _gen(seed))
    elif kind == "fno":
        from diffnano_b200.surrogate.fno import FNO2d

        cfg, s["eps"], s["target"], p = _fno_inputs(c, seed)
        s["net"] = FNO2d(cfg, "cuda")
        s["net"].load_state_dict(p)
    else:
        s["rho"], s["g"] = _density_inputs(c, seed)
        s["rho"].requires_grad_(True)
    return s


def run(state):
    c, kind = state["case"], state["case"]["kind"]
    if kind in ("solve2d", "solve3d"):
        from diffnano_b200.solvers import fom_abs2

        r = state["solver"].forward(state["eps"], source=dict(state["source"]))
        out = {"field": r.field.detach()}
        if c["monitors"]:
            dft = r.metadata["monitors"][0]["dft"]
            out["dft"] = dft.detach().to(torch.complex64 if c["dtype"] == "f32" else dft.dtype)
        if c["grad"]:
            (out["grad"],) = torch.autograd.grad(fom_abs2(dft), state["eps"])
        return out
    if kind == "lens":
        fom, grad, dft = state["model"].evaluate(state["rho"], 8.0)
        return {"fom": fom, "grad": grad, "dft": dft.to(torch.complex64)}
    if kind == "batch2d":
        from diffnano_b200.solvers import fom_abs2

        fields, dfts = state["batch"].forward(state["eps"])
        grads = torch.autograd.grad(sum(fom_abs2(d) for d in dfts), state["eps"])
        return {"field": [f.detach() for f in fields], "grad": list(grads),
                "dft": [d.detach().to(torch.complex64) for d in dfts]}
    if kind == "labels":
        from diffnano_b200.surrogate.data import label_scale, to_targets

        labels = state["labeler"].label(state["eps"])
        return {"targets": to_targets(labels, label_scale(labels))}
    if kind == "fno":
        net = state["net"]
        pred = net.forward(state["eps"])
        if not c["train"]:
            return {"pred": pred.clone()}
        net.loss(state["target"])
        net.ps.g.zero_()
        net.backward(B=c["batch"])
        net.adam_step(lr=1e-3)
        names = list(net.ps.offsets)
        return {"pred": pred, "grad": {k: net.ps.G(k) for k in names},
                "param": {k: net.ps.P(k) for k in names}}
    from diffnano_b200.design.projection import density_to_eps, dilate, erode

    rho, outs = state["rho"], []
    for x in (rho, erode(rho), dilate(rho)):
        outs.append(density_to_eps(x, c["radius"], c["beta"], 0.5, "tanh", EPS_SIO2, EPS_SI))
    (grad,) = torch.autograd.grad(outs, rho, state["g"])
    return {"eps": [o.detach() for o in outs], "grad": grad}


# ---------------------------------------------------------------------------
# what a call cannot do without
# ---------------------------------------------------------------------------
# operations of one cell's update: 2-D three fields, 3-D six; a reverse step does
# the transposed update and the gradient's products on top of the recomputed one
_STEP2, _STEP3 = 19.0, 42.0


def work(case):
    c, kind = case, case["kind"]
    if kind in ("solve2d", "solve3d", "lens"):
        cells = c["h"] * c["w"] * (1 if kind == "solve2d" else c["d"])
        grad = c.get("grad", True)
        word = 8 if c.get("dtype") == "f64" else 4
        fields = 1 if kind == "solve2d" else 3
        flops = cells * c["steps"] * (_STEP2 if kind == "solve2d" else _STEP3) * (3 if grad else 1)
        return {"bytes": cells * word * (1 + fields + (1 if grad else 0)), "flops": flops}
    if kind == "batch2d":
        shapes = _batch_shapes(c)
        return {"bytes": sum(h * w for h, w, _, _ in shapes) * 12,
                "flops": sum(h * w * t for h, w, t, _ in shapes) * _STEP2 * 3}
    if kind == "labels":
        return {"bytes": c["n"] * 128 * (128 + 6) * 4,
                "flops": c["n"] * 256 * 256 * c["steps"] * _STEP2}
    if kind == "fno":
        # the activations written and read once between layers, parameters with
        # gradients and moments; operations with transforms taken one axis at a time
        b, n, C, M, L, K = c["batch"], c["side"], 64, 16, 4, 128
        image = b * C * n * n
        params = L * (2 * 2 * M * M * C * C + C * C)
        transform = 2.0 * b * C * n * (2 * M) * n + 2.0 * b * C * M * (4 * M) * (2 * n)
        layer = 2 * transform + 8.0 * b * 2 * M * M * C * C + 2.0 * image * C
        head = 2.0 * b * n * (n * C + C * K + K * 6)
        if not c["train"]:
            return {"bytes": b * n * (n + 6) * 4 + (2 * L + 1) * image * 2 + params * 2,
                    "flops": L * layer + head}
        return {"bytes": b * n * (n + 6) * 4 + (6 * L + 3) * image * 2 + params * 28,
                "flops": 3 * (L * layer + head)}
    cells = c["layers"] * c["h"] * c["w"]
    taps = 2 * int(c["radius"]) + 1
    return {"bytes": cells * 4 * 8, "flops": cells * 3 * (8.0 * taps + 20)}


# ---------------------------------------------------------------------------
# the same results in 64 bits, plain torch
# ---------------------------------------------------------------------------
def _profile(n, pml, dl, dt):
    """Damping ``b`` and curl scale ``1 + c`` of one axis (cubic grading)."""
    sigma = torch.zeros(n, dtype=F64)
    for i in range(pml):
        sigma[i] = sigma[n - 1 - i] = 0.8 * ((pml - i) / pml) ** 3
    s = sigma * dl / dt
    a = 0.02 * s
    b = torch.exp(-(s + a) * dt)
    return b.cuda(), (1.0 + torch.where(s > 0, s * (b - 1.0) / (s + a + 1e-30), 0 * s)).cuda()


def _wave(steps, dt, omega, src):
    """The pulse per step; its sine is of the FP32 argument, in FP32, by definition."""
    t = torch.from_numpy(np.arange(steps, dtype=np.float64) * dt)
    env = torch.exp(-((t - src["t0"]) ** 2) / (2 * src["spread"] ** 2))
    return ((omega * t).float().sin() * src["amplitude"]).double() * env


def _phases(steps, dt, wavelengths):
    w = 2.0 * np.pi / np.asarray(wavelengths)
    return torch.from_numpy(np.exp(-1j * np.outer(np.arange(steps) * dt, w)) * dt).cuda()


def _fwd(f, dim, inv):
    n = f.shape[dim]
    d = (f.narrow(dim, 1, n - 1) - f.narrow(dim, 0, n - 1)) * inv
    return torch.cat([d, torch.zeros_like(f.narrow(dim, 0, 1))], dim)


def _bwd(f, dim, inv):
    n = f.shape[dim]
    d = (f.narrow(dim, 1, n - 1) - f.narrow(dim, 0, n - 1)) * inv
    return torch.cat([torch.zeros_like(f.narrow(dim, 0, 1)), d], dim)


def _march(step, state, steps, grad):
    """``state = step(n, *state)`` for every n, in recomputed segments under autograd."""
    seg = 25 if grad else steps

    def piece(a, b, *st):
        for n in range(a, b):
            st = step(n, *st)
        return st

    for a in range(0, steps, seg):
        b = min(steps, a + seg)
        state = (checkpoint(piece, a, b, *state, use_reentrant=False) if grad
                 else piece(a, b, *state))
    return state


def _run2d(eps, *, pol, pml, steps, center, row, mon_row, wavelengths, courant=0.5, dl=20.0,
           grad=False):
    """Final injected field and monitor-row DFT of eps ``(..., h, w)``."""
    h, w = eps.shape[-2:]
    dt = courant * dl / math.sqrt(2.0)
    (bx, gx), (by, gy) = _profile(w, pml, dl, dt), _profile(h, pml, dl, dt)
    by, gy = by[:, None], gy[:, None]
    wave = _wave(steps, dt, 2 * math.pi / center, _pulse(center)).tolist()
    ph = _phases(steps, dt, wavelengths) if mon_row is not None else None
    ce, inv = dt / eps, 1.0 / dl
    line = torch.zeros(h, 1, dtype=F64, device="cuda")
    line[row] = 1.0

    def step(n, f, a, b, acc):
        if pol == "TM":
            a = by * a - dt * gy * _fwd(f, -1, inv)
            b = bx * b + dt * gx * _fwd(f, -2, inv)
            f = bx * by * f + ce * (gx * _bwd(b, -2, inv) - gy * _bwd(a, -1, inv))
        else:
            a = bx * a + ce * gx * _bwd(f, -1, inv)
            b = by * b - ce * gy * _bwd(f, -2, inv)
            f = bx * by * f + dt * (gx * _fwd(b, -2, inv) - gy * _fwd(a, -1, inv))
        f = f + wave[n] * line
        if ph is not None:
            acc = acc + ph[n][:, None, None] * f[..., None, mon_row:mon_row + 1, :]
        return f, a, b, acc

    z = torch.zeros_like(eps)
    nw = len(wavelengths) if ph is not None else 1
    acc = torch.zeros(*eps.shape[:-2], nw, 1, w, dtype=torch.complex128, device="cuda")
    f, _, _, acc = _march(step, (z, z, z, acc), steps, grad)
    return f, acc


def _run3d(eps, *, pml, dl, steps, axes, src, comp, z_src, mon, mon_comp, wavelengths, grad=False):
    """Final (Ez, Ex, Ey) and the monitor's DFT; z_src None: the mid line source."""
    d, h, w = eps.shape
    dt = 0.4 * dl / math.sqrt(3.0)
    (bx, gx), (by, gy), (bz, gz) = (_profile(n, pml, dl, dt) for n in (w, h, d))
    i, j, k = (-1, 1, 1), (1, -1, 1), (1, 1, -1)
    # the reference mapping indexes no profile by z, and the x profile by y where
    # it scales Hy's and Ey's x differences and damps Ey
    zv, xv = (k, j) if axes == "reference" else (i, k)
    Bx, Gx, By, Gy = bx.view(k), gx.view(k), by.view(j), gy.view(j)
    Bz, Gz, Bx2, Gx2 = bz.view(zv), gz.view(zv), bx.view(xv), gx.view(xv)
    wave = _wave(steps, dt, 2 * math.pi / 1550.0, src).tolist()
    ph = _phases(steps, dt, wavelengths) if mon is not None else None
    ce, inv = dt / eps, 1.0 / dl
    mask = torch.zeros(d, h, 1, dtype=F64, device="cuda")
    if z_src is None:
        mask[d // 2, h // 2] = 1.0
    else:
        mask[z_src] = 1.0

    def step(n, ex, ey, ez, hx, hy, hz, acc):
        hx = By * hx - dt * (Gy * _fwd(ez, 1, inv) - Gz * _fwd(ey, 0, inv))
        hy = Bz * hy - dt * (Gz * _fwd(ex, 0, inv) - Gx2 * _fwd(ez, 2, inv))
        hz = Bx * hz - dt * (Gx * _fwd(ey, 2, inv) - Gy * _fwd(ex, 1, inv))
        ex = By * Bz * ex + ce * (Gy * _bwd(hz, 1, inv) - Gz * _bwd(hy, 0, inv))
        ey = Bz * Bx2 * ey + ce * (Gz * _bwd(hx, 0, inv) - Gx2 * _bwd(hz, 2, inv))
        ez = Bx * By * ez + ce * (Gx * _bwd(hy, 2, inv) - Gy * _bwd(hx, 1, inv))
        add = wave[n] * mask
        ex, ey, ez = (e + add if c == comp else e
                      for e, c in ((ex, "Ex"), (ey, "Ey"), (ez, "Ez")))
        if ph is not None:
            f = {"Ex": ex, "Ey": ey, "Ez": ez}[mon_comp]
            acc = acc + ph[n][:, None, None, None] * f[mon]
        return ex, ey, ez, hx, hy, hz, acc

    z = torch.zeros_like(eps)
    acc = torch.zeros(len(wavelengths), *z[mon].shape, dtype=torch.complex128,
                      device="cuda") if mon is not None else torch.zeros(1, device="cuda")
    ex, ey, ez, _, _, _, acc = _march(step, (z,) * 6 + (acc,), steps, grad)
    return torch.stack([ez, ex, ey]), acc


def _fom(dft):
    return torch.view_as_real(dft).square().sum()


def _taps(radius):
    n = int(2 * radius + 1)
    n += 1 - n % 2
    t = torch.arange(n, dtype=F64, device="cuda") - n // 2
    g = torch.exp(-(t ** 2) / (2 * (radius / 2.0) ** 2 + 1e-12))
    return g / g.sum()


def _design(rho, radius, beta, lo, hi):
    g = _taps(radius)
    n = g.numel()
    x = F.conv2d(rho[:, None], g.view(1, 1, 1, n), padding=(0, n // 2))
    x = F.conv2d(x, g.view(1, 1, n, 1), padding=(n // 2, 0))[:, 0]
    t = math.tanh(0.5 * beta)
    return lo + (hi - lo) * (t + torch.tanh(beta * (x - 0.5))) / (2 * t)


def _exact_fno(c, seed):
    cfg, eps, target, p = _fno_inputs(c, seed)
    train, n, M = c["train"], c["side"], cfg.modes
    p = {k: v.double().requires_grad_(train) for k, v in p.items()}
    eps, target = eps.double(), target.double()

    def layer(l, X):
        Z = torch.fft.rfft2(X)
        w = torch.complex(p[f"wre{l}"], p[f"wim{l}"]).view(2 * M, M, cfg.width, cfg.width)
        low = torch.cat([Z[:, :, :M, :M], Z[:, :, n - M:, :M]], 2)
        low = torch.einsum("bixy,xyoi->boxy", low, w)
        low = F.pad(low, (0, n // 2 + 1 - M))
        mid = torch.zeros(*low.shape[:2], n - 2 * M, n // 2 + 1, dtype=low.dtype, device="cuda")
        Y = torch.fft.irfft2(torch.cat([low[:, :, :M], mid, low[:, :, M:]], 2), s=(n, n))
        Y = Y + torch.einsum("bihw,oi->bohw", X, p[f"W{l}"]) + p[f"b{l}"][:, None, None]
        return F.gelu(Y, approximate="tanh") if l < cfg.layers - 1 else Y

    def net(eps):
        x = torch.linspace(0, 1, n, dtype=F64, device="cuda")
        f = torch.zeros(*eps.shape, 8, dtype=F64, device="cuda")
        f[..., 0] = (eps - cfg.eps_lo) / (cfg.eps_hi - cfg.eps_lo)
        f[..., 1], f[..., 2] = x, x[:, None]
        X = torch.einsum("bhwf,cf->bchw", f, p["P"]) + p["p"][:, None, None]
        for l in range(cfg.layers):
            X = checkpoint(layer, l, X, use_reentrant=False) if train else layer(l, X)
        R = torch.einsum("bchw,hc->bwc", X, p["r"])
        U = F.gelu(R @ p["Q1"].T + p["q1"], approximate="tanh")
        return (U @ p["Q2"].T + p["q2"])[..., :cfg.n_out]

    parts = range(0, c["batch"], 16)
    if not train:
        with torch.no_grad():
            return {"pred": torch.cat([net(eps[a:a + 16]) for a in parts])}
    preds = []
    for a in parts:  # sums over the samples: gradients add up part by part
        pred = net(eps[a:a + 16])
        ((pred - target[a:a + 16]) ** 2).sum().div(target.numel()).backward()
        preds.append(pred.detach())
    grad = {k: v.grad for k, v in p.items()}
    # the first Adam step: both moments' bias corrections cancel
    param = {k: v.detach() - 1e-3 * grad[k] / (grad[k].abs() + 1e-8) for k, v in p.items()}
    return {"pred": torch.cat(preds), "grad": grad, "param": param}


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind == "solve2d":
        dt = torch.float32 if c["dtype"] == "f32" else F64
        eps = _eps2d(c["h"], c["w"], c["pml"], _gen(seed)).to(dt).double()
        eps.requires_grad_(c["grad"])
        src = _source2d(c)
        f, dft = _run2d(eps, pol=c["pol"], pml=c["pml"], steps=c["steps"], center=1550.0,
                        row=src["row"], mon_row=_monitor2d(c)["row"] if c["monitors"] else None,
                        wavelengths=WAVELENGTHS, grad=c["grad"])
        out = {"field": f.detach()[None]}
    elif kind == "solve3d":
        dt = torch.float32 if c["dtype"] == "f32" else F64
        eps = _eps3d(c, _gen(seed)).to(dt).double().requires_grad_(c["grad"])
        src, mon = _source3d(c), _monitor3d(c)
        box = (slice(mon["z"], mon["z"] + 1),) + tuple(slice(*r) for r in mon["extent"])
        f, dft = _run3d(eps, pml=c["pml"], dl=c["dl"], steps=c["steps"], axes=c["axes"], src=src,
                        comp=src.get("component", "Ez"), z_src=src.get("z"),
                        mon=box if c["monitors"] else None, mon_comp=mon["component"],
                        wavelengths=mon["wavelengths_nm"], grad=c["grad"])
        out = {"field": f.detach()}
    elif kind == "lens":
        s = _lens_setup(c)
        rho = _lens_rho(c, _gen(seed)).double().requires_grad_(True)
        e2 = _design(rho[None], s.radius, 8.0, s.eps_lo, s.eps_hi)[0]
        (z0, z1), (a, b) = s.design_z, s.design_xy
        eps = torch.full(s.shape, s.eps_lo, dtype=F64, device="cuda")
        eps[:z0] = s.eps_sub
        eps[z0:z1, a:b, a:b] = e2[:, None, :].expand(z1 - z0, b - a, b - a)
        y = c["h"] // 2
        box = (slice(s.focus_z, s.focus_z + 1), slice(y, y + 1), slice(a, b))
        _, dft = _run3d(eps, pml=s.pml, dl=s.dl, steps=s.n_steps, axes="physical", src=_pulse(),
                        comp="Ey", z_src=s.src_z, mon=box, mon_comp="Ey",
                        wavelengths=list(s.wavelengths_nm), grad=True)
        dft = dft.reshape(len(s.wavelengths_nm), -1)
        fom = _fom(dft[s.center_index, s.focus_col:s.focus_col + 1])
        (grad,) = torch.autograd.grad(fom, rho)
        return {"fom": float(fom.detach()), "grad": grad, "dft": dft.detach()}
    elif kind == "batch2d":
        g, out = _gen(seed), {"field": [], "grad": [], "dft": []}
        for h, w, steps, wl in _batch_shapes(c):
            eps = _eps2d(h, w, c["pml"], g).double().requires_grad_(True)
            f, dft = _run2d(eps, pol="TM", pml=c["pml"], steps=steps, center=wl, row=c["pml"] + 5,
                            mon_row=_monitor_row(h, c["pml"], steps), wavelengths=[wl], grad=True)
            out["field"].append(f.detach())
            out["grad"].append(torch.autograd.grad(_fom(dft), eps)[0])
            out["dft"].append(dft.detach())
        return out
    elif kind == "labels":
        from diffnano_b200.surrogate.data import TMzSetup

        s = replace(TMzSetup(), n_steps=c["steps"])
        eps = torch.full((c["n"], s.side, s.side), EPS_SIO2, dtype=F64, device="cuda")
        a, b = s.offset, s.offset + s.design
        eps[:, a:b, a:b] = EPS_SIO2 + (EPS_SI - EPS_SIO2) * _blobs(c["n"], 128, 128, _gen(seed))
        _, dft = _run2d(eps, pol="TM", pml=s.pml, steps=s.n_steps, center=s.center_nm,
                        row=s.src_row, mon_row=s.mon_row, wavelengths=list(s.wavelengths_nm))
        d = dft[:, :, 0, a:b]
        scale = torch.sqrt((d.abs() ** 2).mean())
        return {"targets": torch.view_as_real(d).permute(0, 2, 1, 3).reshape(c["n"], 128, -1) / scale}
    elif kind == "fno":
        return _exact_fno(c, seed)
    else:
        rho, g = _density_inputs(c, seed)
        rho = rho.double().requires_grad_(True)
        grown = F.max_pool2d(rho[:, None], 3, 1, 1)[:, 0]
        shrunk = -F.max_pool2d(-rho[:, None], 3, 1, 1)[:, 0]
        outs = [_design(x, c["radius"], c["beta"], EPS_SIO2, EPS_SI) for x in (rho, shrunk, grown)]
        (grad,) = torch.autograd.grad(outs, rho, [x.double() for x in g])
        return {"eps": [o.detach() for o in outs], "grad": grad}
    if c["monitors"]:
        out["dft"] = dft.detach()
    if c["grad"]:
        (out["grad"],) = torch.autograd.grad(_fom(dft), eps)
    return out
