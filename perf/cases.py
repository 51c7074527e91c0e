"""The work that users of this framework have it do, as timed cases.

A case is a dict of plain values; ``prepare`` makes what a program holds before
the call (measured intensities, the problem, a live solver), ``run`` is one pass
through the public entry points, ``exact`` the same pass in 64 bits with torch
alone.

Kinds of pass:

* ``solver`` - a program that reconstructs a stream of diffraction patterns of
  one shape keeps a ``Solver``, loads each pattern with its starting objects
  (``reset``), runs the recipe and takes the results, all on the device;
* ``host`` - one ``reconstruct()`` call on numpy arrays, the call most programs
  make;
* ``batch`` - a ``BatchSolver`` over problems of several shapes, results on the
  host;
* ``loss`` - one step of gradient-based reconstruction: the amplitude loss of a
  batch of objects and its gradient.

The data are the square-object patterns of ``qoraphasecu_b200.workloads``
(random amplitude and phase in a centred box of 24/64 of the field), with
Poisson counts and a beamstop. Starts are given, as in a refinement: the object
with a tenth of noise on it, so that a pass of many iterations has a definite
result (from random starts the feedback iterations amplify rounding until two
programs no longer have the same answer).
"""

from __future__ import annotations

import math

import numpy as np
import torch

import qoraphasecu_b200 as qpc
from qoraphasecu_b200 import autograd
from qoraphasecu_b200.recipe import ER, HIO, RAAR, Recipe, Shrinkwrap

EPS = 1e-12


def _solver(name, n0, n1, n2, starts, *, raar=20, hio=0, shrink=True, er=80, amp="f32", stop=True):
    """A ``solver`` case; 2D when ``n0`` is 0."""
    return {"name": name, "kind": "solver", "n0": n0, "n1": n1, "n2": n2, "starts": starts,
            "raar": raar, "hio": hio, "shrink": shrink, "er": er, "amp": amp, "stop": stop}


def listed():
    return [
        # One small frame, refined from one start: launches and latency.
        _solver("frame_64_s1", 0, 64, 64, 1, shrink=False, er=30),
        # The small benchmark problem: 8 starts of 64 x 64, support updated on the way.
        _solver("frame_64_s8", 0, 64, 64, 8),
        # A few starts of a medium frame, amplitude stored in fp16.
        _solver("frame_128_s4_f16", 0, 128, 128, 4, amp="f16"),
        # The headline benchmark's ensemble: 32 starts of 256 x 256.
        _solver("ensemble_256_s32", 0, 256, 256, 32),
        # A cropped detector whose side is no power of two.
        _solver("crop_240_s16", 0, 240, 240, 16, hio=20, raar=0),
        # An uneven crop, each axis with its own factors.
        _solver("crop_300x200_s4", 0, 300, 200, 4),
        # A large frame, several starts (the differentiable benchmark's side).
        _solver("frame_512_s16", 0, 512, 512, 16, er=60),
        # The 3D benchmark's size: a Bragg peak of 128^3, 4 starts, no beamstop.
        _solver("volume_128_s4", 128, 128, 128, 4, raar=10, er=30, stop=False),
        # A 3D crop whose sides are no powers of two.
        _solver("volume_96_s2", 96, 96, 96, 2, raar=10, er=30, stop=False),
        # A scan of patterns of mixed shapes in one batch, two starts each.
        {"name": "scan_mixed_s2", "kind": "batch", "starts": 2, "problems": 10, "mix": 3,
         "raar": 0, "hio": 20, "shrink": True, "er": 60, "amp": "f32", "stop": True},
        # reconstruct() on numpy arrays, 8 starts of 256 x 256.
        {"name": "host_256_s8", "kind": "host", "n0": 0, "n1": 256, "n2": 256, "starts": 8,
         "raar": 20, "hio": 0, "shrink": True, "er": 80, "amp": "f32", "stop": True},
        # A gradient step's loss and gradient: 16 objects of 512 x 512.
        {"name": "loss_512_b16", "kind": "loss", "n0": 0, "n1": 512, "n2": 512, "starts": 16,
         "stop": True},
    ]


def _side(rng, lo, hi):
    """A side in [lo, hi], even over its logarithm: half of the time a power of
    two, else a size with small prime factors (7 at most, now and then 11 or 13)."""
    n = round(lo * (hi / lo) ** rng.random())
    if rng.random() < 0.5:
        return min(hi, max(lo, 2 ** round(math.log2(n))))
    largest = 13 if rng.random() < 0.2 else 7
    while True:
        m = n
        for p in (2, 3, 5, 7, 11, 13):
            while p <= largest and m % p == 0:
                m //= p
        if m == 1:
            return n
        n = n - 1 if n > lo else hi


def draw(rng):
    kind = rng.choice(["solver", "solver", "solver", "solver", "volume", "batch", "host", "loss"])
    amp = rng.choice(["f32", "f32", "f16", "bf16"])
    feedback = rng.choice([(20, 0), (0, 20), (10, 5)])
    if kind == "volume":
        sides = [_side(rng, 24, 128) for _ in range(3)]
        most = max(1, min(4, 4 * 128**3 // (sides[0] * sides[1] * sides[2])))
        return {"kind": "solver", "n0": sides[0], "n1": sides[1], "n2": sides[2],
                "starts": rng.randint(1, most), "raar": feedback[0] // 2, "hio": feedback[1] // 2,
                "shrink": rng.random() < 0.5, "er": rng.randint(10, 30), "amp": amp, "stop": False}
    if kind == "batch":
        return {"kind": "batch", "starts": 2, "problems": rng.randint(3, 10),
                "mix": rng.randint(10, 10**6), "raar": feedback[0], "hio": feedback[1],
                "shrink": rng.random() < 0.5, "er": rng.randint(20, 60), "amp": "f32",
                "stop": True}
    n1 = _side(rng, 48, 512)
    n2 = n1 if rng.random() < 0.5 else _side(rng, 48, 512)
    most = max(1, min(32, 16 * 512 * 512 // (n1 * n2)))
    starts = max(1, round(most ** rng.random()))
    if kind == "loss":
        return {"kind": "loss", "n0": 0, "n1": n1, "n2": n2, "starts": starts,
                "stop": rng.random() < 0.8}
    return {"kind": kind, "n0": 0, "n1": n1, "n2": n2,
            "starts": min(starts, 20) if kind == "host" else starts,
            "raar": feedback[0], "hio": feedback[1], "shrink": rng.random() < 0.7,
            "er": rng.randint(20, 80), "amp": amp, "stop": rng.random() < 0.8}


# ------------------------------------------------------------------- inputs
def _shape(case):
    return tuple(n for n in (case["n0"], case["n1"], case["n2"]) if n)


def _scan_shapes(case):
    """The shapes of a ``batch`` case: mostly the benchmark's sides, some crops."""
    rng = np.random.default_rng(case["mix"])
    shapes = []
    for _ in range(case["problems"]):
        n = int(rng.choice([64, 128, 256, 512, 96, 200]))
        shapes.append((n, n))
    return shapes


def _coords(shape):
    axes = [torch.arange(n, device="cuda") - n // 2 for n in shape]
    return torch.meshgrid(*axes, indexing="ij")


def _measure(shape, stop, seed):
    """A square object on ``shape`` and its measurement: object (scaled to the
    counts), intensity, mask and support, centre-origin, on the device."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    dims = tuple(range(len(shape)))
    amp = 0.4 + 0.6 * torch.rand(shape, generator=g, device="cuda", dtype=torch.float64)
    phase = (2 * torch.rand(shape, generator=g, device="cuda", dtype=torch.float64) - 1) * math.pi
    inside = torch.ones(shape, dtype=torch.bool, device="cuda")
    for c, n in zip(_coords(shape), shape):
        m = max(1, round(24 * n / 64))
        inside &= (c >= -(m // 2)) & (c < m - m // 2)
    obj = torch.polar(amp, phase) * inside
    wave = torch.fft.fftshift(torch.fft.fftn(torch.fft.ifftshift(obj, dim=dims), norm="ortho"), dim=dims)
    intensity = wave.abs() ** 2
    scale = (1e6 if len(shape) == 2 else 1e7) / float(intensity.max())
    counts = torch.poisson(intensity * scale, generator=g).to(torch.float32)
    mask = torch.zeros(shape, dtype=torch.bool, device="cuda")
    if stop:
        mask = sum(c.double() ** 2 for c in _coords(shape)) <= (min(shape) / 32) ** 2
    return obj * math.sqrt(scale), counts, mask, inside


def _starts(obj, count, noise, seed):
    g = torch.Generator(device="cuda").manual_seed(seed + 1)
    re, im = (torch.randn((count, *obj.shape), generator=g, device="cuda", dtype=torch.float64)
              for _ in range(2))
    return (obj * (1 + noise * torch.complex(re, im))).to(torch.complex64)


def _recipe(case):
    stages = []
    if case["raar"]:
        stages.append(RAAR(case["raar"]))
    if case["hio"]:
        stages.append(HIO(case["hio"]))
    if case["shrink"]:
        stages.append(Shrinkwrap(0.1, 1.0))
    stages.append(ER(case["er"]))
    return Recipe(*stages)


def _loss_inputs(case, seed):
    shape = _shape(case)
    obj, counts, mask, support = _measure(shape, case["stop"], seed)
    x = torch.fft.ifftshift(_starts(obj, case["starts"], 0.5, seed), dim=(-2, -1)).contiguous()
    return counts, mask, support, x


def prepare(case, seed):
    kind = case["kind"]
    if kind == "loss":
        counts, mask, support, x = _loss_inputs(case, seed)
        problem = qpc.make_problem(counts.cpu().numpy(), support=support.cpu().numpy(),
                                   mask=mask.cpu().numpy())
        return {"kind": kind, "model": autograd.AmplitudeModel(problem), "x": x.requires_grad_(True)}
    if kind == "batch":
        problems, init = [], []
        for k, shape in enumerate(_scan_shapes(case)):
            obj, counts, mask, support = _measure(shape, case["stop"], seed + 17 * k)
            problems.append(qpc.make_problem(counts.cpu().numpy(), support=support.cpu().numpy(),
                                             mask=mask.cpu().numpy()))
            init.append(_starts(obj, case["starts"], 0.1, seed + 17 * k).cpu().numpy())
        solver = qpc.BatchSolver(problems, starts=case["starts"], amp_storage=case["amp"], init=init)
        return {"kind": kind, "solver": solver, "problems": problems, "init": init,
                "recipe": _recipe(case)}
    obj, counts, mask, support = _measure(_shape(case), case["stop"], seed)
    init = _starts(obj, case["starts"], 0.1, seed)
    state = {"kind": kind, "recipe": _recipe(case), "starts": case["starts"], "amp": case["amp"]}
    if kind == "host":
        return state | {"intensity": counts.cpu().numpy(), "mask": mask.cpu().numpy(),
                        "support": support.cpu().numpy(), "init": init.cpu().numpy()}
    problem = qpc.make_problem(counts, support=support, mask=mask)
    solver = qpc.Solver(problem, starts=case["starts"], amp_storage=case["amp"], init=init)
    return state | {"problem": problem, "solver": solver, "init": init}


def run(state):
    kind = state["kind"]
    if kind == "loss":
        x, model = state["x"], state["model"]
        x.grad = None
        losses = autograd.amplitude_loss(x, model)
        losses.sum().backward()
        errors = torch.sqrt(losses.detach() / (model.energy + EPS)).to(torch.float32)
        return {"errors": errors, "grad": x.grad}
    if kind == "batch":
        solver = state["solver"]
        solver.reset(state["problems"], init=state["init"])
        solver.run(state["recipe"])
        runs = [r for of_problem in solver.results() for r in of_problem]
    elif kind == "host":
        found = qpc.reconstruct(state["intensity"], support=state["support"], mask=state["mask"],
                                recipe=state["recipe"], starts=state["starts"],
                                init=state["init"], amp_storage=state["amp"])
        runs = list(found) if state["starts"] > 1 else [found]
    else:
        solver = state["solver"]
        solver.reset(state["problem"], init=state["init"])
        solver.run(state["recipe"])
        runs = solver.results()
    supports = [r.support for r in runs]
    errors = [r.errors for r in runs]
    if len(runs) > 20:  # a large ensemble's supports and histories as one array each
        supports = torch.stack(supports)
        errors = np.stack(errors)
    return {"objects": [r.object for r in runs], "supports": supports, "errors": errors}


def _iterations(case):
    return case["raar"] + case["hio"] + case["er"]


def _numel(case):
    """Elements of all starts, and of all problems, of a pass."""
    if case["kind"] == "batch":
        per_start = sum(math.prod(s) for s in _scan_shapes(case))
    else:
        per_start = math.prod(_shape(case))
    return case["starts"] * per_start, per_start


def _transform_flops(case):
    """FLOPs of one n-D transform of every start, 5 n log2 n each."""
    shapes = _scan_shapes(case) if case["kind"] == "batch" else [_shape(case)]
    return case["starts"] * sum(5 * math.prod(s) * math.log2(math.prod(s)) for s in shapes)


def work(case):
    """An iteration reads the iterate (8 bytes), its support (1) and the shared
    amplitude (4, or 2 stored in 16 bits) once and writes the iterate once (8);
    it transforms forward and back and spends about 20 operations per element
    on the projection and the update. Around the iterations the starts come in
    and the objects (8) and supports (1) go out."""
    elements, shared = _numel(case)
    if case["kind"] == "loss":  # x in, the gradient out, one amplitude
        return {"bytes": 16.0 * elements + 4.0 * shared,
                "flops": 2 * _transform_flops(case) + 15.0 * elements}
    it = _iterations(case)
    amp = 4.0 if case["amp"] == "f32" else 2.0
    flops = it * (2 * _transform_flops(case) + 20.0 * elements)
    if case["shrink"]:
        flops += 2 * _transform_flops(case)
    return {"bytes": it * (17.0 * elements + amp * shared) + 17.0 * elements + 6.0 * shared,
            "flops": float(flops)}


# -------------------------------------------------------------------- exact
def _exact_runs(case, shape, counts, mask, support, init):
    """Objects (centre-origin) and error histories of every start, in 64 bits."""
    dims = tuple(range(-len(shape), 0))
    amp = torch.fft.ifftshift(torch.sqrt(counts.double()), dim=dims)
    bad = torch.fft.ifftshift(mask, dim=dims)
    s = torch.fft.ifftshift(support, dim=dims).expand(case["starts"], *shape)
    x = torch.fft.ifftshift(init.to(torch.complex128), dim=dims) * s
    usable = amp[~bad]
    energy = float((usable * usable).sum())
    errors = []

    def iterate(count, a, b):
        nonlocal x
        for _ in range(count):
            y = torch.fft.fftn(x, dim=dims, norm="ortho")
            mag = y.abs()
            off = torch.where(bad, torch.zeros_like(mag), mag - amp)
            errors.append(torch.sqrt((off * off).sum(dims) / (energy + EPS)))
            target = torch.where(bad, mag, amp)
            p = torch.fft.ifftn(y * (target / (mag + EPS)), dim=dims, norm="ortho")
            x = torch.where(s, p, a * x + b * p)

    beta = 0.9
    iterate(case["raar"], beta, 1 - 2 * beta)
    iterate(case["hio"], 1.0, -beta)
    if case["shrink"]:
        f2 = sum(f * f for f in torch.meshgrid(
            *[torch.fft.fftfreq(n, device="cuda", dtype=torch.float64) for n in shape], indexing="ij"))
        blurred = torch.fft.ifftn(torch.fft.fftn(x.abs(), dim=dims)
                                  * torch.exp(-2 * (math.pi * 1.0) ** 2 * f2), dim=dims).real
        s = blurred > 0.1 * blurred.amax(dims, keepdim=True)
    iterate(case["er"], 0.0, 0.0)
    objects = torch.fft.fftshift(x, dim=dims)
    history = torch.stack(errors, dim=1)  # (starts, iterations)
    return list(objects), [h.cpu().numpy() for h in history]


def exact(case, seed):
    kind = case["kind"]
    if kind == "loss":
        counts, mask, support, x = _loss_inputs(case, seed)
        amp = torch.fft.ifftshift(torch.sqrt(counts.double()))
        bad = torch.fft.ifftshift(mask)
        y = torch.fft.fft2(x.to(torch.complex128), norm="ortho")
        mag = y.abs()
        off = torch.where(bad, torch.zeros_like(mag), mag - amp)
        grad = torch.fft.ifft2(2 * off * y / (mag + EPS), norm="ortho")
        usable = amp[~bad]
        energy = float((usable * usable).sum())
        return {"errors": torch.sqrt((off * off).sum((-2, -1)) / (energy + EPS)), "grad": grad}
    if kind == "batch":
        parts = [(s, seed + 17 * k) for k, s in enumerate(_scan_shapes(case))]
    else:
        parts = [(_shape(case), seed)]
    objects, errors = [], []
    for shape, part_seed in parts:
        obj, counts, mask, support = _measure(shape, case["stop"], part_seed)
        init = _starts(obj, case["starts"], 0.1, part_seed)
        o, e = _exact_runs(case, shape, counts, mask, support, init)
        objects += o
        errors += e
    if len(objects) > 20:
        return {"objects": objects, "supports": None, "errors": np.stack(errors)}
    return {"objects": objects, "supports": [None] * len(objects), "errors": errors}
