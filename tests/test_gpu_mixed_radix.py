"""The mixed-radix passes (lengths that are no power of two, or a power of two
whose lines do not fill the other passes' tiles) against the FP64 oracle."""

import numpy as np
import pytest
from oracle import fp64
from synthetic import random_field, triangle

import qoraphasecu_b200 as qpc
from qoraphasecu_b200.recipe import ER, HIO, Recipe, Shrinkwrap

pytestmark = pytest.mark.gpu

# Every radix 2..16 alone, lines of 1 to 5 stages, line counts that leave the
# last block of a start part empty, 3D middle axes, axes of length 1.
SHAPES = [(2, 3), (4, 5), (6, 7), (9, 10), (11, 12), (13, 14), (15, 9), (1, 30), (26, 1), (30, 44),
          (16, 15), (35, 64), (100, 96), (225, 91), (240, 33), (300, 200), (1001, 6), (9, 3125),
          (8190, 2), (5, 14, 33), (15, 2, 16), (24, 40, 18), (32, 12, 64)]


def problem(shape, seed):
    rng = np.random.default_rng(seed)
    intensity = rng.random(shape).astype(np.float32) * 100
    mask = rng.random(shape) < 0.05
    mask.flat[0] = False
    support = rng.random(shape) < 0.5
    support.flat[-1] = True
    return (fp64.make_problem(intensity, support, mask),
            qpc.make_problem(intensity, support=support, mask=mask))


@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_operators(gpu, shape):
    ref, p = problem(shape, 5)
    x = random_field(int(np.prod(shape)), 7).reshape(shape)
    want, want_err = fp64.modulus_project(ref, x)
    for storage in ("f32", "f16", "bf16"):
        got, err = qpc.modulus_project(p, x, amp_storage=storage)
        # FP32 rounding; 16-bit amplitudes to their relative spacing
        tol = {"f32": 1e-5, "f16": 2.0**-10, "bf16": 2.0**-7}[storage]
        assert fp64.relative_diff(got, want) < tol, storage
        assert abs(err - want_err) <= tol * max(want_err, 1.0), storage
    image = np.abs(x)
    want = fp64.gaussian_blur(image, 0.8)
    assert np.abs(qpc.gaussian_blur(image, 0.8) - want).max() < 1e-5 * np.abs(want).max()


@pytest.mark.parametrize("shape", [(30, 44), (225, 91), (24, 40, 18), (32, 12, 64)],
                         ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("method", ["max", "rms"])
def test_solver(gpu, shape, method):
    obj, support, intensity = triangle(shape, 8)
    ref = fp64.make_problem(intensity, support)
    p = qpc.make_problem(intensity, support=support)
    recipe = Recipe(HIO(2), ER(2), Shrinkwrap(0.2, 1.0, method), ER(1))
    want = fp64.reconstruct(ref, recipe.ops(), starts=3, seed=4)
    with qpc.Solver(p, starts=3, seed=4) as solver:
        solver.run(recipe)
        runs = solver.results()
    for (obj_w, _, err_w), run in zip(want, runs):
        np.testing.assert_allclose(run.errors, err_w, rtol=1e-4, atol=1e-7)
        assert fp64.relative_diff(run.object, obj_w) < 1e-4


def test_gradient(gpu):
    import torch

    from qoraphasecu_b200 import autograd

    for shape in [(30, 44), (100, 96), (12, 20, 18)]:
        ref, p = problem(shape, 9)
        x = np.stack([random_field(int(np.prod(shape)), s).reshape(shape) for s in (1, 2)])
        xt = autograd.to_fft_order(torch.from_numpy(x).cuda(), len(shape)).contiguous().requires_grad_()
        losses = autograd.amplitude_loss(xt, autograd.AmplitudeModel(p))
        losses.sum().backward()
        grad = autograd.to_centred(xt.grad, len(shape)).cpu().numpy()
        for b in range(2):
            want, _ = fp64.modulus_project(ref, x[b])
            free = 2 * (x[b] - want)
            # masked pixels keep their own magnitude in the projection
            assert np.linalg.norm(grad[b] - free) < 1e-5 * np.linalg.norm(x[b])
