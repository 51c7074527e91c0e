"""Every length of the two-stage passes, along columns and rows, against the
FP64 oracle (operators at 1e-5 relative L2, as everywhere)."""

import numpy as np
import pytest
from oracle import fp64
from synthetic import random_field

import qoraphasecu_b200 as qpc
from qoraphasecu_b200.recipe import ER, HIO, Recipe

pytestmark = pytest.mark.gpu


def radix(r):
    return 2 <= r <= 10 or r in (12, 14, 15, 16, 18, 20, 21, 24, 25)


LENGTHS = [n for n in range(17, 626)
           if any(n % a == 0 and n // a <= a and radix(a) and radix(n // a) for a in range(2, 26))]


@pytest.mark.parametrize("part", range(8))
def test_lengths(gpu, part):
    import torch

    from qoraphasecu_b200 import autograd

    for n in LENGTHS[part::8]:
        for shape in ((n, 11), (11, n)):
            rng = np.random.default_rng(n)
            intensity = rng.random(shape).astype(np.float32) * 100
            mask = rng.random(shape) < 0.05
            support = rng.random(shape) < 0.5
            ref = fp64.make_problem(intensity, support, mask)
            p = qpc.make_problem(intensity, support=support, mask=mask)
            x = random_field(n * 11, 3).reshape(shape)
            want, want_err = fp64.modulus_project(ref, x)
            got, err = qpc.modulus_project(p, x)
            assert fp64.relative_diff(got, want) < 1e-5, shape
            assert abs(err - want_err) <= 1e-5 * want_err, shape
            xt = autograd.to_fft_order(torch.from_numpy(x[None]).cuda(), 2).contiguous()
            xt.requires_grad_()
            autograd.amplitude_loss(xt, autograd.AmplitudeModel(p)).sum().backward()
            grad = autograd.to_centred(xt.grad, 2).cpu().numpy()[0]
            assert fp64.relative_diff(grad, 2 * (x - want)) < 1e-5, shape
        # an update that keeps the iterate, and one that leaves it alone
        start = random_field(2 * n * 11, 4).reshape(2, *shape)
        runs = fp64.reconstruct(ref, Recipe(HIO(1), ER(2)).ops(), starts=2, start=start)
        with qpc.Solver(p, starts=2, init=start) as s:
            s.run(Recipe(HIO(1), ER(2)))
            for (obj, _, errors), run in zip(runs, s.results()):
                np.testing.assert_allclose(run.errors, errors, rtol=1e-4, atol=1e-7)
                assert fp64.relative_diff(run.object, obj) < 1e-4, shape


def test_middle_axes(gpu):
    """Forward and inverse columns between two other axes."""
    for n in LENGTHS[::9]:
        shape = (3, n, 10)
        rng = np.random.default_rng(n)
        ref = fp64.make_problem(rng.random(shape).astype(np.float32), np.ones(shape, bool))
        p = qpc.make_problem(ref.amplitude.astype(np.float32) ** 2, support=np.ones(shape, bool))
        x = random_field(3 * n * 10, 3).reshape(shape)
        want, _ = fp64.modulus_project(ref, x)
        got, _ = qpc.modulus_project(p, x)
        assert fp64.relative_diff(got, want) < 1e-5, shape
