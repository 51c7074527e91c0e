"""The length of a resident launch is bounded by the work in it: starts that run
in several waves split a long stage into more launches."""

import numpy as np
import pytest
from synthetic import triangle

import qoraphasecu_b200 as qpc
from qoraphasecu_b200.recipe import ER, Recipe

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("starts,launches", [(8, 1), (300, 4)])
def test_launches_of_a_long_stage(gpu, starts, launches):
    _, support, intensity = triangle((64, 64), 16)
    p = qpc.make_problem(intensity, support=support)
    counts = {}
    with qpc.Solver(p, starts=starts, seed=1, schedule="resident") as s:
        for iterations in (10, 1000):
            s.reset(p, seed=1)
            before = qpc.api.kernel_launches()
            s.run(Recipe(ER(iterations)))
            counts[iterations] = qpc.api.kernel_launches() - before
        last = s.results()
    # a launch is the kernel and the counter's advance
    assert counts[1000] - counts[10] == 2 * (launches - 1)
    with qpc.Solver(p, starts=starts, seed=1, schedule="streamed") as s:
        s.run(Recipe(ER(1000)))
        for a, b in zip(last, s.results(), strict=True):
            np.testing.assert_array_equal(a.object, b.object)
            np.testing.assert_allclose(a.errors, b.errors, rtol=1e-6)
