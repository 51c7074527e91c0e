"""Resident classes of one batch in the clusters they share the SMs with, each
start against the streamed passes of its problem alone."""

import numpy as np
import pytest
from synthetic import triangle

import qoraphasecu_b200 as qpc
from qoraphasecu_b200.recipe import ER, HIO, Recipe

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sides,starts", [((64, 128, 256), 4), ((64, 64, 128), 9), ((64, 256), 8),
                                          ((128, 256), 20), ((64, 128), 1)])
def test_resident_classes(gpu, sides, starts):
    problems = []
    for k, side in enumerate(sides):
        _, support, intensity = triangle((side, side), side // 4)
        problems.append(qpc.make_problem(intensity * (k + 1), support=support))
    recipe = Recipe(HIO(13), ER(7))
    with qpc.BatchSolver(problems, starts=starts, seed=3, schedule="resident") as s:
        s.run(recipe)
        together = s.results()
    for p, runs in zip(problems, together, strict=True):
        with qpc.Solver(p, starts=starts, seed=3, schedule="streamed") as s:
            s.run(recipe)
            alone = s.results()
        for a, b in zip(runs, alone, strict=True):
            np.testing.assert_array_equal(a.object, b.object)
            np.testing.assert_allclose(a.errors, b.errors, rtol=1e-6)
