"""Supports written right before a stage (shrinkwrap, detwin and its end) on the
two-stage passes, which read the support ahead of their wait for the kernel
before, against the FP64 oracle."""

import numpy as np
import pytest
from oracle import fp64
from synthetic import triangle

import qoraphasecu_b200 as qpc
from qoraphasecu_b200.recipe import ER, HIO, Recipe, Shrinkwrap, detwin

pytestmark = pytest.mark.gpu

RECIPES = {
    "shrinkwrap": Recipe(HIO(2), Shrinkwrap(0.2, 1.0), ER(1), Shrinkwrap(0.25, 1.0), HIO(1)),
    "detwin": Recipe(HIO(2), detwin(ER(1)), HIO(1), detwin(HIO(1)), ER(1)),
    "both": Recipe(ER(1), Shrinkwrap(0.2, 1.0), detwin(HIO(1)), ER(1)),
}


@pytest.mark.parametrize("shape", [(96, 100), (225, 60), (24, 20, 18)],
                         ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("recipe", RECIPES)
@pytest.mark.parametrize("variant", ["batched", "plain"])
def test_the_next_stage_sees_the_support(gpu, shape, recipe, variant):
    _, support, intensity = triangle(shape, 8)
    ref = fp64.make_problem(intensity, support)
    p = qpc.make_problem(intensity, support=support)
    recipe = RECIPES[recipe]
    want = fp64.reconstruct(ref, recipe.ops(), starts=2, seed=4)
    with qpc.Solver(p, starts=2, seed=4, variant=variant) as solver:
        solver.run(recipe)
        runs = solver.results()
    for (obj, sup, errors), run in zip(want, runs, strict=True):
        np.testing.assert_array_equal(run.support, sup)
        np.testing.assert_allclose(run.errors, errors, rtol=1e-4, atol=1e-7)
        assert fp64.relative_diff(run.object, obj) < 1e-4
