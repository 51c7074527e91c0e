"""Given starts loaded into an existing batch, one array per problem."""

import numpy as np
import pytest
from synthetic import random_field, triangle

import qoraphasecu_b200 as qpc
from qoraphasecu_b200.recipe import ER, HIO, Recipe

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shapes", [[(64, 64), (30, 44), (64, 64), (16, 20, 12)], [(48, 40)] * 3],
                         ids=["mixed", "one shape"])
@pytest.mark.parametrize("layout", ["per start", "shared", "strided"])
def test_reset_equals_construction(gpu, shapes, layout):
    problems, init = [], []
    for k, shape in enumerate(shapes):
        _, support, intensity = triangle(shape, 8)
        problems.append(qpc.make_problem(intensity * (k + 1), support=support))
        starts = np.stack([random_field(int(np.prod(shape)), 7 * k + s).reshape(shape)
                           for s in (1, 2)])
        init.append({"per start": starts, "shared": starts[0],
                     "strided": np.asfortranarray(starts)}[layout])
    recipe = Recipe(HIO(3), ER(2))
    with qpc.BatchSolver(problems, starts=2, init=init) as s:
        s.run(recipe)
        first = s.results()
        s.reset(problems, seed=5)  # drawn starts in between
        s.run(recipe)
        s.reset(problems, init=init)
        s.run(recipe)
        again = s.results()
    for a, b in zip(first, again, strict=True):
        for ra, rb in zip(a, b, strict=True):
            np.testing.assert_array_equal(ra.object, rb.object)
            np.testing.assert_allclose(ra.errors, rb.errors, rtol=1e-6)
