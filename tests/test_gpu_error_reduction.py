"""Error reduction leaves the iterate behind in the last iteration of a chunk
only: any chunk length gives the run whose every iteration writes it."""

import numpy as np
import pytest
from synthetic import triangle

import qoraphasecu_b200 as qpc
from qoraphasecu_b200.recipe import ER, HIO, Recipe, Shrinkwrap

pytestmark = pytest.mark.gpu

# register-resident, column, two-stage and run-time radix rows, 3D, and rows
# with a prime factor above 13 (34 = 2 x 17)
SHAPES = [(16, 16), (64, 32), (256, 256), (48, 512), (40, 1024), (30, 96), (50, 77), (20, 34),
          (24, 20, 18), (16, 32, 64)]


@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("variant", ["batched", "half", "mixed"])
def test_chunk_length_does_not_matter(gpu, shape, variant):
    if variant != "batched" and not all(16 <= n <= 1024 and n & (n - 1) == 0 for n in shape):
        pytest.skip("the fp16 variants take power-of-two extents")
    if variant != "batched" and shape == (16, 16):
        pytest.skip("too few lines for a tile of the fp16 variants")
    _, support, intensity = triangle(shape, 8)
    p = qpc.make_problem(intensity, support=support)
    recipe = Recipe(HIO(2), ER(5), Shrinkwrap(0.2, 1.0), ER(4), HIO(2), ER(1))
    runs = {}
    for every in (1, 3, 50):
        with qpc.Solver(p, starts=2, seed=6, sync_every=every, variant=variant,
                        schedule="streamed") as s:
            s.run(recipe)
            runs[every] = s.results()
    for every in (3, 50):
        for a, b in zip(runs[every], runs[1], strict=True):
            np.testing.assert_array_equal(a.object, b.object)
            np.testing.assert_array_equal(a.support, b.support)
            np.testing.assert_allclose(a.errors, b.errors, rtol=1e-6)
