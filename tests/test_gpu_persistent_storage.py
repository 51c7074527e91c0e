"""The persistent schedule with the amplitude stored in 16 bits."""

import numpy as np
import pytest
from synthetic import triangle

import qoraphasecu_b200 as qpc
from qoraphasecu_b200.recipe import ER, HIO, Recipe

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("storage", ["f16", "bf16"])
@pytest.mark.parametrize("shape", [(64, 64), (128, 64), (64, 256)])
def test_persistent_reads_the_stored_amplitude(gpu, shape, storage):
    """Same amplitude, same arithmetic: the same objects as the streamed passes."""
    _, support, intensity = triangle(shape, 20)
    p = qpc.make_problem(intensity, support=support)
    runs = {}
    for schedule in ("persistent", "streamed"):
        with qpc.Solver(p, starts=3, seed=2, schedule=schedule, amp_storage=storage) as s:
            s.run(Recipe(HIO(6), ER(4)))
            runs[schedule] = s.results()
    for a, b in zip(runs["persistent"], runs["streamed"], strict=True):
        np.testing.assert_array_equal(a.object, b.object)
        np.testing.assert_allclose(a.errors, b.errors, rtol=1e-6)
