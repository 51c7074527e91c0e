"""The resident kernel at every cluster size it picks: few starts (clusters of
up to 16 CTAs) to many (the smallest cluster, more starts than fit at once),
and stages longer than one launch, against the streamed passes."""

import numpy as np
import pytest
from synthetic import triangle

import qoraphasecu_b200 as qpc
from qoraphasecu_b200.recipe import ER, HIO, Recipe

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side,starts", [(64, 1), (64, 18), (64, 19), (64, 37), (64, 74), (64, 75),
                                         (64, 160), (128, 1), (128, 9), (128, 18), (128, 37),
                                         (128, 80), (256, 1), (256, 9), (256, 20)])
@pytest.mark.parametrize("storage", ["f32", "bf16"])
def test_cluster_sizes(gpu, side, starts, storage):
    _, support, intensity = triangle((side, side), side // 4)
    p = qpc.make_problem(intensity, support=support)
    runs = {}
    for schedule in ("resident", "streamed"):
        with qpc.Solver(p, starts=starts, seed=3, schedule=schedule, amp_storage=storage) as s:
            s.run(Recipe(HIO(3), ER(2)))
            runs[schedule] = s.results()
    for a, b in zip(runs["resident"], runs["streamed"], strict=True):
        np.testing.assert_array_equal(a.object, b.object)
        np.testing.assert_allclose(a.errors, b.errors, rtol=1e-6)


def test_long_stage(gpu):
    _, support, intensity = triangle((64, 64), 16)
    p = qpc.make_problem(intensity, support=support)
    runs = {}
    for schedule in ("resident", "streamed"):
        with qpc.Solver(p, starts=2, seed=3, schedule=schedule, sync_every=50) as s:
            s.run(Recipe(ER(2003)))
            runs[schedule] = s.results()
    for a, b in zip(runs["resident"], runs["streamed"], strict=True):
        assert a.errors.shape == (2003,)
        np.testing.assert_array_equal(a.object, b.object)
        np.testing.assert_allclose(a.errors, b.errors, rtol=1e-6)
