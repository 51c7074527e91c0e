"""The two-stage passes with full tiles (8 lines a block along columns, about 128
threads along rows), which a launch takes once it has 296 blocks: every length
with enough starts for them and a part of a tile at the end, against one start
a launch (small tiles) and, for a few shapes, the FP64 oracle."""

import numpy as np
import pytest
from oracle import fp64
from test_gpu_two_stage import LENGTHS, radix

import qoraphasecu_b200 as qpc
from qoraphasecu_b200.recipe import ER, HIO, Recipe, Shrinkwrap

pytestmark = pytest.mark.gpu

BLOCKS = 296


def full_tile_starts(rows, columns):
    """Starts with which both directions of a rows x columns start run full tiles."""
    threads = next(a for a in range(2, 26)
                   if columns % a == 0 and columns // a <= a and radix(a) and radix(columns // a))
    row_tiles = -(-rows // max(1, 128 // threads))
    column_tiles = -(-columns // 8)
    return -(-BLOCKS // min(row_tiles, column_tiles))


def problem(shape, seed):
    rng = np.random.default_rng(seed)
    intensity = rng.random(shape).astype(np.float32) * 100
    mask = rng.random(shape) < 0.05
    support = rng.random(shape) < 0.5
    return intensity, support, mask


@pytest.mark.parametrize("part", range(8))
def test_full_tiles_equal_small_ones(gpu, part):
    for k, n in enumerate(LENGTHS[part::8]):
        intensity, support, mask = problem((n, n), n)
        p = qpc.make_problem(intensity, support=support, mask=mask)
        runs = {}
        for variant in ("batched", "plain"):
            with qpc.Solver(p, starts=full_tile_starts(n, n), seed=2, variant=variant, batch=None
                            if variant == "plain" else full_tile_starts(n, n),
                            amp_storage=("f32", "f16", "bf16")[k % 3]) as s:
                s.run(Recipe(HIO(2), Shrinkwrap(0.1, 1.0), ER(2)))
                runs[variant] = s.results()
        for a, b in zip(runs["batched"], runs["plain"], strict=True):
            np.testing.assert_array_equal(a.object, b.object, err_msg=str(n))
            np.testing.assert_array_equal(a.support, b.support, err_msg=str(n))
            np.testing.assert_allclose(a.errors, b.errors, rtol=1e-6)


@pytest.mark.parametrize("shape,starts", [((240, 250), 16), ((300, 200), 16), ((100, 63), 40),
                                          ((96, 100, 90), 2)], ids=str)
def test_full_tiles_against_the_oracle(gpu, shape, starts):
    intensity, support, mask = problem(shape, 5)
    ref = fp64.make_problem(intensity, support, mask)
    p = qpc.make_problem(intensity, support=support, mask=mask)
    recipe = Recipe(HIO(1), ER(2))
    want = fp64.reconstruct(ref, recipe.ops(), starts=starts, seed=3)
    with qpc.Solver(p, starts=starts, seed=3, batch=starts) as s:
        s.run(recipe)
        runs = s.results()
    for (obj, _, errors), run in zip(want, runs, strict=True):
        np.testing.assert_allclose(run.errors, errors, rtol=1e-4, atol=1e-7)
        assert fp64.relative_diff(run.object, obj) < 1e-4


def test_two_problems_in_one_launch(gpu):
    problems = [qpc.make_problem(i, support=s, mask=m)
                for i, s, m in (problem((120, 90), seed) for seed in (1, 2))]
    recipe = Recipe(HIO(2), ER(2))
    with qpc.BatchSolver(problems, starts=20, seed=4) as s:
        s.run(recipe)
        together = s.results()
    for p, runs in zip(problems, together, strict=True):
        with qpc.Solver(p, starts=20, seed=4, variant="plain") as s:
            s.run(recipe)
            for a, b in zip(runs, s.results(), strict=True):
                np.testing.assert_array_equal(a.object, b.object)
                np.testing.assert_allclose(a.errors, b.errors, rtol=1e-6)
