"""Graphs of a solver's chunks: error reduction replays the graph of the HIO and
RAAR stages until one of its own has paid for itself, with the same results."""

import os
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest
from synthetic import triangle

import qoraphasecu_b200 as qpc
from qoraphasecu_b200.recipe import ER, HIO, RAAR, Recipe, Shrinkwrap

pytestmark = pytest.mark.gpu

HERE = Path(__file__).resolve().parent

TRACED = """
import sys
sys.path[:0] = [{root!r}, {here!r}]
import qoraphasecu_b200 as qpc
from qoraphasecu_b200.recipe import *
from synthetic import triangle
_, support, intensity = triangle({shape!r}, 16)
p = qpc.make_problem(intensity, support=support)
with qpc.Solver(p, starts={starts}, batch={batch}, schedule="streamed", sync_every=10) as s:
    for recipe in [{recipes}]:
        s.run(recipe)
        print("--", file=sys.stderr, flush=True)
"""


def captures(shape, starts, batch, recipes):
    """Graphs captured in each of the runs of one solver."""
    code = TRACED.format(root=str(HERE.parent), here=str(HERE), shape=shape, starts=starts,
                         batch=batch, recipes=recipes)
    done = subprocess.run([sys.executable, "-c", code], env={**os.environ, "QPB_TRACE": "1"},
                          capture_output=True, text=True, check=True)
    return [part.count("graph=capture") for part in done.stderr.split("--")[:-1]]


def test_one_graph_serves_a_single_recipe(gpu):
    assert captures((256, 256), 8, 1, "Recipe(RAAR(20), ER(80)), Recipe(HIO(10), ER(10))") == [1, 0]


def test_error_reduction_alone_has_its_own(gpu):
    assert captures((256, 256), 8, 1, "Recipe(ER(20)), Recipe(RAAR(20), ER(20))") == [1, 1]


def test_a_kept_solver_ends_up_with_both(gpu):
    runs = captures((240, 240), 16, 2, ", ".join(["Recipe(RAAR(20), ER(30))"] * 40))
    assert runs[0] == 1 and sum(runs) == 2 and runs[-1] == 0


def test_one_chain_of_launches_has_both_at_once(gpu):
    # the making hides behind the RAAR stage
    assert captures((240, 240), 16, 16, "Recipe(RAAR(20), ER(80)), Recipe(RAAR(20))") == [2, 0]


@pytest.mark.parametrize("shape", [(64, 128), (240, 90), (256, 256), (32, 20, 64)],
                         ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("variant", ["batched", "half", "mixed"])
def test_runs_of_a_kept_solver_agree(gpu, shape, variant):
    if variant != "batched" and not all(n & (n - 1) == 0 for n in shape):
        pytest.skip("the fp16 variants take power-of-two extents")
    _, support, intensity = triangle(shape, 8)
    p = qpc.make_problem(intensity, support=support)
    recipe = Recipe(HIO(4), ER(7), Shrinkwrap(0.2, 1.0), RAAR(3), ER(13))
    with qpc.Solver(p, starts=4, seed=6, variant=variant, schedule="streamed", sync_every=2) as s:
        s.run(recipe)
        first = s.results()
        for _ in range(60):
            s.reset(p, seed=6)
            s.run(recipe)
        last = s.results()
    for a, b in zip(first, last, strict=True):
        np.testing.assert_array_equal(a.object, b.object)
        np.testing.assert_array_equal(a.support, b.support)
        np.testing.assert_allclose(a.errors, b.errors, rtol=1e-6)


def test_batch_of_two_shapes(gpu):
    problems = []
    for shape in [(48, 64), (256, 128)]:
        _, support, intensity = triangle(shape, 8)
        problems.append(qpc.make_problem(intensity, support=support))
    recipe = Recipe(HIO(4), ER(9), RAAR(3), ER(4))
    with qpc.BatchSolver(problems, starts=2, seed=6, schedule="streamed", sync_every=3) as s:
        s.run(recipe)
        first = s.results()
        for _ in range(80):
            s.reset(problems, seed=6)
            s.run(recipe)
        last = s.results()
    for p, a, b in zip(problems, first, last, strict=True):
        with qpc.Solver(p, starts=2, seed=6, schedule="streamed") as s:
            s.run(recipe)
            alone = s.results()
        for x, y, z in zip(a, b, alone, strict=True):
            np.testing.assert_array_equal(x.object, y.object)
            np.testing.assert_array_equal(x.object, z.object)
