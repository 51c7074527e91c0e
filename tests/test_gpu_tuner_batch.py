"""A batch runs its stages in chunks, so the resident candidate of its classes is
timed in chunks, and the choice is kept apart from a solver's own."""

import os
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

HERE = Path(__file__).resolve().parent

CODE = """
import sys
sys.path[:0] = [{root!r}, {here!r}]
import qoraphasecu_b200 as qpc
from synthetic import triangle
problems = []
for side in (64, 128):
    _, support, intensity = triangle((side, side), side // 4)
    problems.append(qpc.make_problem(intensity, support=support))
{make}
print(qpc.api.tuning_report())
"""


def tuned(make):
    code = CODE.format(root=str(HERE.parent), here=str(HERE), make=make)
    done = subprocess.run([sys.executable, "-c", code], env={**os.environ, "QPB_TRACE": "1"},
                          capture_output=True, text=True, check=True)
    return done.stdout, done.stderr


def test_classes_of_a_batch_are_timed_in_chunks(gpu):
    report, trace = tuned("qpc.BatchSolver(problems, starts=2)")
    assert report.count("in a batch") == 2
    assert "run op 1/2 kind=2 n=10 " in trace and "n=20 " not in trace


def test_a_solver_is_timed_in_one_stage(gpu):
    report, trace = tuned("qpc.Solver(problems[0], starts=2); qpc.BatchSolver(problems[:1], starts=2)")
    assert "in a batch" not in report
    assert "run op 0/1 kind=2 n=20 " in trace and "run op 1/2" not in trace
