"""The cache-free search's table of small formulas: one proposition to many
(the table then holds from nine sizes down to the propositions alone), one
trace to 128, solutions at every size below, at and above the table's, none at
all, and a budget with no room for the table.  Results equal the oracle's
enumeration."""
import pytest

import oracle
import vfb_b200
from tests import cases

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1, 9), (1, 5, 9), (2, 2, 8), (2, 7, 8), (3, 9, 7), (3, 128, 6), (5, 6, 6), (8, 12, 5), (20, 33, 4), (64, 128, 3)]


def _check(engine, inst):
    got = engine.solve_exhaustive(vfb_b200.Problem.from_instance(inst))
    want = oracle.exhaustive(oracle.Problem.from_instance(inst), 1 << 26)
    assert got.status == (vfb_b200.OK if want["status"] == oracle.FOUND else vfb_b200.NOT_FOUND)
    assert (got.size, got.level_cands) == (want["size"], want["level_cands"])
    if got.status == vfb_b200.OK:
        assert (got.rpn, got.solution_index) == (want["rpn"], want["solution_index"])


@pytest.mark.parametrize("budget", [8 << 30, 96 << 10])
def test_shapes(budget):
    with vfb_b200.Engine(mem_limit_bytes=budget) as engine:
        for a, t, size in SHAPES:
            for seed in range(3):
                inst = cases.random_instance(40 * a + t + 1000 * seed, a, (t + 1) // 2, t // 2, [3 + (7 * i + seed) % 62 for i in range(t)], size)
                _check(engine, inst)
