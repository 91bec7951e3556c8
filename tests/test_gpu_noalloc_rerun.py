"""vfb_solve_noalloc runs the engine's level step, skipping operators past the
first solution: levels whose first solving candidate shares its relaxed key
with an earlier one are built again, and bounds below, at and above the
solution's size end as the oracle's search does."""
import pytest

import oracle
import vfb_b200
from tests import cases
from vfb_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("inst", cases.mirrored_cases(count=8) + cases.mirrored_cases(count=6, num_vars=8, length=20, max_size=5)
                         + cases.planted_cases(3), ids=lambda i: f"{i.name}_a{i.num_vars}")
def test_every_bound(inst):
    for k in range(1, min(inst.max_size, 6) + 1):
        c = synth.Instance(inst.num_vars, inst.pos, inst.neg, k, inst.names, None, inst.rlx_type, inst.name)
        r = oracle.solve(oracle.Problem.from_instance(c))
        g = vfb_b200.solve_noalloc(vfb_b200.Problem.from_instance(c))
        assert (g.rpn, g.level_rows, g.level_cands) == (r["rpn"], r["level_rows"], r["level_cands"]), k
