"""k_p1 with four lanes to a stream row (small levels of few instances, keys
that take every word): trace counts around the words four lanes share and
either half of the hash, every key rule, levels on both sides of the rule's
tile count, operand levels whose rows do not fill a tile; against the oracle."""
import pytest

import oracle
import vfb_b200
from tests import cases

pytestmark = pytest.mark.gpu


def _check(inst):
    r = oracle.solve(oracle.Problem.from_instance(inst))
    with vfb_b200.Engine() as e:
        g = e.solve(vfb_b200.Problem.from_instance(inst))
    assert (g.rpn, g.level_rows, g.level_cands) == (r["rpn"], r["level_rows"], r["level_cands"])


# rows of 7, 8 (the narrowest split), 9, 10, 15-17, 31, 33, 65 and 127, 128 words
@pytest.mark.parametrize("traces", [7, 8, 9, 10, 15, 16, 17, 31, 33, 65, 127, 128])
@pytest.mark.parametrize("rule", [1, 2, 3])
def test_trace_counts(traces, rule):
    inst = cases.random_instance(500 + traces, 4, (traces + 1) // 2, traces // 2, 33, 5)
    inst.rlx_type = rule
    _check(inst)
    inst.neg[0] = inst.pos[0]   # no solution: every level is built in full
    _check(inst)


# levels from a few tiles to past the rule's count: 4 to 8 propositions, sizes to 7
@pytest.mark.parametrize("aps", [1, 2, 4, 6, 8])
@pytest.mark.parametrize("traces", [20, 40, 96])
def test_levels_on_both_sides_of_the_rule(aps, traces):
    inst = cases.random_instance(900 + 10 * aps + traces, aps, traces // 2, traces // 2, 24, 7 if aps <= 4 else 6)
    inst.neg[0] = inst.pos[0]
    _check(inst)
