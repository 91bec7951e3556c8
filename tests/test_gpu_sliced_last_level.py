"""A served request's last level built in slices (step_candidates): its buffers
are checked once, when the last slice is through, against the level's owners.
Solutions in a late slice and none at all, under a byte cap that just holds the
request and with a memory budget that just holds a solo solve: the results are
those of the level built in one piece."""
import pytest

import oracle
import vfb_b200
from tests import cases
from vfb_b200 import synth

pytestmark = pytest.mark.gpu


def _key(r):
    return (r.status, r.size, r.rpn, r.level_rows, r.level_cands, r.solution_index)


def _serve_one(eng, prob, cap, step):
    """The result of prob as the only request of a session."""
    eng.serve_limits(1.0, cap, step)
    eng.serve_open(1, 128)
    try:
        eng.serve_submit(prob, 0)
        for _ in range(20000):
            done, _, _ = eng.serve_step()
            if done:
                return _key(done[0][1])
    finally:
        eng.serve_close()
    return None


# seeds of planted formulas found at sizes 5 to 7, at the end of that level's
# 745 to 143,000 candidates before them (late slices hold them)
SEEDS = [2, 3, 9, 12, 17, 23, 24, 36]


@pytest.mark.parametrize("seed", SEEDS)
def test_byte_cap_of_whole_levels_holds_slices(seed):
    inst = synth.planted_instance(synth.Rng(8100 + seed), 5, 7, 14, 14, (12, 40), 0.5, 8, name=f"late{seed}")
    r = oracle.solve(oracle.Problem.from_instance(inst))
    for max_size in (r["size"], r["size"] - 1):   # the last level solved, and not
        prob = vfb_b200.Problem.from_instance(
            synth.Instance(inst.num_vars, inst.pos, inst.neg, max_size, inst.names, None, 3, inst.name))
        with vfb_b200.Engine(mem_limit_bytes=2 << 30) as eng:
            want = _key(eng.solve(prob))   # (the sessions then start from its final buffer sizes)
            # the smallest cap, within a percent, that holds the level in one piece
            lo, hi = 1 << 16, 1 << 29
            assert _serve_one(eng, prob, hi, 0) == want
            while hi - lo > hi // 128:
                mid = (lo + hi) // 2
                if _serve_one(eng, prob, mid, 0) == want:
                    hi = mid
                else:
                    lo = mid
            for step in (150, 600, 2500, 20000):
                assert _serve_one(eng, prob, hi, step) == want, (max_size, hi, step)


def test_budget_of_a_solo_solve_holds_slices():
    prob = vfb_b200.Problem.from_instance(cases.unsatisfiable_cases((4242,))[0])
    with vfb_b200.Engine() as eng:
        full = eng.solve(prob)
    budget = cases.smallest_solo_budget([prob], [full])
    assert budget is not None
    for step in (0, 5000, 100000):
        with vfb_b200.Engine(mem_limit_bytes=budget) as eng:
            assert _serve_one(eng, prob, 4 * budget, step) == _key(full), step
