"""Launches of up to four instances in which some are done: the buffers that
their records still name went back (to the arena, the block cache or, when
another engine of the process ends, to the device) and nothing may be read
behind them.  The others' results stay the solo ones."""
import pytest

import vfb_b200
from tests import cases

pytestmark = pytest.mark.gpu


def _key(r):
    return (r.status, r.size, r.rpn, r.level_rows, r.level_cands, r.solution_index)


@pytest.mark.parametrize("slots", [2, 4])
@pytest.mark.parametrize("arena_mb", [1, 64])
def test_finished_slots_beside_a_long_search(monkeypatch, slots, arena_mb):
    monkeypatch.setenv("VFB_SERVE_ARENA_MB", str(arena_mb))
    long_one = vfb_b200.Problem.from_instance(cases.unsatisfiable_cases((4242,))[0])
    short = [vfb_b200.Problem.from_instance(i) for i in cases.small_exact_cases()[:slots - 1]]
    probs = [long_one] + short
    with vfb_b200.Engine() as eng:
        want = [_key(eng.solve(p)) for p in probs]
    budget = cases.smallest_solo_budget([long_one], [vfb_b200.Result(*want[0][:5], 0, want[0][5], 0.0)])
    assert budget is not None
    # the long search's growth drops the finished ones' cached blocks (the
    # budget just holds it), and each ended engine trims the pool they went to
    with vfb_b200.Engine(mem_limit_bytes=budget) as eng:
        eng.serve_limits(1.0, 4 * budget, 0)
        eng.serve_open(slots, 64)
        try:
            for i, p in enumerate(probs):
                eng.serve_submit(p, i)
            got = {}
            for _ in range(2000):
                done, active, queued = eng.serve_step()
                got.update({tag: _key(r) for tag, r in done})
                if len(got) == len(probs):
                    break
                with vfb_b200.Engine(mem_limit_bytes=16 << 20):
                    pass
        finally:
            eng.serve_close()
    assert [got.get(i) for i in range(len(probs))] == want


def test_reclaimed_instances_of_a_small_batch():
    """A budget that holds one long search: the finished instances' buffers are
    taken back while it goes on."""
    probs = [vfb_b200.Problem.from_instance(i)
             for i in cases.unsatisfiable_cases((4242,)) + cases.small_exact_cases()[:3]]
    with vfb_b200.Engine() as eng:
        want = [eng.solve(p) for p in probs]
    budget = cases.smallest_solo_budget(probs[:1], want[:1])
    assert budget is not None
    for n in (2, 3, 4):
        with vfb_b200.Engine(mem_limit_bytes=budget) as eng:
            assert [_key(r) for r in eng.batch_solve(probs[:n])] == [_key(r) for r in want[:n]]
