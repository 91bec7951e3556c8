"""A last level (size max_size) whose first solving candidate does not own its
relaxed key is built a second time, in full.  In a launch of more than four
instances one warp finds that out while other CTAs still scan the instance's
table: the owner bitmap that the second build starts from must be clear.  Many
instances side by side, many times over: the answers are the oracle's in every
run."""
import pytest

import oracle
import vfb_b200
from tests import cases
from vfb_b200 import serve, synth

pytestmark = pytest.mark.gpu


def _key(g):
    return (g.rpn, g.level_rows, g.level_cands)


def _bounded(inst, max_size):
    return synth.Instance(inst.num_vars, inst.pos, inst.neg, max_size, inst.names, None, inst.rlx_type,
                          f"{inst.name}-{max_size}")


@pytest.fixture(scope="module")
def insts():
    """Strided keys (rule 1) of few long traces and mirrored hash keys, bounded
    at the level of the first solving candidate, which an earlier candidate's
    key shadows there: seeds found by an enumeration of the levels in order."""
    mirrored = cases.mirrored_cases(count=24, num_vars=5, length=18, max_size=5)
    out = [cases.random_instance(254, 8, 3, 3, 28, 5, rlx_type=1),
           _bounded(cases.random_instance(110, 6, 3, 3, 32, 5, rlx_type=1), 4),
           _bounded(cases.random_instance(112, 6, 3, 3, 32, 5, rlx_type=1), 3),
           mirrored[6], mirrored[15], _bounded(mirrored[9], 2)]
    refs = [oracle.solve(oracle.Problem.from_instance(i)) for i in out]
    return [(vfb_b200.Problem.from_instance(i), (r["rpn"], r["level_rows"], r["level_cands"]))
            for i, r in zip(out, refs)]


@pytest.mark.parametrize("copies,runs", [(1, 20), (40, 10)])
def test_batches(insts, copies, runs):
    part = insts * copies   # 6 instances, and 240 (more chunks than CTAs)
    with vfb_b200.Engine(mem_limit_bytes=8 << 30) as eng:
        for _ in range(runs):
            got = eng.batch_solve([p for p, _ in part])
            bad = [i for i, (g, (_, w)) in enumerate(zip(got, part)) if _key(g) != w]
            assert not bad, bad


def test_served(insts):
    part = insts * 20
    with vfb_b200.Engine(mem_limit_bytes=8 << 30) as eng:
        for _ in range(5):
            got, _, _ = serve.run_stream(eng, [(0.0, p) for p, _ in part], slots=64, max_steps=20000)
            bad = [i for i, (g, (_, w)) in enumerate(zip(got, part)) if _key(g) != w]
            assert not bad, bad
