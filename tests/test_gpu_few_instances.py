"""The table scan's two forms, up to four instances and more than four, must
agree: the same instances alone, in batches of 2 to 6, with levels from a few
candidates (one CTA scans, checks and compacts) to tens of thousands (several
CTAs, k_compact), relaxed-key collisions that build a level again, and buffers
that grow in between.  Results equal the oracle's."""
import pytest

import oracle
import vfb_b200
from tests import cases

pytestmark = pytest.mark.gpu


def _key(g):
    return (g.rpn, g.level_rows, g.level_cands)


@pytest.fixture(scope="module")
def insts():
    out = cases.mirrored_cases(count=6) + cases.small_exact_cases()[:3] + cases.planted_cases(3)
    out += cases.unsatisfiable_cases((4243, 4244)) + cases.relaxed_cases(3)[:2]
    refs = [oracle.solve(oracle.Problem.from_instance(i)) for i in out]
    return [(vfb_b200.Problem.from_instance(i), i.name, (r["rpn"], r["level_rows"], r["level_cands"]))
            for i, r in zip(out, refs)]


@pytest.mark.parametrize("size", [1, 2, 3, 4, 5, 6])
def test_batches_of(insts, size):
    with vfb_b200.Engine(mem_limit_bytes=8 << 30) as eng:
        for _ in range(2):   # cold, then with the final buffer sizes
            for at in range(0, len(insts), size):
                part = insts[at:at + size]
                got = eng.batch_solve([p for p, _, _ in part])
                bad = [n for g, (_, n, w) in zip(got, part) if _key(g) != w]
                assert not bad, bad
