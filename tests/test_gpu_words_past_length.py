"""Words with bits set at and past their trace's length.  Such bits are carried
along as the operators move them (F, G and U see them; a key field does not),
in every key rule and at every level: results equal the oracle's, which works
on whole words."""
import pytest

import oracle
import vfb_b200
from tests import cases
from vfb_b200 import synth

pytestmark = pytest.mark.gpu


def _dirty(inst, seed, p):
    rng = synth.Rng(seed)
    def words(length, ws):
        return length, [w | (rng.bernoulli_word(64 - length, p) << length) if length < 64 else w for w in ws]
    return synth.Instance(inst.num_vars, [words(*t) for t in inst.pos], [words(*t) for t in inst.neg], inst.max_size,
                          inst.names, None, inst.rlx_type, f"{inst.name}-past")


def _insts(rule):
    if rule == 0:   # exact keys
        out = cases.small_exact_cases() + [cases.random_instance(600 + s, 3, 3, 3, 5 + 2 * s, 6) for s in range(6)]
        out += [cases.random_instance(640, 3, 10, 10, 6, 6)]   # (rows of 20 words)
    else:
        out = cases.relaxed_cases(rule) + [cases.random_instance(660 + s, 3, 6, 6, 12 + 9 * s, 6, rlx_type=rule)
                                           for s in range(4)]
        out += [cases.random_instance(680, 3, 35, 34, 20, 5, rlx_type=rule)]
    return [_dirty(i, 77 + n, p) for n, i in enumerate(out) for p in (0.05, 0.5)]


@pytest.mark.parametrize("rule", [0, 1, 2, 3])
def test_results_equal_the_oracle(rule):
    insts = _insts(rule)
    refs = [oracle.solve(oracle.Problem.from_instance(i)) for i in insts]
    want = [(r["rpn"], r["level_rows"], r["level_cands"]) for r in refs]
    probs = [vfb_b200.Problem.from_instance(i) for i in insts]
    key = lambda g: (g.rpn, g.level_rows, g.level_cands)  # noqa: E731
    with vfb_b200.Engine(mem_limit_bytes=8 << 30) as eng:
        solo = [key(eng.solve(p)) for p in probs]
        batch = [key(r) for r in eng.batch_solve(probs)]
    static = [key(vfb_b200.solve_noalloc(p)) for p in probs]
    for name, got in (("solo", solo), ("batch", batch), ("noalloc", static)):
        bad = [i.name for i, g, w in zip(insts, got, want) if g != w]
        assert not bad, (name, bad)
