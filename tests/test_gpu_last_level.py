"""The last level of a search (size max_size) is counted, not written, unless
something needs its rows: nothing found, a solution at that very level (& | ~ X F
G or U), relaxed-key collisions there, a BS stage afterwards, a
batch whose instances end at different levels, buffers that grow at that
level.  Results equal the oracle's."""
import pytest

import oracle
import vfb_b200
from tests import cases
from vfb_b200 import synth

pytestmark = pytest.mark.gpu


def _key(g):
    return (g.rpn, g.level_rows, g.level_cands)


def _ref(i):
    r = oracle.solve(oracle.Problem.from_instance(i))
    return (r["rpn"], r["level_rows"], r["level_cands"])


def _each_max_size(inst, top):
    out = []
    for k in range(1, top + 1):
        c = synth.Instance(inst.num_vars, inst.pos, inst.neg, k, inst.names, None, inst.rlx_type,
                                 f"{inst.name}-{k}")
        out.append(c)
    return out


def test_every_bound_of_a_search():
    """Bounds below, at and above the solution's size, solo and in one batch."""
    insts = []
    for base in (cases.planted_cases(4) + cases.small_exact_cases()[:4] + cases.relaxed_cases(1)[:2]
                 + cases.mirrored_cases(count=4) + cases.unsatisfiable_cases((4242,))):
        insts += _each_max_size(base, min(base.max_size, 7))
    want = [_ref(i) for i in insts]
    probs = [vfb_b200.Problem.from_instance(i) for i in insts]
    with vfb_b200.Engine(mem_limit_bytes=8 << 30) as eng:
        cold = [_key(eng.solve(p)) for p in probs]      # buffers grow on the way
        warm = [_key(eng.solve(p)) for p in probs]
        batch = [_key(r) for r in eng.batch_solve(probs)]
    for name, got in (("cold", cold), ("warm", warm), ("batch", batch)):
        bad = [i.name for i, g, w in zip(insts, got, want) if g != w]
        assert not bad, (name, bad)


def test_bs_stage_reads_the_last_level():
    inst = cases.random_instance(31, 3, 6, 6, 12, 4)
    r = oracle.solve_bs(oracle.Problem.from_instance(inst), 9)
    with vfb_b200.Engine(mem_limit_bytes=8 << 30) as eng:
        p = vfb_b200.Problem.from_instance(inst)
        eng.solve(p)
        g = eng.solve_bs(p, 9)
    assert _key(g) == (r["rpn"], r["level_rows"], r["level_cands"])
