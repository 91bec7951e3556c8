"""k_p1 at the row lengths, key modes and level sizes where its loops have
edges: one trace to the most there may be (words are taken two and four at a
time, the hash folds the halves below and above T/2, the staged rows of a tile
shrink at 17, 33 and 65 words), exact keys (every operator on the packed key)
up to the full 126 bits, relaxed rules 1-3, ragged lengths with full 64-step
words.  Whole numbers: results equal the oracle's."""
import pytest

import oracle
import vfb_b200
from tests import cases
from vfb_b200 import synth

pytestmark = pytest.mark.gpu

TRACES = [1, 2, 3, 5, 8, 16, 17, 18, 32, 33, 34, 63, 64, 65, 66, 127, 128]


def _lengths(seed, n, lo, hi):
    rng = synth.Rng(seed)
    return [rng.uniform_int(lo, hi) for _ in range(n)]


def _check(insts, **kw):
    refs = [oracle.solve(oracle.Problem.from_instance(i)) for i in insts]
    probs = [vfb_b200.Problem.from_instance(i) for i in insts]
    with vfb_b200.Engine(mem_limit_bytes=8 << 30) as eng:
        got = [eng.solve(p) for p in probs] + eng.batch_solve(probs)
    for inst, g, r in zip(insts + insts, got, refs + refs):
        assert (g.rpn, g.level_rows, g.level_cands) == (r["rpn"], r["level_rows"], r["level_cands"]), inst.name


@pytest.mark.parametrize("rule", [1, 2, 3])
def test_relaxed_keys(rule):
    insts = []
    for t in TRACES:
        lens = _lengths(100 + t, t, min(64, max(4, 130 // t)), 64)
        insts.append(cases.random_instance(200 + t, 3, (t + 1) // 2, t // 2, lens, 5, rlx_type=rule))
    _check(insts)


def test_exact_keys():
    insts = []
    for t in [1, 2, 3, 5, 7, 9, 18, 31, 42, 63, 126]:
        for lens in ([126 // t if t > 1 else 64] * t, _lengths(300 + t, t, 1, min(64, 126 // t))):
            insts.append(cases.random_instance(400 + t, 3, (t + 1) // 2, t // 2, lens, 6))
    _check(insts)


@pytest.mark.parametrize("aps,t,size", [(8, 63, 6), (5, 50, 7), (6, 24, 7)])
def test_levels_of_many_tiles(aps, t, size):
    """Tiles of several staged rows and of several blocks of a unary level,
    and keys that meet other keys' slots."""
    inst = cases.random_instance(500 + t, aps, t // 2, t - t // 2, _lengths(t, t, 4, 64), size)
    _check([inst])


@pytest.mark.parametrize("solver", ["coop", "cluster"])
@pytest.mark.parametrize("t", [17, 64, 128])
def test_other_solvers(monkeypatch, solver, t):
    monkeypatch.setenv("VFB_SOLVER", solver)
    _check([cases.random_instance(600 + t, 3, t // 2, t - t // 2, _lengths(t, t, 8, 64), 5)])


@pytest.mark.parametrize("t", [1, 18, 33, 64, 128])
def test_no_alloc(t):
    inst = cases.random_instance(700 + t, 3, (t + 1) // 2, t // 2, _lengths(t, t, 7, 64), 5)
    r = oracle.solve(oracle.Problem.from_instance(inst))
    g = vfb_b200.solve_noalloc(vfb_b200.Problem.from_instance(inst))
    assert (g.rpn, g.level_rows, g.level_cands) == (r["rpn"], r["level_rows"], r["level_cands"])
