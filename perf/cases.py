"""The work that users have this engine do, as cases with sizes.

Every case goes through the Python entry points (Engine.solve, batch_solve,
solve_costs, solve_bs, solve_exhaustive, the serving loop, solve_noalloc) on
host data, as the engine takes it: trace words and lengths, uploaded by the
call.  What comes back is whole numbers: status, size, formula, the unique
sets and candidates of every size and the solution's index, which do not
depend on timing.  An engine (and a serving session) is a handle that a
program opens once and keeps.

listed() gives the fixed cases, draw(rng) one more of the same ranges,
prepare(case, seed) the inputs, run(state) one pass, work(case) its bytes and
operations, exact(case, seed) nothing: there are no rounded outputs.
"""
from __future__ import annotations

import random

import numpy as np

import vfb_b200
from vfb_b200 import synth

LARGE_BYTES = synth.LARGE_MEM_BYTES   # budget of the solving engine
SERVE_BYTES = 24 << 30                # budget of the serving engine (its session's arena)
SERVE_SLOTS = 64
SERVE_TRACES = 64                     # traces of a served request at most
OPS = {c: -(1 + i) for i, c in enumerate(vfb_b200.OPS)}
UNIT_COSTS = "1 1 1 1 1 1 1 1"


def _case(kind, name=None, **kw):
    c = {"kind": kind, "aps": 4, "pos": 20, "neg": 20, "len_lo": 16, "len_hi": 16, "p": 0.5, "planted": 0,
         "max_size": 8, "rule": 3, "count": 1, "costs": UNIT_COSTS, "neg_type": 1, "bs_max": 0}
    c.update(kw)
    if name is not None:
        c["name"] = name
    return c


def listed():
    return [
        # a handful of short traces, as in the small test configurations: an
        # answer within a few levels, all latency
        _case("solve", "tiny", aps=3, pos=4, neg=4, len_lo=6, len_hi=6, max_size=10),
        # the ordinary interactive call: 20+20 traces labelled by a formula of
        # size 9, as in the benchmark's planted configuration
        _case("solve", "planted", planted=9, max_size=10),
        # exact keys: 18 traces of 7 steps (126 bits), labels without a planted
        # formula, so the search ends where the sets become many enough
        _case("solve", "exact", pos=9, neg=9, len_lo=7, len_hi=7, max_size=9),
        # ragged lengths, an odd number of traces, no formula up to the bound:
        # the whole space of size 9 and less is enumerated
        _case("solve", "ragged", aps=6, pos=24, neg=25, len_lo=4, len_hi=64, max_size=9),
        # relaxed uniqueness rule 1 (strided samples), the most traces an
        # instance may have
        _case("solve", "strided", aps=5, pos=64, neg=64, len_lo=32, len_hi=32, max_size=8, rule=1),
        # the benchmark's large instance (8 propositions, 31+32 traces of
        # length 64, solved at size 10), propositions and traces in another order
        _case("large", "large", aps=8, pos=31, neg=32, len_lo=64, len_hi=64, p=0.3, planted=13, max_size=17),
        # many samples in one call: the mixed batch (2..8 propositions, 4..63
        # traces of 4..64 steps), searched to size 8
        _case("batch", "batch", aps=8, pos=31, neg=32, len_lo=4, len_hi=64, planted=8, count=256),
        # a burst of such requests at an open serving session
        _case("serve", "serve", aps=8, pos=31, neg=32, len_lo=4, len_hi=64, planted=7, max_size=7, count=48),
        # operator costs other than 1 (levels are costs)
        _case("costs", "costs", pos=20, neg=21, max_size=12, costs="1 1 2 2 1 1 1 2"),
        # the search to size 5, then combinations of the cached formulas
        _case("bs", "combine", pos=8, neg=8, len_lo=12, len_hi=12, max_size=5, bs_max=12),
        # the cache-free search in formula-number order, few traces: it ends at
        # its first formula, of size 5 to 9
        _case("exhaustive", "nocache", aps=3, pos=5, neg=5, len_lo=4, len_hi=24, max_size=9),
        # the call that may not allocate, within its static scratch
        _case("noalloc", "noalloc", planted=6, max_size=7),
    ]


def _cands(case):
    """Estimated unique sets and candidates of a search: (sets, candidates).
    Blocks of the size (or cost) order; about 0.55 of a level's candidates are
    new on traces long and many enough to tell them apart, and a search whose
    labels follow no formula ends where the sets outnumber the labellings."""
    atom, c_not, c_and, c_or, c_x, c_f, c_g, c_u = (int(x) for x in case["costs"].split())
    t = case["pos"] + case["neg"]
    top = 10 if case["kind"] == "large" else case["max_size"]
    if case["planted"] and case["kind"] != "large":
        top = min(top, case["planted"])
    room = 2.0 ** min(60.0, t * (case["len_lo"] + case["len_hi"]) / 2)
    n, total = {atom: float(case["aps"])}, float(case["aps"])
    for k in range(atom + 1, top + 1):
        g = sum(n.get(k - w, 0.0) for w in (c_not, c_x, c_f, c_g))
        for w, half in ((c_and, True), (c_or, True), (c_u, False)):
            for i in range(atom, k - w - atom + 1):
                j = k - w - i
                if not half or i <= j:
                    g += n.get(i, 0.0) * n.get(j, 0.0)
        if case["kind"] == "large" and k == top:
            g *= 0.55   # up to its solution
        total += g
        n[k] = min(0.55 * g, max(0.0, room - sum(n.values())))
        if not case["planted"] and sum(n.values()) > 2.0 ** min(60, t):
            break
    return sum(n.values()), total


def draw(rng):
    """One more case: a kind, then sizes over its range; the size bound is the
    largest whose estimated candidates stay within the largest listed case's."""
    kind = rng.choice(["solve"] * 6 + ["costs", "batch", "batch", "serve", "bs", "exhaustive", "noalloc"])
    c = _case(kind, aps=rng.randint(2, 8), p=rng.choice([0.3, 0.5]))
    if kind in ("batch", "serve"):
        c.update(pos=31, neg=32, len_lo=4, len_hi=64, planted=rng.randint(5, 7), count=round(2 ** rng.uniform(1, 7 if kind == "batch" else 5)))
        c["max_size"] = c["planted"]
        return c
    t = round(2 ** rng.uniform(2, 7))
    c.update(pos=max(1, t // 2), neg=max(1, t - t // 2))
    c["len_lo"] = rng.randint(3, 40)
    c["len_hi"] = rng.choice([c["len_lo"], rng.randint(c["len_lo"], 64)])
    c["rule"] = rng.choice([3, 3, 3, 1, 2])
    if kind in ("solve", "noalloc"):
        c["planted"] = rng.choice([0, 0, rng.randint(4, 9)])
    limit = 2.0 ** rng.uniform(10, 24.5)
    if kind == "noalloc":
        limit = min(limit, 2.0 ** 17)
    if kind == "bs":
        c.update(aps=min(c["aps"], 4), pos=rng.randint(4, 8), neg=rng.randint(4, 8), bs_max=rng.randint(7, 11))
        limit = min(limit, 2.0 ** 14)
    if kind == "exhaustive":
        c.update(aps=min(c["aps"], 4), pos=rng.randint(2, 6), neg=rng.randint(2, 6), max_size=rng.randint(5, 7))
        return c
    if kind == "costs":
        c["costs"] = " ".join(str(rng.randint(1, 3)) for _ in range(8))
        c["neg_type"] = rng.choice([1, 1, 2])
    c["max_size"] = 3
    while c["max_size"] < 16 and _cands(dict(c, planted=0, pos=64, neg=64, max_size=c["max_size"] + 1))[1] <= limit:
        c["max_size"] += 1
    return c


# --------------------------------------------------------------------- inputs
def _traces(case, seed):
    """Random traces without a planted formula; words[i * aps + v]."""
    g = np.random.default_rng(seed)
    t, a = case["pos"] + case["neg"], case["aps"]
    lens = g.integers(case["len_lo"], case["len_hi"] + 1, t)
    bits = (g.random((t, a, 64)) < case["p"]) & (np.arange(64) < lens[:, None, None])
    words = np.packbits(bits, axis=-1, bitorder="little").view(np.uint64).reshape(-1)
    return words.tolist(), lens.tolist()


def _problem(case, seed):
    if case["planted"]:
        inst = synth.planted_instance(synth.Rng(seed), case["aps"], case["planted"], case["pos"], case["neg"],
                                      (case["len_lo"], case["len_hi"]), case["p"], case["max_size"])
        inst.rlx_type = case["rule"]
        return vfb_b200.Problem.from_instance(inst)
    words, lens = _traces(case, seed)
    names = [f"a{v}" for v in range(case["aps"])]
    return vfb_b200.Problem(case["aps"], case["pos"], words, lens, names, case["max_size"], case["rule"], max(lens))


def _large(case, seed):
    """The large instance with its propositions renumbered and its positive
    and its negative traces reordered: the same search depth for every seed."""
    inst = synth.config_large_deep(case["max_size"])
    r = random.Random(seed)
    order = r.sample(range(inst.num_vars), inst.num_vars)
    move = lambda ts: [(n, [w[v] for v in order]) for n, w in r.sample(ts, len(ts))]  # noqa: E731
    inst.pos, inst.neg = move(inst.pos), move(inst.neg)
    return vfb_b200.Problem.from_instance(inst)


def _mixed(case, seed):
    """count samples of the mixed batch's shapes, searched to max_size."""
    rng = synth.Rng(seed)
    probs = []
    for _ in range(case["count"]):
        a = rng.uniform_int(2, case["aps"])
        t = rng.uniform_int(4, case["pos"] + case["neg"])
        size = rng.uniform_int(min(5, case["planted"]), case["planted"])
        inst = synth.planted_instance(rng, a, size, t // 2, t - t // 2, (case["len_lo"], case["len_hi"]), case["p"],
                                      case["max_size"])
        probs.append(vfb_b200.Problem.from_instance(inst))
    return probs


_engines = {}


def _engine(kind):
    """The engine (for "serve", with an open session) that the program keeps."""
    if kind not in _engines:
        e = vfb_b200.Engine(mem_limit_bytes=SERVE_BYTES if kind == "serve" else LARGE_BYTES)
        if kind == "serve":
            e.serve_open(slots=SERVE_SLOTS, max_traces=SERVE_TRACES)
        _engines[kind] = e
    return _engines[kind]


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("batch", "serve"):
        probs = _mixed(case, seed)
    elif kind == "large":
        probs = [_large(case, seed)]
    else:
        probs = [_problem(case, seed)]
    eng = None if kind == "noalloc" else _engine("serve" if kind == "serve" else "solve")
    return {"case": case, "probs": probs, "engine": eng, "costs": [int(x) for x in case["costs"].split()]}


# ----------------------------------------------------------------------- pass
def _pack(results):
    n = len(results)
    head = np.zeros((n, 4), np.int64)
    rows = np.zeros((n, vfb_b200.MAX_SIZE), np.int64)
    cands = np.zeros((n, vfb_b200.MAX_SIZE), np.int64)
    rpn = np.zeros((n, vfb_b200.MAX_SIZE), np.int64)
    for i, r in enumerate(results):
        head[i] = (r.status, r.size, r.total_rows, r.solution_index if r.found else -1)
        rows[i, :len(r.level_rows)] = r.level_rows
        cands[i, :len(r.level_cands)] = r.level_cands
        if r.rpn:
            rpn[i, :len(r.rpn)] = [OPS.get(tok, tok) for tok in r.rpn]
    return {"head": head, "rows": rows, "cands": cands, "rpn": rpn}


def run(state):
    case, eng, probs = state["case"], state["engine"], state["probs"]
    kind = case["kind"]
    if kind in ("solve", "large"):
        res = [eng.solve(probs[0])]
    elif kind == "batch":
        res = eng.batch_solve(probs)
    elif kind == "serve":
        res = [None] * len(probs)
        for i, p in enumerate(probs):
            eng.serve_submit(p, i)
        left = len(probs)
        while left:
            for tag, r in eng.serve_step()[0]:
                res[tag] = r
                left -= 1
    elif kind == "costs":
        res = [eng.solve_costs(probs[0], state["costs"], case["neg_type"])]
    elif kind == "bs":
        res = [eng.solve_bs(probs[0], case["bs_max"])]
    elif kind == "exhaustive":
        res = [eng.solve_exhaustive(probs[0])]
    else:
        res = [vfb_b200.solve_noalloc(probs[0])]
    return _pack(res)


def work(case):
    """Bytes and integer operations of one pass: every stored set's words
    written once and read once as an operand, its 16-byte key and 8-byte owner
    written, 16 key bytes read for a candidate; an operator and a
    six-operation key step for each trace of a candidate.  Searches that end
    at a formula are counted to the planted size."""
    t = case["pos"] + case["neg"]
    if case["kind"] == "exhaustive":
        counts = synth.formula_counts(case["aps"], case["max_size"])
        n = sum(counts[k][7] for k in range(1, case["max_size"] + 1))
        # (most formulas fail within the first two traces)
        return {"bytes": 8.0 * case["aps"] * t, "flops": n * 2.0 * case["max_size"]}
    sets, cands = _cands(case)
    if case["kind"] in ("batch", "serve"):
        # half the traces, 2..aps propositions, planted sizes from 5 on
        sets, cands, t = sets * case["count"] / 16, cands * case["count"] / 16, t / 2
    return {"bytes": sets * (16.0 * t + 24.0) + 16.0 * cands, "flops": 7.0 * t * cands}


def exact(case, seed):
    return None   # whole numbers only
