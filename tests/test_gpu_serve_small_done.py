"""Serving steps whose done[] holds fewer results than a step has: every request
is reported once, in some step, refused ones (too many traces for the session,
a bad rule) among finished ones."""
import ctypes

import pytest

import vfb_b200
from tests import cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cap", [1, 3])
def test_no_request_is_lost(cap):
    fine = [vfb_b200.Problem.from_instance(i) for i in cases.small_exact_cases()[:4]]
    wide = vfb_b200.Problem.from_instance(cases.random_instance(3, 2, 20, 20, 8, 4))
    odd = vfb_b200.Problem.from_instance(cases.random_instance(4, 2, 2, 2, 8, 4))
    odd.rlx_type = 9
    probs = [wide, fine[0], odd, wide, wide, fine[1], odd, fine[2], wide, fine[3], wide, odd]
    with vfb_b200.Engine(mem_limit_bytes=4 << 30) as eng:
        want = [vfb_b200.LIMIT if p is wide else vfb_b200.BAD_INPUT if p is odd else eng.solve(p).status for p in probs]
        eng.serve_open(4, 16)
        try:
            for i, p in enumerate(probs):
                eng.serve_submit(p, i)
            done = (vfb_b200._Served * cap)()
            nd, act, q = ctypes.c_int(), ctypes.c_int(), ctypes.c_int()
            got = {}
            for _ in range(400):
                rc = eng._lib.vfb_serve_step(eng._ctx, done, cap, ctypes.byref(nd), ctypes.byref(act), ctypes.byref(q))
                assert rc == vfb_b200.OK and 0 <= nd.value <= cap
                for j in range(nd.value):
                    assert done[j].tag not in got
                    got[done[j].tag] = done[j].result.status
                if act.value == 0 and q.value == 0:
                    break
        finally:
            eng.serve_close()
    assert got == dict(enumerate(want))
