"""Several engines of one process on a device that is nearly full: what an idle
engine keeps cached from earlier calls is there for the others."""
import threading

import pytest

import vfb_b200
from tests import cases

pytestmark = pytest.mark.gpu
GB = 1 << 30


def _key(r):
    return (r.status, r.size, r.rpn, r.level_rows, r.level_cands, r.solution_index)


@pytest.fixture(scope="module")
def problems():
    """A search that holds about 6.5 GB at its peak, and a small one."""
    big = cases.random_instance(4711, 6, 24, 25, 32, 9)
    big.neg[0] = big.pos[0]
    return (vfb_b200.Problem.from_instance(big),
            vfb_b200.Problem.from_instance(cases.small_exact_cases()[0]))


@pytest.fixture(scope="module")
def nearly_full(problems):
    """All of the device but 9.5 GB taken: room for one big search, not for one
    and another engine's cache."""
    torch = pytest.importorskip("torch")
    with vfb_b200.Engine(mem_limit_bytes=64 * GB) as eng:
        want = [_key(eng.solve(p)) for p in problems]
    # (the engine's end gave the pool's spare memory back)
    free, _ = torch.cuda.mem_get_info()
    filler = torch.empty(free - 19 * GB // 2, dtype=torch.uint8, device="cuda")
    yield want
    del filler
    torch.cuda.empty_cache()


def test_an_idle_engines_cache_is_given_back(problems, nearly_full):
    with vfb_b200.Engine(mem_limit_bytes=64 * GB) as first, vfb_b200.Engine(mem_limit_bytes=64 * GB) as second:
        for eng in (first, second, first):
            # the big call's blocks stay cached through the small one
            assert [_key(eng.solve(p)) for p in problems] == nearly_full


def test_a_session_opens_beside_an_idle_engine(problems, nearly_full):
    with vfb_b200.Engine(mem_limit_bytes=64 * GB) as first, vfb_b200.Engine(mem_limit_bytes=8 * GB) as second:
        assert [_key(first.solve(p)) for p in problems] == nearly_full
        second.serve_limits(1.0, 8 * GB, 0)
        second.serve_open(2, 64)
        try:
            second.serve_submit(problems[0], 0)
            got = []
            while not got:
                got, _, _ = second.serve_step()
        finally:
            second.serve_close()
        assert _key(got[0][1]) == nearly_full[0]


def test_engines_in_threads(problems, nearly_full):
    """Two threads whose searches do not fit side by side: every call ends with
    the stored search or, without the room, the one tested on the fly."""
    got, errors = [], []

    def work():
        try:
            with vfb_b200.Engine(mem_limit_bytes=64 * GB) as eng:
                for _ in range(4):
                    got.append((_key(eng.solve(problems[0])), _key(eng.solve(problems[1]))))
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=work) for _ in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors and len(got) == 8
    for big, small in got:
        assert small == nearly_full[1]
        assert big == nearly_full[0] or big[0] in (vfb_b200.LIMIT, vfb_b200.OOM)
