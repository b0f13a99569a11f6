"""Queries that a batch refuses (an invalid one, one beyond a slot's
capacity) get their status whenever their preparation ends relative to the
admission of the others, and are never admitted."""
import ctypes as C

import pytest

from nigiri_b200 import _abi as A
from nigiri_b200 import routing as R
from nigiri_b200.timetable import HostTimetable, QuerySet

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 5, 40])
@pytest.mark.parametrize("refusal", ["invalid", "capacity"])
def test_refused_queries_keep_their_status(n, refusal):
    h = HostTimetable.generate(1)
    eng = R.Engine(R.Timetable(h.desc, owner=h), max_slots=32, max_starts=2, host_threads=4)
    qs = QuerySet(h, 1, n, seed=51)
    for i in range(n):
        q = qs.arr[i]
        if refusal == "invalid":  # pong: no footpaths at the start of a door-to-door query
            q.algorithm, q.start_match_mode, q.use_start_footpaths = A.B2R_ALGO_PONG, A.B2R_MATCH_INTERMODAL, 1
        q.is_interval, q.interval_from, q.interval_to = 1, q.start_time, q.start_time + 360
    out = (A.Result * n)()
    want = []  # a single query is prepared before the loop starts
    for i in range(n):
        assert A.lib().b2r_search_batch(eng.handle, C.byref(qs.arr[i]), 1, out) == 0, A.lib().b2r_last_error()
        want.append(out[0].status)
    assert want.count(A.B2R_ERR_INVALID_ARGUMENT if refusal == "invalid" else A.B2R_ERR_CAPACITY) > n // 2
    for _ in range(400):
        assert A.lib().b2r_search_batch(eng.handle, qs.arr, n, out) == 0, A.lib().b2r_last_error()
        assert [r.status for r in out] == want
