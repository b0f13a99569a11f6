"""Searches whose last round still reaches stations: few transfers, windows
from several start stops, interval extension, one search after the other in
the same slot.  raptor::next_start_time clears the station marks
(raptor.h:179-188), so no search may start on the marks that the one before
left; against the oracle, round counts included, by every call that runs
searches."""
import ctypes as C

import pytest

import oracle_lib
from journeys import records
from nigiri_b200 import _abi as A
from nigiri_b200 import routing as R
from nigiri_b200.timetable import HostTimetable, QuerySet
from test_algo_adapter import helper

pytestmark = pytest.mark.gpu

N = {1: 48, 2: 24}
CASES = [(1, 0, 0, False), (1, 120, 0, False), (1, 120, 1, False), (1, 120, 2, False), (1, 120, 3, False),
         (1, 60, 1, True), (1, 60, 2, True), (2, 120, 1, False), (2, 120, 2, False), (2, 60, 1, True)]


@pytest.fixture(scope="module")
def timetables():
    out = {}
    for workload in N:
        h = HostTimetable.generate(workload)
        out[workload] = (h, R.Timetable(h.desc, owner=h))
    return out


def queries(h, workload, window, transfers, extend):
    qs = QuerySet(h, workload, N[workload], seed=71)
    keep = []
    for i in range(qs.n):
        q = qs.arr[i]
        q.direction = i % 2
        q.max_transfers = transfers
        if workload == 1:  # a city's stream leaves from one stop: six of them, walks of 0 to 5 minutes
            st = (A.Offset * 6)()
            for j in range(6):
                st[j].target = 9 + (q.start[0].target - 9 + j) % (h.desc.n_locations - 9)
                st[j].duration = j
            keep.append(st)
            q.start, q.n_start, q.start_match_mode = st, 6, A.B2R_MATCH_INTERMODAL
        if window:
            q.is_interval, q.interval_from, q.interval_to = 1, q.start_time, q.start_time + window
        if extend:
            q.min_connection_count = 8
            q.extend_interval_earlier = q.extend_interval_later = 1
    return qs, keep


def answer(r):
    return r.status, records(r), r.interval_from, r.interval_to, r.n_rounds


@pytest.mark.parametrize("workload,window,transfers,extend", CASES)
@pytest.mark.parametrize("call", ["batch", "plain", "served"])
def test_searches_that_end_with_their_last_round(timetables, call, workload, window, transfers, extend):
    h, tt = timetables[workload]
    lib = A.lib()
    eng = R.Engine(tt, max_slots=32, max_journeys=512)
    qs, keep = queries(h, workload, window, transfers, extend)
    out = (A.Result * qs.n)()
    if call == "batch":
        assert lib.b2r_search_batch(eng.handle, qs.arr, qs.n, out) == 0, lib.b2r_last_error()
        got = [answer(r) for r in out]
    elif call == "plain":
        got = []
        for i in range(qs.n):
            assert lib.b2r_search_plain(eng.handle, C.byref(qs.arr[i]), C.byref(out[0])) == 0, i
            got.append(answer(out[0]))
    else:
        srv = R.Server(eng)
        got = [answer(srv.wait(t)) for t in [srv.submit_raw(q) for q in qs.arr[:qs.n]]]
        srv.stop()
    found = 0
    for i in range(qs.n):
        r = oracle_lib.OracleResult(h.desc, qs.arr[i])
        assert got[i] == answer(r.view), i
        found += r.view.n_journeys
    assert found > 0 or transfers == 0
    if call != "batch":  # nothing is left for the next batch to fail for
        assert lib.b2r_search_batch(eng.handle, qs.arr, 1, out) == 0, lib.b2r_last_error()


@pytest.mark.parametrize("workload,window,transfers,extend", [c for c in CASES if c[1]])
def test_step_driven_searches_that_end_with_their_last_round(timetables, tmp_path, workload, window, transfers,
                                                             extend):
    h, tt = timetables[workload]
    run = helper(str(tmp_path)).algo_search
    qs, keep = queries(h, workload, window, transfers, extend)
    for i in range(qs.n):
        got = A.Result()
        assert run(tt.handle, C.byref(h.desc), C.byref(qs.arr[i]), C.byref(got)) == 0, i
        r = oracle_lib.OracleResult(h.desc, qs.arr[i])
        assert answer(got)[:4] == answer(r.view)[:4], i
