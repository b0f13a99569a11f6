"""A query that a kernel fails (more footpaths into its destination reached in
one round than the kernel has room for: 64) reports it by every call that runs
queries; the queries beside it, and those run in its slot afterwards, have
their answers."""
import ctypes as C

import numpy as np
import pytest

import oracle_lib
from journeys import records
from nigiri_b200 import _abi as A
from nigiri_b200 import routing as R
from test_algo_adapter import helper

pytestmark = pytest.mark.gpu

DAY0 = 19723
START, HUB, FIRST = 9, 10, 11  # the line's first stop, the walks' target, the line's other stops


class Line:
    """One line whose trips call at START and then at n stops, a minute apart;
    every stop has a footpath to HUB."""

    def __init__(self, n):
        n_loc, n_trips = FIRST + n, 4
        days = np.array([[0] * 8, [((1 << 20) - 1) << 5] + [0] * 7], np.uint64)
        first = [7 * 60 + 30 * t for t in range(n_trips)]
        self.keep = {
            "tt": np.array([0] * 9 + [2] * (n_loc - 9), np.uint8),
            "fi": np.concatenate([np.zeros(FIRST + 1), np.arange(1, n + 1)]).astype(np.uint32),
            "fp": np.full(n, HUB | 5 << 23, np.uint32),
            "ri": np.array([0, n + 1], np.uint32),
            "rs": np.array([s | 0xF << 28 for s in [START, *range(FIRST, n_loc)]], np.uint32),
            "nt": np.array([n_trips], np.uint32),
            "st": np.array([(t + x) << 5 for x in range(2 * n) for t in first], np.uint16),
            "bf": np.ones(n_trips, np.uint32), "days": days}
        b = A.TtBase()
        ptr = lambda k, t: self.keep[k].ctypes.data_as(C.POINTER(t))  # noqa: E731
        b.n_locations, b.date_range_from, b.date_range_to = n_loc, DAY0, DAY0 + 20
        b.transfer_time = ptr("tt", C.c_uint8)
        b.footpaths_out_index, b.footpaths_out = ptr("fi", C.c_uint32), ptr("fp", C.c_uint32)
        b.n_routes, b.route_stop_index, b.route_stops = 1, ptr("ri", C.c_uint32), ptr("rs", C.c_uint32)
        b.route_n_transports, b.route_stop_times = ptr("nt", C.c_uint32), ptr("st", C.c_uint16)
        b.transport_bitfield, b.n_bitfields, b.bitfields = ptr("bf", C.c_uint32), 2, ptr("days", C.c_uint64)
        self.handle = C.c_void_p()
        assert A.lib().b2r_tt_build(C.byref(b), C.byref(self.handle)) == 0, A.lib().b2r_last_error()
        self.desc = A.TimetableDesc()
        assert A.lib().b2r_tt_desc(self.handle, C.byref(self.desc)) == 0


def queries(destinations):
    """From START to one destination each, a window of two trips."""
    arr, keep = (A.Query * len(destinations))(), []
    for q, d in zip(arr, destinations):
        A.lib().b2r_query_init(C.byref(q))
        st, de = (A.Offset * 1)(), (A.Offset * 1)()
        st[0].target, de[0].target = START, d
        keep += [st, de]
        q.start, q.n_start, q.destination, q.n_destination = st, 1, de, 1
        q.is_interval, q.interval_from = 1, (DAY0 + 7) * 1440 + 7 * 60
        q.interval_to = q.interval_from + 45
    return arr, keep


@pytest.mark.parametrize("n", [63, 64, 65, 90])
@pytest.mark.parametrize("call", ["batch", "plain", "served", "step-driven"])
def test_a_failed_query_says_so_and_fails_alone(tmp_path, call, n):
    line = Line(n)
    tt = R.Timetable(line.desc, owner=line)
    eng = R.Engine(tt, max_slots=32)
    lib = A.lib()
    arr, keep = queries([FIRST + 3, HUB, FIRST + n - 1, FIRST + 7])
    want_rc = A.B2R_ERR_DEVICE_STATUS if n > 64 else 0
    out = (A.Result * len(arr))()
    status, got, rc = [], [], 0
    if call == "batch":
        rc = lib.b2r_search_batch(eng.handle, arr, len(arr), out)
        status, got = [r.status for r in out], [records(r) for r in out]
    elif call == "served":
        srv = R.Server(eng)
        res = [srv.wait(t) for t in [srv.submit_raw(q) for q in arr]]
        status, got, rc = [r.status for r in res], [records(r) for r in res], want_rc
        srv.stop()
    else:
        run = helper(str(tmp_path)).algo_search
        for i in range(len(arr)):
            if call == "plain":
                x = lib.b2r_search_plain(eng.handle, C.byref(arr[i]), C.byref(out[i]))
                assert x == out[i].status, i
            else:
                x = run(tt.handle, C.byref(line.desc), C.byref(arr[i]), C.byref(out[i]))
            rc = rc or x
            status.append(x)
            got.append(records(out[i]) if x == 0 else [])
    assert rc == want_rc
    assert status == [0, want_rc, 0, 0]
    for i in range(len(arr)):
        if status[i] == 0:
            want = oracle_lib.OracleResult(line.desc, arr[i]).records()
            assert got[i] == want and want, i
    # the slots are as good as new
    arr, keep = queries([FIRST + (5 * i) % n for i in range(40)])
    out = (A.Result * len(arr))()
    assert lib.b2r_search_batch(eng.handle, arr, len(arr), out) == 0, lib.b2r_last_error()
    for i in range(len(arr)):
        o = oracle_lib.OracleResult(line.desc, arr[i])
        assert (records(out[i]), out[i].n_rounds) == (o.records(), o.view.n_rounds), i
