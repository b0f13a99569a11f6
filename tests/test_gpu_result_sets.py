"""Result sets of more than two warps' worth of journeys (pareto_add,
list_recon and next_slot take 32 at a time), collected and rebuilt between
start times; against the oracle."""
import ctypes as C

import pytest

import oracle_lib
from journeys import records
from nigiri_b200 import _abi as A
from nigiri_b200 import routing as R
from nigiri_b200.timetable import HostTimetable, QuerySet

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("call", ["batch", "plain"])
def test_result_sets_above_two_warps(call):
    h = HostTimetable.generate(1)
    eng = R.Engine(R.Timetable(h.desc, owner=h), max_slots=32, max_journeys=512)
    qs = QuerySet(h, 1, 10, seed=7)
    for i in range(qs.n):
        q = qs.arr[i]
        q.direction = i % 2
        q.is_interval, q.interval_from = 1, q.start_time - q.start_time % 1440 + 5 * 60
        q.interval_to = q.interval_from + 1080
    want = [oracle_lib.OracleResult(h.desc, qs.arr[i]) for i in range(qs.n)]
    sizes = [o.view.n_journeys for o in want]
    assert max(sizes) > 96 and any(64 < x <= 96 for x in sizes), sizes
    out = (A.Result * qs.n)()
    if call == "batch":
        assert A.lib().b2r_search_batch(eng.handle, qs.arr, qs.n, out) == 0, A.lib().b2r_last_error()
    for i in range(qs.n):
        if call == "plain":
            assert A.lib().b2r_search_plain(eng.handle, C.byref(qs.arr[i]), C.byref(out[i])) == 0, A.lib().b2r_last_error()
        assert (out[i].status, records(out[i])) == (want[i].view.status, want[i].records()), i
