"""A batch that ends with an error (an interval extension with more start
labels than a slot holds) leaves nothing of its searches behind: the next
batches of the engine are answered as by a new one."""
import pytest

import oracle_lib
from journeys import records
from nigiri_b200 import _abi as A
from nigiri_b200 import routing as R
from nigiri_b200.timetable import HostTimetable, QuerySet

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("transfers", [1, 7])
def test_a_batch_after_one_that_failed(transfers):
    h = HostTimetable.generate(1)
    eng = R.Engine(R.Timetable(h.desc, owner=h), max_slots=32, max_starts=96)
    lib = A.lib()
    # windows that run for dozens of steps, to every tenth stop, and one that
    # wants to grow until its start labels no longer fit
    qs = QuerySet(h, 1, 32, seed=83)
    dest = (A.Offset * 100)()
    for i in range(len(dest)):
        dest[i].target = 9 + 10 * i
    for i in range(qs.n):
        q = qs.arr[i]
        q.direction = i % 2
        q.max_transfers = transfers
        q.is_interval, q.interval_from, q.interval_to = 1, q.start_time, q.start_time + 120
        if i != 21:
            q.destination, q.n_destination = dest, len(dest)
    q = qs.arr[21]
    q.max_transfers, q.interval_to = 0, q.interval_from + 20
    q.min_connection_count, q.extend_interval_earlier, q.extend_interval_later = 3, 1, 1
    out = (A.Result * qs.n)()
    assert lib.b2r_search_batch(eng.handle, qs.arr, qs.n, out) != 0
    nxt = QuerySet(h, 1, 64, seed=84)
    out = (A.Result * nxt.n)()
    assert lib.b2r_search_batch(eng.handle, nxt.arr, nxt.n, out) == 0, lib.b2r_last_error()
    for i in range(nxt.n):
        o = oracle_lib.OracleResult(h.desc, nxt.arr[i])
        assert (out[i].status, records(out[i]), out[i].n_rounds) == (o.view.status, o.records(), o.view.n_rounds), i
