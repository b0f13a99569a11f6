"""The chunk of super-steps that the batch loop launches ahead of reading the
last one's summary: windows do not end by waiting for one in which nothing
runs, and windows that are extended while one is in flight are answered as by
the oracle."""
import ctypes as C

import pytest

import oracle_lib
from journeys import records
from nigiri_b200 import _abi as A
from nigiri_b200 import routing as R
from nigiri_b200.timetable import HostTimetable, QuerySet

pytestmark = pytest.mark.gpu

CHUNK = 4


@pytest.fixture(scope="module")
def city():
    h = HostTimetable.generate(1)
    return h, R.Timetable(h.desc, owner=h)


def windows(h, n, minutes, seed):
    qs = QuerySet(h, 1, n, seed=seed)
    for i in range(n):
        q = qs.arr[i]
        q.direction = i % 2
        q.is_interval, q.interval_from, q.interval_to = 1, q.start_time, q.start_time + minutes
    return qs


def test_few_steps_without_a_running_query(city):
    """An engine without graphs launches nothing ahead.  The other may run one
    chunk more where the chunk in flight ends all start times that are left."""
    h, tt = city
    ahead = R.Engine(tt, max_slots=32, steps_per_sync=CHUNK)
    behind = R.Engine(tt, max_slots=32, steps_per_sync=CHUNK, use_graphs=False)
    qs = windows(h, 24, 60, seed=91)
    out = A.Result()
    extra = []
    for i in range(qs.n):
        steps = []
        for eng in (ahead, behind):
            assert A.lib().b2r_search_batch(eng.handle, C.byref(qs.arr[i]), 1, C.byref(out)) == 0
            steps.append(eng.stats().super_steps)
        extra.append(steps[0] - steps[1])
    assert set(extra) <= {0, CHUNK}, extra
    assert extra.count(CHUNK) <= qs.n // 4, extra


@pytest.mark.parametrize("n", [1, 3, 30])
@pytest.mark.parametrize("transfers", [2, 7])
def test_windows_extended_while_a_chunk_is_in_flight(city, n, transfers):
    h, tt = city
    eng = R.Engine(tt, max_slots=32, steps_per_sync=CHUNK, max_journeys=512)
    qs = windows(h, n, 20, seed=92)
    for i in range(n):
        q = qs.arr[i]
        q.max_transfers, q.min_connection_count = transfers, 12 + i % 5
        q.extend_interval_earlier, q.extend_interval_later = i % 3 != 1, i % 3 != 0
    out = (A.Result * n)()
    assert A.lib().b2r_search_batch(eng.handle, qs.arr, n, out) == 0, A.lib().b2r_last_error()
    for i in range(n):
        o = oracle_lib.OracleResult(h.desc, qs.arr[i])
        got, want = out[i], o.view
        assert (got.status, got.interval_from, got.interval_to, got.n_rounds) == \
            (want.status, want.interval_from, want.interval_to, want.n_rounds), i
        assert records(got) == o.records(), i
