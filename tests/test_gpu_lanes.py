"""The super-step's warp-per-slot passes where their lanes wrap: start labels,
destinations and result sets around 32 and 64, in both directions, against the
oracle (complete journey records)."""
import pytest

import oracle_lib
from journeys import records
from nigiri_b200 import _abi as A
from nigiri_b200 import routing as R
from nigiri_b200.timetable import HostTimetable, QuerySet

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def city():
    h = HostTimetable.generate(1)
    return h, R.Engine(R.Timetable(h.desc, owner=h), max_slots=32)


def offsets(h, first, n, step, duration):
    """n stops from `first` on, `step` apart, reached in 0.. minutes."""
    out = (A.Offset * n)()
    stops = h.desc.n_locations - 9
    for i in range(n):
        out[i].target = 9 + (first + i * step) % stops
        out[i].duration = i % 7 if duration else 0
    return out


@pytest.mark.parametrize("window", [0, 45])
@pytest.mark.parametrize("mode", [A.B2R_MATCH_EXACT, A.B2R_MATCH_INTERMODAL])
@pytest.mark.parametrize("n_start,n_dest", [(1, 1), (31, 1), (32, 2), (33, 31), (64, 32), (40, 33), (2, 40)])
def test_starts_and_destinations_around_a_warp(city, n_start, n_dest, mode, window):
    h, eng = city
    qs = QuerySet(h, 1, 12, seed=7 * n_start + n_dest)
    keep = []
    for i in range(qs.n):
        q = qs.arr[i]
        st = offsets(h, 31 * i, n_start, 1, mode == A.B2R_MATCH_INTERMODAL)
        de = offsets(h, 500 + 17 * i, n_dest, 11, mode == A.B2R_MATCH_INTERMODAL)
        keep += [st, de]
        q.start, q.n_start, q.destination, q.n_destination = st, n_start, de, n_dest
        q.start_match_mode = q.dest_match_mode = mode
        q.direction = i % 2
        q.use_start_footpaths = i % 3 == 0
        if window:
            q.is_interval, q.interval_from, q.interval_to = 1, q.start_time, q.start_time + window
    out = (A.Result * qs.n)()
    assert A.lib().b2r_search_batch(eng.handle, qs.arr, qs.n, out) == 0, A.lib().b2r_last_error()
    found = 0
    for i in range(qs.n):
        r = oracle_lib.OracleResult(h.desc, qs.arr[i])
        assert out[i].status == r.view.status, i
        assert records(out[i]) == records(r.view), i
        found += out[i].n_journeys
    assert found > 0


def test_result_sets_above_a_warp(city):
    """Eight-hour windows: more than 32 and more than 64 Pareto journeys."""
    h, eng = city
    qs = QuerySet(h, 1, 8, seed=5)
    for i in range(qs.n):
        q = qs.arr[i]
        q.direction = i % 2
        q.is_interval, q.interval_from = 1, q.start_time - q.start_time % 1440 + 7 * 60
        q.interval_to = q.interval_from + 480
    out = (A.Result * qs.n)()
    assert A.lib().b2r_search_batch(eng.handle, qs.arr, qs.n, out) == 0, A.lib().b2r_last_error()
    for i in range(qs.n):
        r = oracle_lib.OracleResult(h.desc, qs.arr[i])
        assert out[i].status == r.view.status, i
        assert records(out[i]) == records(r.view), i
    most = max(out[i].n_journeys for i in range(qs.n))
    assert most > 32, most
