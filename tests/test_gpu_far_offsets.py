"""Destination offsets around and beyond the travel-time limit, which bound
their own stop and nothing around it: the same journeys with lower bounds from
the all-pairs tables, from the solver on the device, from the host's Dijkstra,
and without any."""
import pytest

from journeys import records
from nigiri_b200 import _abi as A
from nigiri_b200 import routing as R
from nigiri_b200.timetable import HostTimetable, QuerySet

pytestmark = pytest.mark.gpu

FAR = [7199, 7200, 7201, 7300, 32000, 32767]


@pytest.fixture(scope="module")
def city():
    h = HostTimetable.generate(1)
    return h, R.Timetable(h.desc, owner=h)


def run(tt, qs, lower_bounds):
    eng = R.Engine(tt, max_slots=64, use_lower_bounds=lower_bounds)
    out = (A.Result * qs.n)()
    assert A.lib().b2r_search_batch(eng.handle, qs.arr, qs.n, out) == 0, A.lib().b2r_last_error()
    return [(r.status, records(r)) for r in out]


@pytest.mark.parametrize("lower_bounds", ["table", "device", "host"])
@pytest.mark.parametrize("window", [0, 60])
def test_bounds_of_far_destinations(city, lower_bounds, window):
    h, tt = city
    qs = QuerySet(h, 1, 64, seed=17)
    keep = []
    for i in range(qs.n):
        q = qs.arr[i]
        q.direction = i % 2
        far = FAR[:1 + i % len(FAR)]
        near = i % 4 != 0  # every fourth has none within the limit of its travel time
        de = (A.Offset * (len(far) + near))()
        for j, d in enumerate(far + [3] * near):
            de[j].target, de[j].duration = 9 + (q.destination[0].target - 9 + 5 * j) % (h.desc.n_locations - 9), d
        keep.append(de)
        q.destination, q.n_destination, q.dest_match_mode = de, len(de), A.B2R_MATCH_INTERMODAL
        q.max_travel_time = 7200
        if window:
            q.is_interval, q.interval_from, q.interval_to = 1, q.start_time, q.start_time + window
    want = run(tt, qs, False)
    assert run(tt, qs, lower_bounds) == want
    assert any(r for _, r in want)
