"""Several footpaths between the same two stops, into a destination: the
shortest decides, wherever it stands in the lists; against the oracle."""
import ctypes as C

import numpy as np
import pytest

import oracle_lib
from journeys import records
from nigiri_b200 import _abi as A
from nigiri_b200 import routing as R

pytestmark = pytest.mark.gpu

DAY0 = 19723
START, MID, HUB = 9, 10, 11


class Line:
    """START to MID in ten minutes, then footpaths of the given durations from
    MID to HUB."""

    def __init__(self, walks):
        first = [7 * 60 + 30 * t for t in range(4)]
        self.keep = {
            "tt": np.array([0] * 9 + [2] * 3, np.uint8),
            "fi": np.array([0] * 11 + [len(walks)] * 2, np.uint32),
            "fp": np.array([HUB | w << 23 for w in walks], np.uint32),
            "ri": np.array([0, 2], np.uint32), "rs": np.array([START | 0xF << 28, MID | 0xF << 28], np.uint32),
            "nt": np.array([4], np.uint32), "st": np.array([(t + x) << 5 for x in (0, 10) for t in first], np.uint16),
            "bf": np.ones(4, np.uint32), "days": np.array([[0] * 8, [((1 << 20) - 1) << 5] + [0] * 7], np.uint64)}
        b = A.TtBase()
        ptr = lambda k, t: self.keep[k].ctypes.data_as(C.POINTER(t))  # noqa: E731
        b.n_locations, b.date_range_from, b.date_range_to = 12, DAY0, DAY0 + 20
        b.transfer_time = ptr("tt", C.c_uint8)
        b.footpaths_out_index, b.footpaths_out = ptr("fi", C.c_uint32), ptr("fp", C.c_uint32)
        b.n_routes, b.route_stop_index, b.route_stops = 1, ptr("ri", C.c_uint32), ptr("rs", C.c_uint32)
        b.route_n_transports, b.route_stop_times = ptr("nt", C.c_uint32), ptr("st", C.c_uint16)
        b.transport_bitfield, b.n_bitfields, b.bitfields = ptr("bf", C.c_uint32), 2, ptr("days", C.c_uint64)
        self.handle = C.c_void_p()
        assert A.lib().b2r_tt_build(C.byref(b), C.byref(self.handle)) == 0, A.lib().b2r_last_error()
        self.desc = A.TimetableDesc()
        assert A.lib().b2r_tt_desc(self.handle, C.byref(self.desc)) == 0


@pytest.mark.parametrize("walks", [(5,), (5, 3), (3, 5), (9, 9, 4, 12), (4, 4)])
@pytest.mark.parametrize("direction", [A.B2R_FORWARD, A.B2R_BACKWARD])
def test_shortest_of_parallel_footpaths(walks, direction):
    line = Line(walks)
    eng = R.Engine(R.Timetable(line.desc, owner=line), max_slots=32)
    q = A.Query()
    A.lib().b2r_query_init(C.byref(q))
    st, de = (A.Offset * 1)(), (A.Offset * 1)()
    st[0].target, de[0].target = (START, HUB) if direction == A.B2R_FORWARD else (HUB, START)
    q.start, q.n_start, q.destination, q.n_destination, q.direction = st, 1, de, 1, direction
    q.use_start_footpaths = 1
    q.is_interval, q.interval_from = 1, (DAY0 + 7) * 1440 + 7 * 60
    q.interval_to = q.interval_from + 90
    out = A.Result()
    assert A.lib().b2r_search_batch(eng.handle, C.byref(q), 1, C.byref(out)) == 0, A.lib().b2r_last_error()
    o = oracle_lib.OracleResult(line.desc, q)
    assert records(out) == o.records() and o.view.n_journeys > 0
    assert out.n_rounds == o.view.n_rounds
