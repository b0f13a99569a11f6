"""hbm_budget bounds what an engine allocates, where the state per route is
large against the state per stop."""
import ctypes as C

import numpy as np
import pytest
import torch

from nigiri_b200 import _abi as A
from nigiri_b200 import routing as R

pytestmark = pytest.mark.gpu

DAY0 = 19723


class Shuttles:
    """n_routes lines of two stops over 64 stops, one trip each."""

    def __init__(self, n_routes):
        n_loc = 9 + 64
        a = 9 + np.arange(n_routes) % 64
        b = 9 + (np.arange(n_routes) + 1 + np.arange(n_routes) // 64 % 63) % 64
        t = (6 * 60 + np.arange(n_routes) % 700).astype(np.uint16)
        self.keep = {
            "tt": np.array([0] * 9 + [2] * 64, np.uint8), "fi": np.zeros(n_loc + 1, np.uint32),
            "fp": np.zeros(1, np.uint32), "ri": 2 * np.arange(n_routes + 1, dtype=np.uint32),
            "rs": (np.stack([a, b], 1).reshape(-1) | 0xF << 28).astype(np.uint32),
            "nt": np.ones(n_routes, np.uint32), "st": np.stack([t << 5, (t + 9) << 5], 1).reshape(-1),
            "bf": np.ones(n_routes, np.uint32),
            "days": np.array([[0] * 8, [((1 << 20) - 1) << 5] + [0] * 7], np.uint64)}
        x = A.TtBase()
        ptr = lambda k, ty: self.keep[k].ctypes.data_as(C.POINTER(ty))  # noqa: E731
        x.n_locations, x.date_range_from, x.date_range_to = n_loc, DAY0, DAY0 + 20
        x.transfer_time = ptr("tt", C.c_uint8)
        x.footpaths_out_index, x.footpaths_out = ptr("fi", C.c_uint32), ptr("fp", C.c_uint32)
        x.n_routes, x.route_stop_index, x.route_stops = n_routes, ptr("ri", C.c_uint32), ptr("rs", C.c_uint32)
        x.route_n_transports, x.route_stop_times = ptr("nt", C.c_uint32), ptr("st", C.c_uint16)
        x.transport_bitfield, x.n_bitfields, x.bitfields = ptr("bf", C.c_uint32), 2, ptr("days", C.c_uint64)
        self.handle = C.c_void_p()
        assert A.lib().b2r_tt_build(C.byref(x), C.byref(self.handle)) == 0, A.lib().b2r_last_error()
        self.desc = A.TimetableDesc()
        assert A.lib().b2r_tt_desc(self.handle, C.byref(self.desc)) == 0


@pytest.mark.parametrize("max_journeys", [32, 256])
def test_engine_stays_within_its_budget(max_journeys):
    s = Shuttles(20000)
    tt = R.Timetable(s.desc, owner=s)
    torch.cuda.init()
    R.Engine(tt, max_slots=32, use_lower_bounds=False).close()  # what the first engine of a process takes
    budget = 2 << 30
    free = torch.cuda.mem_get_info()[0]
    eng = R.Engine(tt, max_slots=65536, hbm_budget=budget, max_journeys=max_journeys, max_starts=32,
                   use_lower_bounds=False)
    used = free - torch.cuda.mem_get_info()[0]
    assert eng.slots % 32 == 0 and eng.slots * eng.bytes_per_slot() <= budget < (eng.slots + 32) * eng.bytes_per_slot()
    # about fifty arrays, each rounded up to the allocator's 2 MiB
    assert used <= budget + 50 * (2 << 20), used
    assert used > 0.9 * budget, used
