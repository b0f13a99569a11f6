"""The route scan at the edges of its 32-stop blocks, 8-lane and whole-warp
tiles: routes of 2 to 100 stops on a built timetable, sections that lack a
required flag, routes whose trips keep no one trip order (the sequential walk),
several transports' traffic days in one route, dense marks (one-to-all from
many starts), both directions; against the oracle, batched (few and many
queries: both tile widths) and without allocation."""
import ctypes as C
import random

import numpy as np
import pytest

import oracle_lib
from nigiri_b200 import _abi as A
from nigiri_b200 import routing as R

pytestmark = pytest.mark.gpu

N_STOPS = 300
LENGTHS = (2, 3, 8, 31, 32, 33, 40, 63, 64, 65, 100)
DAY0 = 19723


def flat(rows, dtype):
    return np.array([x for r in rows for x in r], dtype)


class Built:
    """A random timetable (seeded): in every third route the trips are held to
    the full hour somewhere, so that some meet there (no one order); every
    fourth mixes two traffic-day sets."""

    def __init__(self, n_routes, seed):
        rnd = random.Random(seed)
        n_loc = N_STOPS + 9
        days = [0, (1 << 20) - 1, 0b1011011101 << 3]  # none, all, some
        stops, n_t, times, bf, flags = [], [], [], [], []
        for r in range(n_routes):
            n = LENGTHS[r % len(LENGTHS)]
            seq = rnd.sample(range(9, n_loc), n)
            k = rnd.choice((1, 2, 5, 33))
            hops = [rnd.randint(1, 4) for _ in range(2 * (n - 1))]
            first = sorted(rnd.sample(range(5 * 60, 19 * 60, 7), k))
            hold = rnd.randrange(1, len(hops) + 1) if r % 3 == 0 else -1
            trips = []
            for t0 in first:
                t, ev = t0, []
                for x, h in enumerate(hops):
                    if x == hold:
                        t = -(-t // 60) * 60
                    ev.append(t)
                    t += h
                trips.append(ev)
            # per event the trips' days and minutes
            times.append([(t // 1440) | ((t % 1440) << 5) for x in range(2 * (n - 1)) for t in (tr[x] for tr in trips)])
            stops.append([s | (1 << 28) * (rnd.random() < 0.95) | (1 << 29) * (rnd.random() < 0.95) | 3 << 30 for s in seq])
            n_t.append(k)
            bf += [rnd.choice((1, 2)) if r % 4 == 0 else 1 for _ in range(k)]
            flags.append([rnd.choice((0b1111, 0b1111, 0b1110)) for _ in range(n)])
        fp = [[] for _ in range(n_loc)]
        for _ in range(N_STOPS):
            a, b = rnd.sample(range(9, n_loc), 2)
            fp[a].append(b | rnd.randint(2, 9) << 23)
        idx = np.concatenate([[0], np.cumsum([len(x) for x in fp])]).astype(np.uint32)
        keep = self.keep = {
            "tt": np.array([0] * 9 + [2] * N_STOPS, np.uint8), "fi": idx, "fp": flat(fp, np.uint32),
            "ri": np.concatenate([[0], np.cumsum([len(x) for x in stops])]).astype(np.uint32),
            "rs": flat(stops, np.uint32), "nt": np.array(n_t, np.uint32), "st": flat(times, np.uint16),
            "bf": np.array(bf, np.uint32), "sf": flat(flags, np.uint8),
            "days": np.array([[d << 5, 0, 0, 0, 0, 0, 0, 0] for d in days], np.uint64)}
        b = A.TtBase()
        ptr = lambda k, t: keep[k].ctypes.data_as(C.POINTER(t))  # noqa: E731
        b.n_locations, b.date_range_from, b.date_range_to = n_loc, DAY0, DAY0 + 20
        b.transfer_time, b.footpaths_out_index, b.footpaths_out = (ptr("tt", C.c_uint8), ptr("fi", C.c_uint32),
                                                                   ptr("fp", C.c_uint32))
        b.n_routes, b.route_stop_index, b.route_stops = n_routes, ptr("ri", C.c_uint32), ptr("rs", C.c_uint32)
        b.route_n_transports, b.route_stop_times = ptr("nt", C.c_uint32), ptr("st", C.c_uint16)
        b.transport_bitfield, b.n_bitfields, b.bitfields = ptr("bf", C.c_uint32), len(days), ptr("days", C.c_uint64)
        rf = []  # bikes: on all sections, or on some
        for f in flags:
            on = [x & 1 for x in f[:-1]]
            rf.append((0b01 if all(on) else 0b10 if any(on) else 0) | 0b010100)
        keep["rf"] = np.array(rf, np.uint8)
        b.route_flags, b.route_section_flags = ptr("rf", C.c_uint8), ptr("sf", C.c_uint8)
        self.handle = C.c_void_p()
        assert A.lib().b2r_tt_build(C.byref(b), C.byref(self.handle)) == 0, A.lib().b2r_last_error()
        self.desc = A.TimetableDesc()
        assert A.lib().b2r_tt_desc(self.handle, C.byref(self.desc)) == 0


def queries(n, n_start, kind, bikes, seed):
    rnd = random.Random(seed)
    arr, keep = (A.Query * n)(), []
    for i in range(n):
        q = arr[i]
        A.lib().b2r_query_init(C.byref(q))
        st, de = (A.Offset * n_start)(), (A.Offset * 1)()
        for o, l in zip(st, rnd.sample(range(9, 9 + N_STOPS), n_start)):
            o.target, o.duration = l, 0
        de[0].target = rnd.randrange(9, 9 + N_STOPS)
        keep += [st, de]
        q.kind, q.direction, q.start, q.n_start = kind, i % 2, st, n_start
        if kind == A.B2R_ONE_TO_ONE:
            q.destination, q.n_destination = de, 1
        q.start_time = (DAY0 + 4 + i % 9) * 1440 + rnd.randint(6 * 60, 20 * 60)
        q.require_bike_transport = bikes and i % 3 != 0
    return arr, keep


def check(desc, arr, n, out):
    want = oracle_lib.answers(desc, arr, range(n))
    from journeys import records
    reached = 0
    for i in range(n):
        if arr[i].kind == A.B2R_ONE_TO_ALL:
            r = out[i]
            got = np.ctypeslib.as_array(r.round_times, shape=(r.n_rows * desc.n_locations,)).reshape(r.n_rows, -1)
            assert np.array_equal(got, want[i][2][:r.n_rows]), i
            reached += int((np.abs(got.astype(int)) < 32767).sum())
        else:
            assert records(out[i]) == want[i][1], i
            reached += out[i].n_journeys
    assert reached > n


@pytest.mark.parametrize("kind", [A.B2R_ONE_TO_ONE, A.B2R_ONE_TO_ALL])
@pytest.mark.parametrize("bikes", [False, True])
@pytest.mark.parametrize("n,n_start,n_routes", [(6, 1, 66), (33, 40, 66), (640, 30, 1100)])
def test_scan_matches_oracle(n, n_start, n_routes, bikes, kind):
    b = Built(n_routes, seed=n + n_routes)
    eng = R.Engine(R.Timetable(b.desc, owner=b), max_slots=min(1024, (n + 31) // 32 * 32))
    arr, keep = queries(n, n_start, kind, bikes, seed=3)
    out = (A.Result * n)()
    assert A.lib().b2r_search_batch(eng.handle, arr, n, out) == 0, A.lib().b2r_last_error()
    check(b.desc, arr, n, out)


@pytest.mark.parametrize("bikes", [False, True])
def test_noalloc_scan_matches_oracle(bikes):
    b = Built(132, seed=9)
    tt = R.Timetable(b.desc, owner=b)
    arr, keep = queries(12, 40, A.B2R_ONE_TO_ALL, bikes, seed=4)
    want = oracle_lib.answers(b.desc, arr, range(12))
    for i in range(12):
        rows, n_rows, day = np.empty((A.B2R_K, b.desc.n_locations), np.int16), C.c_uint32(), C.c_int32()
        assert A.lib().b2r_one_to_all_noalloc(tt.handle, C.byref(arr[i]), rows.ctypes.data_as(C.POINTER(C.c_int16)),
                                              rows.size, C.byref(n_rows), C.byref(day), None) == 0
        got = rows.reshape(-1)[:n_rows.value * b.desc.n_locations].reshape(n_rows.value, -1)
        assert np.array_equal(got, want[i][2][:n_rows.value]), i
