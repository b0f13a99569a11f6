"""Measured workloads of the routing engine: what a program that embeds it
asks of it, through the public entry points (include/b2r.h by way of
nigiri_b200).

The three timetables are the repository's own seeded ones: a city (1,009
stops), a region (40,009 stops) and a country (300,009 stops).  A program
uploads its timetable and creates its engine once and keeps both, so these are
made once per process here too; a state holds one set of requests.

Requests are what the host hands over and journeys are what it gets back, so
states and outputs live in host memory; every pass takes them through the
whole call.  All outputs are whole numbers.
"""
import ctypes as C
import math

import numpy as np
import torch

from nigiri_b200 import _abi as A
from nigiri_b200 import routing as R
from nigiri_b200.timetable import HostTimetable, QuerySet

# timetable and request stream of each scale (the workload numbers of
# b2r_tt_generate / b2r_queries_generate)
TIMETABLE = {"city": 1, "regional": 2, "national": 4}
ONTRIP = {"city": 1, "regional": 2, "national": 4}
RANGE = 3
MIX = 4

RESULT = np.dtype([("status", "i4"), ("n_journeys", "u4"), ("journeys", "u8"), ("legs", "u8"),
                   ("interval_from", "i4"), ("interval_to", "i4"), ("n_rows", "u4"), ("base_day", "i4"),
                   ("round_times", "u8"), ("n_rounds", "u8"), ("n_start_times", "u8"), ("latency_ms", "f8")])
JOURNEY = np.dtype([("start_time", "i4"), ("dest_time", "i4"), ("dest", "u4"), ("transfers", "u1"), ("error", "u1"),
                    ("n_legs", "u2"), ("first_leg", "u4")])
assert RESULT.itemsize == C.sizeof(A.Result) and JOURNEY.itemsize == C.sizeof(A.Journey)
# values that answers hold: journeys per request (plus a few for small batches) and legs per journey; one start
# time gives a journey per useful number of transfers, a window of up to four hours some dozens
JOURNEYS = {"ontrip": 8, "mix": 24, "range": 96, "pong": 96, "one_to_all": 0}
LEGS = 6


def case(name, scale, kind, n, call="batch", direction="fwd", option="none", window=0):
    """scale: which timetable.  kind: ontrip (leave at a time), range (leave
    within a window of minutes), pong (the same by alternating searches),
    one_to_all, mix (70% ontrip, 20% one-hour range, 10% one-to-all).  n:
    requests.  call: batch (b2r_search_batch), plain (b2r_search_plain, one
    after the other), noalloc (b2r_one_to_all_noalloc, likewise), serve
    (b2r_submit / b2r_wait).  direction: fwd, bwd or both.  option: none,
    filters (transport classes and bike transport), wheelchair (profile 2),
    realtime (delayed runs over the timetable)."""
    c = {"scale": scale, "kind": kind, "n": n, "call": call, "direction": direction, "option": option,
         "window": window}
    return dict(c, name=name) if name else c


def listed():
    return [
        # one traveller asks, nothing else runs: latency of the smallest call
        case("city_single", "city", "ontrip", 1),
        # the same on a region, by the one-query call
        case("regional_single_plain", "regional", "ontrip", 1, call="plain"),
        # isochrones from one place for a caller that may not allocate
        case("regional_isochrone_noalloc", "regional", "one_to_all", 1, call="noalloc"),
        # a city's requests of some seconds in one batch
        case("city_batch_1000", "city", "ontrip", 1000),
        # a small batch on a region: door to door, several stops at each end
        case("regional_batch_64", "regional", "ontrip", 64),
        # the benchmark's batch
        case("regional_batch_1024", "regional", "ontrip", 1024),
        # "arrive by" with transport classes and bikes: section checks
        case("regional_filters_bwd_333", "regional", "ontrip", 333, direction="bwd", option="filters"),
        # the same region while runs are late
        case("regional_realtime_250", "regional", "ontrip", 250, option="realtime"),
        # timetable information: all departures of a window, both directions
        case("regional_range_96", "regional", "range", 96, direction="both", window=240),
        # windows by the alternating search
        case("regional_pong_48", "regional", "pong", 48, direction="both", window=120),
        # a server's request loop with a burst of requests
        case("regional_served_500", "regional", "ontrip", 500, call="serve"),
        # a country's mixed traffic
        case("national_mix_256", "national", "mix", 256),
    ]


def _size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    family = rng.choice(["single", "batch", "batch", "option", "range", "pong", "all", "noalloc", "mix", "serve"])
    either = rng.choice(["fwd", "bwd"])
    scale = rng.choice(["city", "regional"])
    if family == "single":
        return case(None, rng.choice(["city", "regional", "national"]), "ontrip", rng.randint(1, 9),
                    call=rng.choice(["batch", "plain"]), direction=either)
    if family == "batch":
        if rng.random() < 0.25:
            return case(None, "national", "ontrip", _size(rng, 8, 256), direction=either)
        return case(None, scale, "ontrip", _size(rng, 10, 1024), direction=either)
    if family == "option":
        return case(None, scale, "ontrip", _size(rng, 10, 700), direction=either,
                    option=rng.choice(["filters", "wheelchair", "realtime"]))
    if family == "range":
        return case(None, scale, "range", _size(rng, 4, 128), direction=rng.choice(["fwd", "bwd", "both"]),
                    window=rng.randint(30, 240))
    if family == "pong":
        return case(None, scale, "pong", _size(rng, 4, 64), window=rng.randint(30, 150),
                    direction=rng.choice(["fwd", "bwd", "both"]))
    if family == "all":
        return case(None, scale, "one_to_all", _size(rng, 2, 48), direction=either)
    if family == "noalloc":
        return case(None, scale, "one_to_all", rng.randint(1, 8), call="noalloc", direction=either)
    if family == "mix":
        return case(None, "national", "mix", _size(rng, 16, 240))
    return case(None, scale, "ontrip", _size(rng, 16, 1000), call="serve", direction=either)


# ------------------------------------------------ what a program keeps
_kept = {}


def _keep(key, make):
    if key not in _kept:
        _kept[key] = make()
    return _kept[key]


def _host(scale):
    return _keep(("host", scale), lambda: HostTimetable.generate(TIMETABLE[scale]))


def _device(scale):
    return _keep(("device", scale), lambda: R.Timetable(_host(scale).desc, owner=_host(scale)))


def _slots(n):
    """A pool for n requests at once, as a program sizes it: a power of two."""
    return min(1024, max(32, 1 << (n - 1).bit_length()))


def _engine(c):
    slots, realtime, serve = _slots(c["n"]), c["option"] == "realtime", c["call"] == "serve"

    def make():
        e = R.Engine(_device(c["scale"]), max_slots=slots)
        if realtime:
            assert A.lib().b2r_engine_set_rt(e.handle, _overlay(c["scale"])) == 0
        return R.Server(e) if serve else e

    return _keep(("engine", c["scale"], slots, realtime, serve), make)


def _today(scale):
    """The service day of the real-time state: a Tuesday."""
    return _host(scale).desc.date_range_from + (1 if scale == "city" else 64)


def _overlay(scale):
    """One trip in a hundred of today's runs late: from some stop on by 1 to
    20 minutes, the delay carried to the end; the planned trip leaves the
    timetable on that day (b2r_rt_upload)."""

    def make():
        h = _host(scale)
        d = h.desc
        rnd = np.random.RandomState(7)
        view = np.ctypeslib.as_array
        rsi = view(d.route_stop_index, (d.n_routes + 1,))
        stops = view(d.route_stops, (int(rsi[-1]),))
        first = view(d.route_transport_from, (d.n_routes,))
        last = view(d.route_transport_to, (d.n_routes,))
        at = view(d.route_stop_time_from, (d.n_routes,))
        times = view(d.route_stop_times, (d.n_route_stop_times,))
        route = view(d.transport_route, (d.n_transports,))
        days = view(d.bitfields, (d.n_bitfields, 8))[view(d.transport_traffic_days, (d.n_transports,))]
        internal = d.date_range_from - 5
        day = _today(scale) - internal
        runs = np.flatnonzero((days[:, day >> 6] >> np.uint64(day & 63)) & np.uint64(1))
        late = np.sort(rnd.choice(runs, max(1, len(runs) // 100), replace=False)).astype(np.uint32)
        changed = days[late].copy()
        changed[:, day >> 6] &= ~np.uint64(1 << (day & 63))
        index, words, events, clasz = [0], [], [], []
        for t in late:
            r = int(route[t])
            n_s, n_t = int(rsi[r + 1] - rsi[r]), int(last[r] - first[r])
            w = times[int(at[r]) + n_t * np.arange(2 * (n_s - 1)) + int(t - first[r])].astype(np.int32)
            ev = (internal + day + (w & 31)) * 1440 + (w >> 5)
            ev[rnd.randint(0, len(ev)):] += rnd.randint(1, 21)
            index.append(index[-1] + n_s)
            words.append(stops[int(rsi[r]):int(rsi[r + 1])])
            events.append(ev)
            clasz.append(int(d.route_clasz[r]) if d.route_clasz else 10)
        keep = [late, np.ascontiguousarray(changed), np.array(index, np.uint32),
                np.concatenate(words).astype(np.uint32), np.concatenate(events).astype(np.int32),
                np.full(len(late), day, np.uint16), np.array(clasz, np.uint8)]
        o = A.RtDesc()
        ptr = lambda x, t: x.ctypes.data_as(C.POINTER(t))  # noqa: E731
        o.n_changed = o.n_rt_transports = len(late)
        o.changed_transport = o.rt_static_transport = ptr(keep[0], C.c_uint32)
        o.changed_days = ptr(keep[1], C.c_uint64)
        o.rt_stop_index = ptr(keep[2], C.c_uint32)
        o.rt_stops = ptr(keep[3], C.c_uint32)
        o.rt_event_times = ptr(keep[4], C.c_int32)
        o.rt_static_day = ptr(keep[5], C.c_uint16)
        o.rt_clasz = ptr(keep[6], C.c_uint8)
        handle = C.c_void_p()
        assert A.lib().b2r_rt_upload(_device(scale).handle, C.byref(o), C.byref(handle)) == 0
        return handle

    return _keep(("overlay", scale), make)


# ------------------------------------------------------------- one case
def _mixed(qs, n):
    """n requests of the mixed stream in its order, with exactly its shares of
    each kind."""
    left = {"range": round(0.2 * n), "all": round(0.1 * n)}
    left["one"] = n - sum(left.values())
    take = []
    for i in range(qs.n):
        q = qs.arr[i]
        kind = "all" if q.kind == A.B2R_ONE_TO_ALL else "range" if q.is_interval else "one"
        if left[kind]:
            left[kind] -= 1
            take.append(i)
    assert len(take) == n
    return qs.subset(take)


def prepare(case, seed):
    c = case
    h = _host(c["scale"])
    workload = RANGE if c["kind"] in ("range", "pong") else MIX if c["kind"] == "mix" else ONTRIP[c["scale"]]
    if c["scale"] == "national" and c["kind"] != "mix":  # the national stream without its ranges and one-to-alls
        workload = ONTRIP["regional"] if c["kind"] == "ontrip" else workload
    qs = QuerySet(h, workload, 3 * c["n"] + 64 if c["kind"] == "mix" else c["n"], seed=1 + seed)
    arr = _mixed(qs, c["n"]) if c["kind"] == "mix" else qs.arr
    rnd = np.random.RandomState(seed & 0x7FFFFFFF)
    for i in range(c["n"]):
        q = arr[i]
        if c["direction"] != "both" and c["kind"] != "mix":
            q.direction = A.B2R_FORWARD if c["direction"] == "fwd" else A.B2R_BACKWARD
        if c["kind"] == "pong":
            q.algorithm = A.B2R_ALGO_PONG
            q.use_start_footpaths = 1
        if q.is_interval and c["window"]:
            q.interval_to = q.interval_from + int(rnd.randint(30, c["window"] + 1))
        if c["kind"] == "one_to_all":
            q.kind = A.B2R_ONE_TO_ALL
            q.n_destination = 0
            q.n_start = 1
        if c["option"] == "filters":  # no subway for some; bikes come along for every second
            q.allowed_claszes = 0xFFFF & ~(1 << 8) if rnd.randint(2) else A.B2R_ALL_CLASZ
            q.require_bike_transport = int(rnd.randint(2))
        if c["option"] == "wheelchair":
            q.prf_idx = A.B2R_PROFILE_WHEELCHAIR
        if c["option"] == "realtime":  # today, from the morning to the evening
            q.start_time = _today(c["scale"]) * 1440 + q.start_time % 1440
    n_j = c["n"] * JOURNEYS[c["kind"]] + 128
    s = {"case": c, "set": qs, "queries": arr, "out": (A.Result * c["n"])(),
         "journeys": np.zeros(n_j, JOURNEY), "legs": np.zeros((n_j * LEGS, C.sizeof(A.Leg) // 4), "i4")}
    if c["call"] == "noalloc":
        n_loc = h.desc.n_locations
        s["timetable"] = _device(c["scale"])
        s["rows"] = [torch.empty(A.B2R_K * n_loc, dtype=torch.int16, pin_memory=True) for _ in range(c["n"])]
        s["n_loc"] = n_loc
    else:
        s["engine"] = _engine(c)
        s["n_loc"] = h.desc.n_locations
    return s


def _check(rc):
    if rc != A.B2R_OK:
        raise RuntimeError("b2r status %d: %s" % (rc, A.lib().b2r_last_error().decode()))


def _journeys(state, res, at=(0, 0)):
    """The journeys and legs of results, copied out of the engine's memory
    behind the first at[0] journeys and at[1] legs; how many there are now."""
    has = np.flatnonzero(res["n_journeys"])
    if len(has) == 0:
        return at
    js, legs = state["journeys"], state["legs"]
    size = JOURNEY.itemsize
    new = np.frombuffer(b"".join([C.string_at(p, k * size) for p, k in zip(
        res["journeys"][has].tolist(), res["n_journeys"][has].tolist())]), JOURNEY)
    js[at[0]:at[0] + len(new)] = new
    end = np.cumsum(res["n_journeys"][has]) - 1
    n_legs = new["first_leg"][end] + new["n_legs"][end]
    size = legs.itemsize * legs.shape[1]
    raw = np.frombuffer(b"".join([C.string_at(p, k * size) for p, k in zip(
        res["legs"][has].tolist(), n_legs.tolist())]), "i4").reshape(-1, legs.shape[1])
    legs[at[1]:at[1] + len(raw)] = raw
    return at[0] + len(new), at[1] + len(raw)


def _answer(state, res, used):
    """What the requests came to; the arrays of journeys and legs have room
    for more and end in zeros."""
    js, legs = state["journeys"], state["legs"]
    js[used[0]:] = np.zeros((), JOURNEY)
    legs[used[1]:] = 0
    rows = [np.ctypeslib.as_array((C.c_int16 * (k * state["n_loc"])).from_address(p))
            for p, k in zip(res["round_times"].tolist(), res["n_rows"].tolist()) if p]
    return {"status": res["status"], "n_journeys": res["n_journeys"].astype("i4"),
            "interval": np.stack([res["interval_from"], res["interval_to"]]), "journeys": js.view("i4"),
            "legs": legs, "rows": rows}


def run(state):
    c, lib, arr, out, n = state["case"], A.lib(), state["queries"], state["out"], state["case"]["n"]
    if c["call"] == "noalloc":
        # on the default stream; a call returns when its rows are on the host
        tt, rows, n_rows, day, got = state["timetable"].handle, state["rows"], C.c_uint32(), C.c_int32(), []
        for i in range(n):
            _check(lib.b2r_one_to_all_noalloc(
                tt, C.byref(arr[i]), C.cast(rows[i].data_ptr(), C.POINTER(C.c_int16)), rows[i].numel(),
                C.byref(n_rows), C.byref(day), None))
            got.append(rows[i][:n_rows.value * state["n_loc"]])
        return got
    res = np.frombuffer(out, RESULT)
    if c["call"] == "serve":
        e = state["engine"].engine.handle
        tickets, t = [], C.c_uint64()
        for i in range(n):
            _check(lib.b2r_submit(e, C.byref(arr[i]), C.byref(t)))
            tickets.append(t.value)
        for i, t in enumerate(tickets):
            _check(lib.b2r_wait(e, t, C.byref(out[i])))
        used = _journeys(state, res)
        for t in tickets:
            _check(lib.b2r_release(e, t))
        return _answer(state, res, used)
    e = state["engine"].handle
    if c["call"] == "plain":
        used = (0, 0)
        for i in range(n):  # a result is read before the next call reuses its memory
            _check(lib.b2r_search_plain(e, C.byref(arr[i]), C.byref(out[i])))
            used = _journeys(state, res[i:i + 1], used)
        return _answer(state, res, used)
    _check(lib.b2r_search_batch(e, arr, n, out))
    return _answer(state, res, _journeys(state, res))


# Bytes a search reads and writes in its route scans (counted on the device: 8
# per route stop of a marked route, 2 per event and 8 per service day a trip
# search looks at, 2 per label written), on average over each timetable's
# request stream: of one start time, of one of a window's start times, and to
# everywhere; and the start times a minute of a window brings.
ONE = {"city": 0.45e6, "regional": 1.0e6, "national": 15e6}
OF_WINDOW = {"city": 0.12e6, "regional": 0.43e6, "national": 3.2e6}
ALL = {"city": 0.83e6, "regional": 65e6, "national": 82e6}
STARTS_PER_MIN = 0.17


def work(case):
    c = case
    s, n = c["scale"], c["n"]
    rows = A.B2R_K * _host(s).desc.n_locations * 2
    minute = STARTS_PER_MIN * OF_WINDOW[s]
    if c["kind"] == "one_to_all":
        return {"bytes": n * (ALL[s] + rows), "flops": 0}
    if c["kind"] == "mix":
        return {"bytes": n * (0.7 * ONE[s] + 0.2 * 60 * minute + 0.1 * (ALL[s] + rows)), "flops": 0}
    if c["kind"] in ("range", "pong"):
        return {"bytes": n * (30 + c["window"]) / 2 * minute, "flops": 0}
    return {"bytes": n * ONE[s], "flops": 0}
