"""Interval extension (search.h:283-316) against the oracle: queries that need
it several times, in both directions, with footpaths from their start stops
and without, whose later phases keep some journeys and drop others."""
import ctypes as C
import random

import pytest

import oracle_lib
from journeys import records
from nigiri_b200 import _abi as A
from nigiri_b200 import routing as R
from nigiri_b200.timetable import HostTimetable, QuerySet
from test_algo_adapter import helper

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def city():
    h = HostTimetable.generate(1)
    tt = R.Timetable(h.desc, owner=h)
    return h, tt, R.Engine(tt, max_slots=64, max_journeys=1024, max_starts=8192)


def queries(h, n, footpaths, seed):
    rnd = random.Random(seed)
    qs = QuerySet(h, 1, n, seed=seed)
    for i in range(n):
        q = qs.arr[i]
        q.direction = rnd.randint(0, 1)
        q.max_transfers = rnd.choice((0, 1, 2, 7))
        q.is_interval, q.interval_from = 1, q.start_time
        q.interval_to = q.start_time + rnd.choice((5, 30, 90))
        q.min_connection_count = rnd.randint(1, 10)
        q.extend_interval_earlier, q.extend_interval_later = rnd.choice(((1, 0), (0, 1), (1, 1)))
        q.use_start_footpaths = footpaths
    return qs


def answer(r):
    return r.status, r.interval_from, r.interval_to, records(r)


@pytest.mark.parametrize("seed", range(6))
@pytest.mark.parametrize("footpaths", [0, 1])
def test_extended_windows_match_oracle(city, footpaths, seed):
    h, tt, eng = city
    qs = queries(h, 160, footpaths, seed)
    out = (A.Result * qs.n)()
    assert A.lib().b2r_search_batch(eng.handle, qs.arr, qs.n, out) == 0, A.lib().b2r_last_error()
    phases = 0
    for i in range(qs.n):
        o = oracle_lib.OracleResult(h.desc, qs.arr[i])
        assert answer(out[i]) == answer(o.view), i
        assert out[i].n_start_times == o.view.n_start_times and out[i].n_rounds == o.view.n_rounds, i
        phases += o.view.interval_to - o.view.interval_from > 150 + 60 * qs.arr[i].min_connection_count
    assert phases > 0  # windows wider than their first extension


@pytest.mark.parametrize("footpaths", [0, 1])
def test_extended_windows_step_driven(city, tmp_path, footpaths):
    h, tt, _ = city
    run = helper(str(tmp_path)).algo_search
    qs = queries(h, 48, footpaths, 11)
    for i in range(qs.n):
        got = A.Result()
        assert run(tt.handle, C.byref(h.desc), C.byref(qs.arr[i]), C.byref(got)) == 0, i
        assert answer(got) == answer(oracle_lib.OracleResult(h.desc, qs.arr[i]).view), i
