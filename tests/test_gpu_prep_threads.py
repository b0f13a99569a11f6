"""A batch is prepared on as many host threads as the engine was given."""
import os
import threading

import pytest

from nigiri_b200 import _abi as A
from nigiri_b200 import routing as R
from nigiri_b200.timetable import HostTimetable, QuerySet

pytestmark = pytest.mark.gpu


def threads_during(call):
    """The most threads of this process beside the caller's while it runs."""
    most, stop = [0], threading.Event()

    def watch():
        while not stop.is_set():
            most[0] = max(most[0], len(os.listdir("/proc/self/task")))

    t = threading.Thread(target=watch)
    t.start()
    before = len(os.listdir("/proc/self/task"))
    call()
    stop.set()
    t.join()
    return most[0] - before


@pytest.mark.parametrize("given", [2, 8])
def test_host_threads_are_the_callers(given):
    h = HostTimetable.generate(1)
    eng = R.Engine(R.Timetable(h.desc, owner=h), max_slots=32, host_threads=given)
    qs = QuerySet(h, 1, 12, seed=3)
    keep = []
    for i in range(qs.n):  # a millisecond of preparation each: a day's departures from 64 stops
        q = qs.arr[i]
        st = (A.Offset * 64)()
        for j in range(64):
            st[j].target = 9 + (7 * j + i) % (h.desc.n_locations - 9)
        keep.append(st)
        q.start, q.n_start, q.start_match_mode = st, 64, A.B2R_MATCH_INTERMODAL
        q.is_interval, q.interval_from, q.interval_to = 1, q.start_time, q.start_time + 1440
    out = (A.Result * qs.n)()

    def call():
        assert A.lib().b2r_search_batch(eng.handle, qs.arr, qs.n, out) == 0, A.lib().b2r_last_error()

    call()  # the process's own first-call threads
    most = 0
    for _ in range(40):  # until the watching thread has seen all of them at once
        most = max(most, threads_during(call))
        if most >= given:
            break
    assert most == given
