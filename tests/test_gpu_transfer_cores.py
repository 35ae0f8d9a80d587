"""A process that may use fewer CPUs than the copies' threads keeps to the calling thread where
the threads would only take turns: states up, and down into pages that are there."""
from __future__ import annotations

import os
import threading
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def most_threads_during(call):
    """the largest number of the process's threads seen while call runs"""
    seen, stop = [0], threading.Event()

    def watch():
        while not stop.is_set():
            seen[0] = max(seen[0], len(os.listdir("/proc/self/task")))

    w = threading.Thread(target=watch)
    w.start()
    try:
        call()
    finally:
        stop.set()
        w.join()
    return seen[0]


def test_no_threads_on_one_cpu(dgrain):
    cpus = os.sched_getaffinity(0)
    if len(cpus) < 2:
        pytest.skip("one CPU only: nowhere to watch from")
    m = dgrain.rectangle(1000, 400, seed=1, datum=7.0)
    rng = np.random.default_rng(2)
    st = [rng.standard_normal(3 * m.num_el) for _ in range(3)] + [np.ones(m.num_el, np.int32)]
    got = [np.ones_like(a) for a in st]
    ptr, iptr = dgrain.mesh._dp, dgrain.mesh._ip
    with dgrain.Solver(m, wet_dry=0) as s:
        def copies():
            os.sched_setaffinity(0, {min(cpus)})  # this thread; the watching one keeps the others
            try:
                for _ in range(20):
                    s.upload_state(*st)
                    assert s.lib.dgr_download_state(s.ctx, *[ptr(a) for a in got[:3]], iptr(got[3])) == 0
            finally:
                os.sched_setaffinity(0, cpus)

        s.upload_state(*st)
        s.download_state()
        time.sleep(0.1)  # whatever the first copies start is there, their own threads are gone
        idle = len(os.listdir("/proc/self/task")) + 1
        assert most_threads_during(copies) <= idle
    for a, b in zip(st, got):
        assert np.array_equal(a, b)
