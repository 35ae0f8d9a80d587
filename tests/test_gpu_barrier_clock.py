"""A step whose grid-barrier wait ran out did not happen: the run's step count, its next dt and
the context's record of the wet/dry flags leave it out, at both fusion depths.  The wait runs
out by the phantom block of dgr_set_barrier_wait, as in test_gpu_barrier.py."""
from __future__ import annotations

import ctypes as C

import pytest

from conftest import bits_equal, land_film_state

pytestmark = pytest.mark.gpu

KW = dict(wet_dry=1, cfl=0.3, tide_on=1, tide_amp=0.5)


@pytest.mark.parametrize("steps", [1, 3, 17])  # 17: two graphs of eight and one step
@pytest.mark.parametrize("fusion", [1, 2])
def test_timed_out_steps_are_not_counted(dgrain, fusion, steps):
    m = dgrain.rectangle(60, 30, jitter=0.1, seed=3)
    st = land_film_state(dgrain, m)
    with dgrain.Solver(m, **KW) as s:
        s.upload_state(*st)
        want_clock = s.time_evolution(1e9, 12)
        want = s.download_state()
    with dgrain.Solver(m, **KW) as s:
        s.set_schedule(128, fusion)
        s.upload_state(*st)
        s.time_evolution(1e9, 3)
        s.upload_state(*st)
        s.set_barrier_wait(1000, 1)
        t, dt, n = C.c_double(0.0), C.c_double(0.25), C.c_int(-1)
        rc = s.lib.dgr_run(s.ctx, steps, 1e9, C.byref(t), C.byref(dt), C.byref(n))
        assert rc == dgrain._lib.DGR_ERR_TIMEOUT
        assert (n.value, dt.value) == (0, 0.25)
        got = s.download_state()
        for a, b in zip(got[:3], st[:3]):
            assert bits_equal(a, b)
        s.set_barrier_wait()
        s.upload_state(*st)
        assert s.time_evolution(1e9, 12) == want_clock
        for a, b in zip(s.download_state(), want):
            assert bits_equal(a, b)
