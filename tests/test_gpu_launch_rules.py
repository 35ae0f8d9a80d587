"""Meshes at the lines between the step's launches: edges and elements share one up to 8,000
triangles (Roe), the limiter takes the node bounds itself up to 100,000.  Sizes either side of the
lower line; the block sizes of the schedule where they reach the element kernel (above the lower
line) and the limiter (above the upper one).  Against the oracle with friction zero, so the
tolerance is none (bit patterns), as in test_gpu_parity.py."""
from __future__ import annotations

import pytest

from conftest import bits_equal, land_film_state, moving_state

pytestmark = pytest.mark.gpu


def case(dgrain, nx, ny, wet_dry):
    m = dgrain.rectangle(nx, ny, jitter=0.1, seed=nx, manning=0.0, datum=0.0 if wet_dry else 7.0)
    st = land_film_state(dgrain, m, film=0.9e-3) if wet_dry else moving_state(dgrain, m, seed=2, depth=9.0, qscale=0.05)
    return m, st


def against_oracle(dgrain, oracle_mod, nx, ny, wet_dry, block_sizes=(64,), steps=4):
    m, st = case(dgrain, nx, ny, wet_dry)
    o = oracle_mod.Oracle(m)
    o.set_state(*st)
    rc, t_o, dt_o, n_o, _ = o.run(steps, 1e9, 0.3, wet_dry=wet_dry, tide_on=1, amp=0.5)
    assert rc == 0
    want = o.get_state()
    with dgrain.Solver(m, wet_dry=wet_dry, cfl=0.3, tide_on=1, tide_amp=0.5) as s:
        for bs in block_sizes:
            s.set_schedule(bs, 0)
            s.upload_state(*st)
            assert s.time_evolution(1e9, steps) == (t_o, dt_o, n_o), bs
            for a, b in zip(s.download_state(), want):
                assert bits_equal(a, b), bs


@pytest.mark.parametrize("wet_dry", [0, 1])
@pytest.mark.parametrize("nx,ny", [(59, 67), (80, 50), (81, 50)])  # 7,906, 8,000 and 8,100 triangles
def test_either_side_of_the_shared_launch(dgrain, oracle_mod, nx, ny, wet_dry):
    against_oracle(dgrain, oracle_mod, nx, ny, wet_dry)


@pytest.mark.parametrize("wet_dry", [0, 1])
@pytest.mark.parametrize("nx,ny", [(81, 53), (331, 163)])  # 8,586 and 107,906: whole in no block size
def test_block_sizes_where_they_count(dgrain, oracle_mod, nx, ny, wet_dry):
    against_oracle(dgrain, oracle_mod, nx, ny, wet_dry, (64, 128, 256))


@pytest.mark.parametrize("wet_dry", [0, 1])
@pytest.mark.parametrize("nx,ny", [(59, 67), (81, 53), (331, 163)])
def test_three_stages(dgrain, nx, ny, wet_dry):
    """SSP(3,3), whose second stage is in place: the three launch forms against the persistent
    kernels (edges apart from elements), at every block size"""
    m, st = case(dgrain, nx, ny, wet_dry)
    kw = dict(wet_dry=wet_dry, cfl=0.3, rk_stages=3, tide_on=1, tide_amp=0.5)
    with dgrain.Solver(m, **kw) as s:
        def run(bs, fusion):
            s.set_schedule(bs, fusion)
            s.upload_state(*st)
            return s.time_evolution(1e9, 4), s.download_state()

        want_clock, want = run(128, 1)
        for bs in (64, 128, 256):
            clock, got = run(bs, 0)
            assert clock == want_clock
            for a, b in zip(got, want):
                assert bits_equal(a, b), bs
