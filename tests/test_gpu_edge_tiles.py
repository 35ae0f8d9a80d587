"""The edge kernel's blocks work through several tiles of 128 edges with the next tile's data
in flight: meshes of more tiles than resident blocks (592), with a ragged last tile, against
the oracle; an ensemble whose scenarios meet inside a block's tiles, against each mesh alone.
Friction zero, so the tolerance is none (bit patterns), as in test_gpu_parity.py."""
from __future__ import annotations

import pytest

from conftest import bits_equal, land_film_state, moving_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("wet_dry", [0, 1])
@pytest.mark.parametrize("nx,ny", [(201, 127), (331, 163)])  # 76,909 and 162,353 edges: 2 and 3 tiles per block
def test_many_tiles_bitexact(dgrain, oracle_mod, nx, ny, wet_dry):
    m = dgrain.rectangle(nx, ny, jitter=0.1, seed=6, manning=0.0)
    st = land_film_state(dgrain, m, film=0.9e-3) if wet_dry else moving_state(dgrain, m, seed=2, qscale=0.05)
    o = oracle_mod.Oracle(m)
    o.set_state(*st)
    rc, t_o, dt_o, n_o, _ = o.run(3, 1e9, 0.3, wet_dry=wet_dry, tide_on=1, amp=0.5)
    assert rc == 0
    with dgrain.Solver(m, wet_dry=wet_dry, cfl=0.3, tide_on=1, tide_amp=0.5) as s:
        s.upload_state(*st)
        assert s.time_evolution(1e9, 3) == (t_o, dt_o, n_o)
        for a, b in zip(s.download_state(), o.get_state()):
            assert bits_equal(a, b)


@pytest.mark.parametrize("flux", [0, 2])
def test_ensemble_tiles_bitexact(dgrain, flux):
    meshes = [dgrain.rectangle(nx, ny, jitter=0.1, seed=k, datum=7.0)
              for k, (nx, ny) in enumerate([(173, 60), (3, 2), (201, 127), (40, 20), (90, 45)])]
    states = [moving_state(dgrain, m, seed=k, depth=9.0, qscale=0.05) for k, m in enumerate(meshes)]
    kw = dict(wet_dry=0, cfl=0.3, flux=flux)
    with dgrain.Ensemble(meshes, [dict(rain=1e-6 * k) for k in range(5)], **kw) as e:
        for k, st in enumerate(states):
            e.upload_state(k, *st)
        t, dt, n = e.run(4)
        got = [e.download_state(k) for k in range(5)]
    for k, m in enumerate(meshes):
        with dgrain.Solver(m, rain=1e-6 * k, **kw) as s:
            s.upload_state(*states[k])
            assert s.time_evolution(1e300, 4) == (t[k], dt[k], n[k])
            for a, b in zip(got[k], s.download_state()):
                assert bits_equal(a, b)
