"""Meshes that leave most of the chip idle: their edges and elements share a launch in blocks of
32 elements, and their limiter takes the node bounds from the element means, six elements
around a node at first and the rest after.  One element short of a block to one over, nodes of
one to 13 elements, sizes either side of both switches, against the oracle; an ensemble
whose scenarios meet inside blocks, against each mesh alone.  Friction zero, so the tolerance
is none (bit patterns), as in test_gpu_parity.py."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import bits_equal, land_film_state, moving_state

pytestmark = pytest.mark.gpu


def fan(dgrain, n):
    """n triangles around one node"""
    a = 2 * np.pi * np.arange(n) / n
    x, y = (np.concatenate([[0.0], 1000.0 * f(a)]) for f in (np.cos, np.sin))
    el2v = np.array([[0, 1 + k, 1 + (k + 1) % n] for k in range(n)], dtype=np.int32)
    none = np.empty((0, 2), dtype=np.int32)
    return dgrain.mesh.build_connectivity(dgrain.mesh.Mesh(x, y, 5.0 + 1e-4 * x, np.zeros(n + 1), el2v, none, none, none))


def against_oracle(dgrain, oracle_mod, m, st, wet_dry, steps=4):
    o = oracle_mod.Oracle(m)
    o.set_state(*st)
    rc, t_o, dt_o, n_o, _ = o.run(steps, 1e9, 0.3, wet_dry=wet_dry, tide_on=1, amp=0.5)
    assert rc == 0
    with dgrain.Solver(m, wet_dry=wet_dry, cfl=0.3, tide_on=1, tide_amp=0.5) as s:
        s.upload_state(*st)
        assert s.time_evolution(1e9, steps) == (t_o, dt_o, n_o)
        for a, b in zip(s.download_state(), o.get_state()):
            assert bits_equal(a, b)


@pytest.mark.parametrize("n", [3, 6, 7, 9, 13])
def test_fans_bitexact(dgrain, oracle_mod, n):
    m = fan(dgrain, n)
    against_oracle(dgrain, oracle_mod, m, moving_state(dgrain, m, seed=n, depth=6.0, qscale=0.05), 0)


@pytest.mark.parametrize("wet_dry", [0, 1])
@pytest.mark.parametrize("nx,ny", [(1, 1), (15, 1), (4, 4), (17, 1), (31, 33), (109, 109), (110, 110), (120, 100), (121, 100),
                                   (250, 200), (251, 200)])
def test_rectangles_bitexact(dgrain, oracle_mod, nx, ny, wet_dry):
    m = dgrain.rectangle(nx, ny, jitter=0.1, seed=nx, manning=0.0, datum=0.0 if wet_dry else 7.0)
    st = land_film_state(dgrain, m, film=0.9e-3) if wet_dry else moving_state(dgrain, m, seed=2, depth=9.0, qscale=0.05)
    against_oracle(dgrain, oracle_mod, m, st, wet_dry)


@pytest.mark.parametrize("stages", [2, 3])
@pytest.mark.parametrize("flux", [0, 1, 2])
def test_small_ensemble_bitexact(dgrain, flux, stages):
    meshes = [dgrain.rectangle(nx, ny, jitter=0.1, seed=k, datum=7.0)
              for k, (nx, ny) in enumerate([(3, 2), (17, 1), (1, 1), (40, 20), (5, 5), (31, 2)])]
    states = [moving_state(dgrain, m, seed=k, depth=9.0, qscale=0.05) for k, m in enumerate(meshes)]
    kw = dict(wet_dry=0, cfl=0.3, flux=flux, rk_stages=stages)
    with dgrain.Ensemble(meshes, [dict(rain=1e-6 * k) for k in range(6)], **kw) as e:
        for k, st in enumerate(states):
            e.upload_state(k, *st)
        t, dt, n = e.run(18)
        got = [e.download_state(k) for k in range(6)]
    for k, m in enumerate(meshes):
        with dgrain.Solver(m, rain=1e-6 * k, **kw) as s:
            s.set_schedule(128, 1)  # the persistent kernels, edges apart from elements
            s.upload_state(*states[k])
            assert s.time_evolution(1e300, 18) == (t[k], dt[k], n[k])
            for a, b in zip(got[k], s.download_state()):
                assert bits_equal(a, b)
