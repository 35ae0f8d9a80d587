"""Items whose operands are outside the range of the shared reciprocals (a momentum below
2^-900, so dividends there) take plain divisions inside the same launch: the same bits as the
oracle, mixed with ordinary items in one warp and alone.  Tolerance: none (bit patterns),
friction zero as in test_gpu_parity.py."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import bits_equal, land_film_state, moving_state

pytestmark = pytest.mark.gpu

TINY = 1e-290  # < 2^-900


@pytest.mark.parametrize("wet_dry", [0, 1])
@pytest.mark.parametrize("share", [0.02, 1.0])
def test_tiny_momentum_bitexact(dgrain, oracle_mod, share, wet_dry):
    m = dgrain.rectangle(33, 17, jitter=0.1, seed=2, manning=0.0)  # 1122 triangles: ragged blocks
    rng = np.random.default_rng(3)
    z, qx, qy, wd = land_film_state(dgrain, m, film=0.9e-3) if wet_dry else moving_state(dgrain, m, seed=4)
    if wet_dry:
        deep = np.repeat(m.z[m.el2v].min(axis=1) > 0.5, 3)
        qx, qy = (np.where(deep, 0.01 * rng.standard_normal(z.size), 0.0) for _ in range(2))
    tiny = np.repeat(rng.random(m.num_el) < share, 3)
    qx, qy = np.where(tiny, TINY * qx, qx), np.where(tiny, TINY * qy, qy)
    o = oracle_mod.Oracle(m)
    o.set_state(z, qx, qy, wd)
    with dgrain.Solver(m, wet_dry=wet_dry, cfl=0.3) as s:
        s.upload_state(z, qx, qy, wd)
        o.boundary_conditions()
        s.set_boundary(*o.get_bc())
        rz, rx, ry, lam = s.compute2DL()
        rc, oz, ox, oy, olam = o.compute_L(wet_dry)
        assert rc == 0 and lam == olam
        for a, b in zip((rz, rx, ry), (oz, ox, oy)):
            assert bits_equal(a, b)
        o.set_state(z, qx, qy, wd)
        s.upload_state(z, qx, qy, wd)
        rc, t_o, dt_o, n_o, _ = o.run(3, 1e9, 0.3, wet_dry=wet_dry)
        assert rc == 0 and s.time_evolution(1e9, 3) == (t_o, dt_o, n_o)
        for a, b in zip(s.download_state(), o.get_state()):
            assert bits_equal(a, b)
