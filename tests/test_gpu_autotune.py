"""Where the block size changes no launch of the step's separate kernels (small meshes, p = 2), the
autotuner times that schedule once, reports it for every block size and keeps the default."""
from __future__ import annotations

import pytest

from conftest import moving_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order,stages,flux,one", [(1, 2, 0, True), (1, 3, 0, False), (1, 2, 2, False), (2, 3, 0, True)])
def test_one_trial_where_block_sizes_agree(dgrain, order, stages, flux, one):
    m = dgrain.rectangle(50, 30, jitter=0.1, seed=1, datum=7.0)
    kw = dict(order=2) if order == 2 else {}
    with dgrain.Solver(m, wet_dry=0, cfl=0.2, rk_stages=stages, flux=flux, **kw) as s:
        if order == 1:
            s.upload_state(*moving_state(dgrain, m, seed=1, depth=9.0, qscale=0.05))
        per_step = -s.kernel_launches()
        s.time_evolution(1e9, 1)
        per_step += s.kernel_launches()  # one step and the clock's end, the wet/dry status off
        before = s.kernel_launches()
        bs, fusion, table = s.autotune(trial_steps=3)
        at_zero = [table[(b, 0)] for b in (64, 128, 256)]
        if one:
            assert len(set(at_zero)) == 1 and (bs == 64 or fusion)
        if order == 2:  # no persistent kernels: one trial of one and three steps
            assert s.kernel_launches() - before == per_step + 3 * (per_step - 1) + 1
