"""One array given for several results holds the last of them, at every size: below and above the
sizes that are copied by threads."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shift", [0, 1000])  # the results' arrays: one and the same; overlapping
@pytest.mark.parametrize("nx,ny", [(40, 20), (241, 121), (500, 400)])
def test_results_in_one_array(dgrain, nx, ny, shift):
    m = dgrain.rectangle(nx, ny, seed=1, datum=7.0)
    n = 3 * m.num_el
    rng = np.random.default_rng(2)
    st = [rng.standard_normal(n) for _ in range(3)] + [np.ones(m.num_el, np.int32)]
    want = np.zeros(n + 2 * shift)
    for v in range(3):
        want[v * shift:v * shift + n] = st[v]
    ptr = dgrain.mesh._dp
    with dgrain.Solver(m, wet_dry=0) as s:
        s.upload_state(*st)
        for _ in range(5):
            got = np.zeros(n + 2 * shift)
            parts = [ptr(got[v * shift:v * shift + n]) for v in range(3)]
            assert s.lib.dgr_download_state(s.ctx, *parts, None) == 0
            assert np.array_equal(got, want)
