"""State up and down again, byte for byte: either side of the size at which a context copies
through threads (4 MB of state), chunks of 512 KB with a remainder, exact multiples of a chunk,
p = 2, the slices of an ensemble (below and above a threaded copy), pinned arrays."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def state(rng, m, nm):
    return [rng.standard_normal(nm * m.num_el) for _ in range(3)] + [rng.integers(0, 2, m.num_el).astype(np.int32)]


# 58,254 triangles hold 4 MB at p = 1; 65,536 hold exactly three chunks a variable
@pytest.mark.parametrize("nx,ny,order", [(240, 121, 1), (241, 121, 1), (256, 128, 1), (331, 163, 1), (121, 122, 2)])
def test_round_trip(dgrain, nx, ny, order):
    m = dgrain.rectangle(nx, ny, seed=1, datum=7.0)
    kw = dict(order=2, rk_stages=3) if order == 2 else {}
    with dgrain.Solver(m, wet_dry=0, **kw) as s:
        for seed in (1, 2):
            st = state(np.random.default_rng(seed), m, s.nm)
            s.upload_state(*st)
            for a, b in zip(st, s.download_state()):
                assert np.array_equal(a, b)


def test_ensemble_slices(dgrain):
    meshes = [dgrain.rectangle(nx, ny, seed=k, datum=7.0) for k, (nx, ny) in enumerate([(9, 4), (300, 101), (60, 31)])]
    rng = np.random.default_rng(3)
    with dgrain.Ensemble(meshes, [dict() for _ in meshes], wet_dry=0) as e:
        st = [state(rng, m, 3) for m in meshes]
        for k in (1, 0, 2):
            e.upload_state(k, *st[k])
        for k in (2, 1, 0):
            for a, b in zip(st[k], e.download_state(k)):
                assert np.array_equal(a, b)


def test_pinned_arrays(dgrain):
    lib = dgrain.load()
    m = dgrain.rectangle(256, 128, seed=1, datum=7.0)
    n = 3 * m.num_el
    p = lib.dgr_host_alloc(3 * n * 8)
    assert p
    try:
        pinned = np.ctypeslib.as_array(C.cast(p, C.POINTER(C.c_double)), (3, n))
        pinned[:] = np.random.default_rng(4).standard_normal((3, n))
        wd = np.ones(m.num_el, dtype=np.int32)
        with dgrain.Solver(m, wet_dry=0) as s:
            s.upload_state(pinned[0], pinned[1], pinned[2], wd)
            got = s.download_state()
        for a, b in zip(pinned, got):
            assert np.array_equal(a, b)
    finally:
        lib.dgr_host_free(p)
