"""Gradients of meshes whose recomputation takes edges and elements in launches of their own (above
8,000 triangles), a ragged size with a shoreline, two and three stages: the recomputed run is the
plain one bit for bit, and adjoint . direction is the tangent-linear derivative to round-off, at
the tolerance of test_gpu_adjoint.py.  Gradients copied by threads (6 MB and more of results),
with results left out and pinned arrays among them, are the same bytes."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from conftest import bits_equal
from test_gpu_adjoint import coastal_case, directions

pytestmark = pytest.mark.gpu

NSTEPS = 12


def make(dgrain, nx, ny, stages, ckpt):
    case = coastal_case(dgrain, nx, ny)
    m, state, n_el, pts = case
    kw = dict(wet_dry=1, cfl=0.3, tide_on=1, tide_amp=0.5, rk_stages=stages)
    s = dgrain.Solver(m, **kw)
    s.set_element_manning(n_el)
    el, w = dgrain.place_gauges(m, pts)
    mis = dgrain.GaugeMisfit(s, NSTEPS, ckpt, el, w)
    _, vals = mis.forward(state)
    mis.set_target(vals + 0.01 * np.random.default_rng(1).standard_normal(vals.shape))
    return case, kw, s, mis


@pytest.mark.parametrize("stages", [2, 3])
def test_gradient_above_the_shared_launch(dgrain, stages):
    case, kw, s, mis = make(dgrain, 81, 53, stages, NSTEPS)  # 8,586 triangles, one segment
    m, state, n_el, _ = case
    J, _ = mis.forward(state)
    with dgrain.Solver(m, **kw) as r:
        r.set_element_manning(n_el)
        r.upload_state(*state)
        r.time_evolution(1e300, NSTEPS)
        want = r.download_state()
    for a, b in zip(s.download_state(), want):
        assert bits_equal(a, b)
    g = mis.backward()
    for a, b in zip(s.download_state()[:3], want[:3]):  # the segment's recomputation
        assert bits_equal(a, b)
    dn, dz, ds = directions(m, 1)
    for kwd, adj in ((dict(dn_el=dn), g["n_el"] @ dn), (dict(dz=dz), g["z"] @ dz),
                     (dict(dstate=ds), g["zeta0"] @ ds[0] + g["qx0"] @ ds[1] + g["qy0"] @ ds[2])):
        Jt, dJ = mis.tlm(state, **kwd)
        assert Jt == J
        assert abs(dJ - adj) <= 1e-10 * max(abs(dJ), abs(adj)) + 1e-14 * J, (kwd.keys(), dJ, adj)
    s.close()


def test_gradient_downloads(dgrain):
    case, _, s, mis = make(dgrain, 331, 163, 2, 8)  # 107,906 triangles: 9 MB of results
    m, state = case[:2]
    mis.forward(state)
    g = mis.backward()
    names = ("n_el", "z", "zeta0", "qx0", "qy0")
    ptr = dgrain.mesh._dp
    pinned = {}
    for k in names:
        p = s.lib.dgr_host_alloc(g[k].nbytes)
        assert p
        pinned[k] = p, np.ctypeslib.as_array(C.cast(p, C.POINTER(C.c_double)), (g[k].size,))
    try:
        for left_out, on_pinned in (((), ()), (("qx0",), ()), (("n_el", "z", "qy0"), ()), (("zeta0", "qx0", "qy0"), ()),
                                    ((), ("zeta0",)), (("z",), ("n_el", "qy0")), ((), names), (names, ())):
            got = {k: pinned[k][1] if k in on_pinned else np.empty(g[k].size) for k in names}
            for k in names:
                got[k][:] = 7.0
            args = [None if k in left_out else ptr(got[k]) for k in names]
            assert s.lib.dgr_adjoint_backward(s.ctx, *args) == 0
            for k in names:
                assert bits_equal(got[k], np.full(g[k].size, 7.0) if k in left_out else g[k]), (k, left_out, on_pinned)
    finally:
        for p, _ in pinned.values():
            s.lib.dgr_host_free(p)
        s.close()
