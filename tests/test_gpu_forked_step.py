"""The captured step of a small FP64 model runs its phases side by side; with
per-kernel timing on, the same step runs as one chain.  Same kernels, same
inputs: every field, nonlinear term and carried grid must agree to the last bit.
"""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "geodynamo.jl_b200"))
import workloads  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lmax,nlat,nlon,nr,kw", [
    (31, 48, 96, 32, dict(bc_mode=2)),
    (20, 34, 48, 7, dict(bc_mode=0, ab_mode=1)),
    (15, 24, 48, 12, dict(bc_mode=0, scheme="eab2")),
    (15, 24, 48, 12, dict(bc_mode=0, scheme="erk2")),
    (15, 24, 48, 12, dict(bc_mode=2, geometry="ball")),
    (15, 24, 50, 12, dict(bc_mode=2, segments=2)),
    (127, 192, 384, 33, dict(bc_mode=2)),   # the largest four-component buffer that forks
    (127, 192, 384, 43, dict(bc_mode=2)),   # just above: one chain
])
def test_side_by_side_equals_chain(gdb, lmax, nlat, nlon, nr, kw):
    kw = dict(kw)
    scheme = kw.pop("scheme", "cnab2")
    out = []
    for timed in (False, True):
        g = gdb.SHTnsKitConfig(lmax, nlat, nlon, nr, dt=1e-5, **kw)
        g.set_scheme(scheme)
        for k, (a, b) in workloads.seeded_state(lmax, lmax, nr, seed=4, amp=1.0).items():
            g.set_field(k, a, b)
        g.profile_enable(timed)
        for _ in range(2):
            g.step(2)
        out.append([x for k in g.field_names() for x in g.get_field(k) + g.get_nl(k)] +
                   [g.get_grid(k) for k in ("u_th", "w_ph", "b_th", "j_ph", "t", "tadv", "vadv_th", "ind_ph")])
        g.close()
    for x, y in zip(*out):
        assert np.array_equal(x, y, equal_nan=True)
