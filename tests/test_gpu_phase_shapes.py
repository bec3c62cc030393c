"""Launch shapes of the FP32 phases: a handle of its own spreads few (shell,
colatitude block) teams over the SMs, each output in CTAs of its own; an
ensemble's member packs them into full CTAs.  Every team does the same arithmetic
in both, so the fields and nonlinear terms agree to the last bit, on both sides of
the team count at which a handle packs too (148 SMs).
"""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "geodynamo.jl_b200"))
import workloads  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lmax,nlat,nlon,nr,magnetic", [
    (7, 12, 24, 3, 1),        # fewer teams than SMs
    (31, 48, 96, 9, 0),       # two components an output
    (31, 48, 96, 98, 1),      # 16 teams a CTA: the last nr with CTAs for each output
    (31, 48, 96, 99, 1),
    (31, 48, 96, 197, 1),     # and the last with fewer warps
    (31, 48, 96, 198, 1),
    (47, 50, 100, 20, 1),     # teams that do not fill a warp
    (63, 66, 128, 60, 1),
    (127, 192, 384, 9, 1),
    (127, 192, 384, 50, 1),
    (200, 202, 1024, 3, 1),   # teams of two warps
    (200, 202, 1024, 12, 1),
])
def test_spread_and_packed_agree(gdb, lmax, nlat, nlon, nr, magnetic):
    cfg = dict(lmax=lmax, nlat=nlat, nlon=nlon, nr=nr, dt=1e-6, bc_mode=2, magnetic=magnetic)
    state = workloads.seeded_state(lmax, lmax, nr, seed=2, amp=1.0)
    g = gdb.SHTnsKitConfig(precision="mixed", **cfg)
    e = gdb.Ensemble([cfg], precision="mixed")
    out = []
    for m, step in ((g, g.step), (e.members[0], e.step)):
        for k in m.field_names():
            m.set_field(k, *state[k])
        step(3)
        out.append([x for k in m.field_names() for x in m.get_field(k) + m.get_nl(k)])
    assert any(np.any(x) for x in out[0])
    for x, y in zip(*out):
        assert np.array_equal(x, y)
    g.close()
    e.close()
