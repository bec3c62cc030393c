"""Row lengths of the FP64 phi transforms that run within one buffer: scalar and
vector transforms against the oracle, and the fused Coriolis stage against the
unfused FP64 chain, with an odd number of colatitude pairs (a last block with empty
rows) and with few or as many orders as the length holds.
"""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "geodynamo.jl_b200"))
import workloads  # noqa: E402

pytestmark = pytest.mark.gpu

LENGTHS = (24, 40, 48, 64, 80, 96, 100, 108, 128, 144, 160, 180, 192, 200, 216, 256, 288, 300, 320, 360, 384, 400,
           432, 450, 500, 512, 576, 600, 720, 768, 900, 1024)
# the bound of every FP64 transform against the oracle (relative, max norm): sums of
# at most 384 x 768 products, 2^-53 each
TOL = 1e-12


def _rel(a, b):
    return float(np.max(np.abs(a - b)) / np.max(np.abs(b)))


def _grid(nlon, mmax):
    nlat = mmax + 1 + (mmax + 1) % 2
    nlat += 2 if nlat // 2 % 2 == 0 else 0  # an odd number of colatitude pairs
    return dict(lmax=mmax, nlat=nlat, nlon=nlon, nr=3)


CASES = [(n, min((n - 1) // 2, 255)) for n in LENGTHS] + [(n, 3) for n in LENGTHS]


@pytest.mark.parametrize("nlon,mmax", CASES)
def test_transforms_match_oracle(gdb, oracle_mod, nlon, mmax):
    cfg = _grid(nlon, mmax)
    g, o = gdb.SHTnsKitConfig(**cfg), oracle_mod.Oracle(**cfg)
    re, im = workloads.transform_batch(mmax, mmax, cfg["nr"], 2, seed=nlon)
    grid = o.synth_scalar(re[0], im[0])
    assert _rel(g.synth_scalar(re[0], im[0]), grid) <= TOL
    for x, y in zip(g.analysis_scalar(grid), o.analysis_scalar(grid)):
        assert _rel(x, y) <= TOL
    degree = workloads.lm_arrays(mmax, mmax)[0]
    re[:, :, degree == 0] = 0
    im[:, :, degree == 0] = 0
    coef = (re[0], im[0], re[1], im[1])
    vec = o.synth_vector(*coef)
    for x, y in zip(g.synth_vector(*coef), vec):
        assert _rel(x, y) <= TOL
    for x, y in zip(g.analysis_vector(*vec), o.analysis_vector(*vec)):
        assert _rel(x, y) <= TOL
    g.close()


@pytest.mark.parametrize("nlon,mmax", [c for c in CASES if c[1] > 3])
def test_fused_coriolis_is_the_unfused_chain(gdb, nlon, mmax):
    cfg = dict(_grid(nlon, mmax), dt=1e-5, bc_mode=2)
    state = workloads.seeded_state(mmax, mmax, cfg["nr"], seed=5, amp=1.0)
    out = []
    for precision in ("fp64", "mixed_vel64"):
        g = gdb.SHTnsKitConfig(precision=precision, **cfg)
        for k, (a, b) in state.items():
            g.set_field(k, a, b)
        g.step(1)
        out.append([x for k in ("u_tor", "u_pol") for x in g.get_nl(k)])
        g.close()
    for x, y in zip(*out):
        assert np.any(x) and np.array_equal(x, y)
