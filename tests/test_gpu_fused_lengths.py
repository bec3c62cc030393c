"""Row lengths of the fused nonlinear phases: the mixed-precision nonlinear terms
of every length with a row plan, in its forms (orders below nlon / 3 or not, a
last colatitude block of one pair, a partial last team), against the FP64 path.
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
# FP32 products and transforms, split-TF32 Legendre sums (about 2^-22 a product): the
# bound the mixed path's nonlinear terms are held to up to lmax 255; above, it grows
# with the number of degrees, since the tensor cores' FP32 sums truncate
TOL = 5e-6


def _tol(lmax):
    return TOL * max(1.0, (lmax + 1) / 256.0)


def _terms(gdb, precision, cfg, state):
    g = gdb.SHTnsKitConfig(precision=precision, **cfg)
    for k, (a, b) in state.items():
        g.set_field(k, a, b)
    g.step(2)  # the second step advects with the first one's velocity
    out = {k: g.get_nl(k) for k in ("temp", "u_tor", "u_pol", "b_tor", "b_pol")}
    g.close()
    return out


@pytest.mark.parametrize("nlon,mmax", [(n, (n - 1) // 2 if n <= 512 or n == 768 else 200) for n in LENGTHS]
                         + [(n, n // 3 - 1) for n in LENGTHS if n % 3 == 0 and n <= 768] + [(256, 5), (125, 40), (810, 200)])
def test_terms_of_every_row_length(gdb, nlon, mmax):
    nlat = mmax + 1 + (mmax + 1) % 2
    nlat += 2 if nlat // 2 % 2 == 0 else 0  # an odd number of colatitude pairs
    cfg = dict(lmax=mmax, nlat=nlat, nlon=nlon, nr=5, dt=1e-5, bc_mode=2)
    state = workloads.seeded_state(mmax, mmax, 5, seed=3, amp=1.0)
    ref = _terms(gdb, "fp64", cfg, state)
    got = _terms(gdb, "mixed", cfg, state)
    for k in ("temp", "u_tor", "u_pol"):
        for x, y in zip(got[k], ref[k]):
            assert np.max(np.abs(x - y)) <= _tol(mmax) * max(np.max(np.abs(y)), 1e-300), k
    for k in ("b_tor", "b_pol"):  # products with the zero radial components
        for x in got[k]:
            assert not np.any(x)
