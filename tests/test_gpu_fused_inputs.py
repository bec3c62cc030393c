"""Every input of the fused velocity and induction phases reaches its product, at
every row length with a row plan and in its forms.  The radial components are zero,
so the products with omega, j and B vanish for finite inputs whatever the
transforms deliver; a NaN does not: one in a coefficient of a shell must appear in
that shell's terms (and, through the radial derivatives of the curls, in four
shells to each side) as in the FP64 step, and nowhere else.
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
NR, SHELL, KL = 12, 2, 4
# orders below nlon / 3 (the three-way split where the plan has it), and as many as
# the length holds up to 160
CASES = [(n, n // 3 - 1 if n <= 480 else 120) for n in LENGTHS] + [(n, min((n - 1) // 2, 160)) for n in LENGTHS]


def _nan(g, state, field, part):
    L, M = workloads.lm_arrays(g.lmax, g.lmax)
    q = int(np.flatnonzero((L == 3) & (M == 1))[0])
    for k, (a, b) in state.items():
        a, b = a.copy(), b.copy()
        if k == field:
            (a, b)[part][SHELL, q] = np.nan
        g.set_field(k, a, b)


def _terms(g):
    return {k: np.stack([np.isnan(x) for x in g.get_nl(k)]) for k in ("temp", "u_tor", "u_pol", "b_tor", "b_pol")}


@pytest.mark.parametrize("nlon,mmax", CASES)
def test_nan_of_every_input_reaches_its_shells(gdb, nlon, mmax):
    nlat = mmax + 1 + (mmax + 1) % 2
    nlat += 2 if nlat // 2 % 2 == 0 else 0  # an odd number of colatitude pairs
    state = workloads.seeded_state(mmax, mmax, NR, seed=3, amp=1.0)
    a, b = (gdb.SHTnsKitConfig(mmax, nlat, nlon, NR, dt=1e-5, precision=p) for p in ("mixed", "fp64"))
    near = np.zeros(NR, dtype=bool)
    near[max(0, SHELL - KL):SHELL + KL + 1] = True
    own = np.arange(NR) == SHELL
    for field, part in (("b_tor", 0), ("b_pol", 1), ("u_tor", 1), ("u_pol", 0)):
        terms = []
        for g in (a, b):
            _nan(g, state, field, part)
            g.magnetic_nl()   # B and j of this state (and u of the phase before)
            g.velocity_nl()   # omega, u; j and B of the phase before
            first = _terms(g)
            g.magnetic_nl()   # the new u
            g.temperature_nl()
            terms.append((first, _terms(g)))
        for got, want in zip(*terms):
            for k in want:
                assert np.array_equal(got[k], want[k]), (field, k)
        first, second = terms[0]
        shells = lambda t, k: t[k].any(axis=(0, 2))  # noqa: E731
        # the velocity terms read the field of their own shell and its curl, whose
        # stencil reaches the shells around (the toroidal part enters it undifferentiated)
        for k in ("u_tor", "u_pol"):
            at = shells(first, k)
            assert at[SHELL] and not np.any(at & ~(near if field.endswith("pol") else own)), (field, k)
        # the induction and the advection read the field of their own shell
        for k in ("b_tor", "b_pol"):
            assert np.array_equal(shells(second, k), own), (field, k)
        assert np.array_equal(shells(second, "temp"), own & (field[0] == "u")), field
        # the next field starts from finite grids
        for g in (a, b):
            for k, (x, y) in state.items():
                g.set_field(k, x, y)
            g.magnetic_nl()
            g.velocity_nl()
            g.magnetic_nl()
    a.close()
    b.close()
