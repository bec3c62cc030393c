"""The pivots' quotient in the whole-step CNAB2 kernel and in its adjoint (a stored
reciprocal with one residual correction) against the division, which the separate
solve (gd_solve_implicit_step) still does: one numerator per mode in the last row,
from the smallest normal numbers to overflow, zeros, infinities and NaN.  The
quotient is bounded by 1/2 + 2^-50 ulp, so a value that differs from the correctly
rounded one at all (chance 2^-49 each) would be a neighbour; below 2^-968, where
the residual underflows, by two ulps.
"""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "geodynamo.jl_b200"))
import workloads  # noqa: E402

pytestmark = pytest.mark.gpu

LMAX, NR, DT, THETA = 31, 12, 1e-4, 0.5
PM, PR = 4.0, 1.0


def _numerators(n):
    rng = np.random.default_rng(7)
    x = np.ldexp(rng.uniform(0.5, 1.0, n) * rng.choice((-1.0, 1.0), n), rng.integers(-1015, 1021, n))
    x[:6] = [np.inf, -np.inf, np.nan, 0.0, -0.0, np.finfo(float).max]
    return x


def _check(got, want, num):
    assert np.array_equal(np.isnan(got), np.isnan(want))
    inf = np.isinf(want)
    assert np.array_equal(got[inf], want[inf]) and not np.any(np.isinf(got[~inf]))
    fin = np.isfinite(want)
    big = fin & (np.abs(num) >= 2.0 ** -968)
    assert np.array_equal(got[big], want[big])
    low = fin & ~big
    assert np.all(np.abs(got[low] - want[low]) <= 2 * np.spacing(np.abs(want[low])))


@pytest.fixture()
def model(gdb):
    g = gdb.SHTnsKitConfig(LMAX, 48, 96, NR, dt=DT, implicit_theta=THETA, bc_mode=0, magnetic_prandtl=PM, prandtl=PR)
    yield g
    g.close()


def _division(gdb, g, nu, num):
    """(re, im) of the solve whose right-hand side is num in the last row, by division."""
    m = gdb.SHTnsImplicitMatrices(g, nu, DT, THETA)
    rhs = [np.zeros(g.spec_shape()) for _ in range(2)]
    rhs[0][-1], rhs[1][-1] = num
    sol = m.solve_implicit_step(rhs)
    m.close()
    return sol


def test_step_quotient_is_the_division(gdb, model):
    import torch
    g = model
    n = g.nlm
    num = np.stack([_numerators(n), _numerators(n)[::-1]])  # reference order (l-major)
    field = 0  # u_tor
    # N in the native order; the first step's terms are 1.5 N - 0.5 N, the second's 1.5 N with no history
    L, M = workloads.lm_arrays(LMAX, LMAX)
    order = np.lexsort((L, M))
    block = torch.zeros((2, NR, n), dtype=torch.float64, device="cuda")
    g.copy_block(2, field, 0, NR, 0, n, block.data_ptr(), False)
    g.implicit_step()  # zero terms become the history
    g.set_field("u_tor", np.zeros(g.spec_shape()), np.zeros(g.spec_shape()))
    block[:, -1] = torch.from_numpy(np.ascontiguousarray(num[:, order])).cuda()
    torch.cuda.synchronize()
    g.copy_block(2, field, 0, NR, 0, n, block.data_ptr(), False)
    g.implicit_step()
    got = g.get_field("u_tor")
    with np.errstate(over="ignore"):
        rhs = 1.5 * num
    want = _division(gdb, g, PM, rhs)
    for x, y, a in zip(got, want, rhs):
        _check(x[-1], y[-1], a)


def test_adjoint_quotient_is_the_division(gdb, model):
    import torch
    g = model
    num = np.stack([_numerators(g.nlm), _numerators(g.nlm)[::-1]])
    x, y = (torch.zeros(2 * NR * g.nlm, dtype=torch.float64, device="cuda") for _ in range(2))
    planes = [np.zeros(g.spec_shape()) for _ in range(2)]
    planes[0][-1], planes[1][-1] = num
    g.spectral_to_device(planes[0], planes[1], x)
    g.cnab2_adjoint("u_tor", 0, x, y)
    got = g.spectral_from_device(y)
    want = _division(gdb, g, PM, num)
    for a, b, v in zip(got, want, num):
        _check(a[-1], b[-1], v)
