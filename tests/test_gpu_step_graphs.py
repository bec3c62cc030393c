"""Graphs of the FP64 step: a new handle, and one whose dt has just changed, steps
through the chain's graph; after 64 steps with the same settings a small model's
phases run side by side.  Both forms give the bits of the eager chain (per-kernel
timing on), also where a start is restored after the change of form.
"""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "geodynamo.jl_b200"))
import workloads  # noqa: E402

pytestmark = pytest.mark.gpu
AFTER = 64


def _model(gdb, lmax, nlat, nlon, nr, timed=False, scheme="cnab2", **kw):
    g = gdb.SHTnsKitConfig(lmax, nlat, nlon, nr, dt=1e-6, **kw)
    g.set_scheme(scheme)
    for k, (a, b) in workloads.seeded_state(lmax, lmax, nr, seed=4, amp=1.0).items():
        g.set_field(k, a, b)
    g.profile_enable(timed)
    return g


def _all(g):
    return [x for k in g.field_names() for x in g.get_field(k) + g.get_nl(k)] + \
           [g.get_grid(k) for k in ("u_th", "w_ph", "b_th", "j_ph", "t", "tadv", "vadv_th", "ind_ph")]


@pytest.mark.parametrize("lmax,nlat,nlon,nr,kw", [
    (31, 48, 96, 32, dict(bc_mode=2)),
    (20, 34, 48, 7, dict(bc_mode=0, ab_mode=1)),
    (15, 24, 48, 12, dict(bc_mode=0, scheme="eab2")),
    (15, 24, 48, 12, dict(bc_mode=0, scheme="erk2")),
    (15, 24, 48, 12, dict(bc_mode=2, geometry="ball")),
    (15, 24, 50, 12, dict(bc_mode=2, segments=2)),
    (127, 192, 384, 42, dict(bc_mode=2)),   # the largest four-component buffer that forks
    (127, 192, 384, 43, dict(bc_mode=2)),   # just above: one chain
])
def test_both_forms_equal_the_eager_chain(gdb, lmax, nlat, nlon, nr, kw):
    out = []
    for timed in (False, True):
        g = _model(gdb, lmax, nlat, nlon, nr, timed, **kw)
        got = []
        for n in (AFTER - 1, 1, 1, 2, 3):  # the last chain step, then both banks side by side
            g.step(n)
            got += _all(g)
        g.set_dt(5e-7)
        g.step(3)
        out.append(got + _all(g))
        g.close()
    for x, y in zip(*out):
        assert np.array_equal(x, y, equal_nan=True)


def test_which_steps_take_the_chain(gdb):
    g = _model(gdb, 31, 48, 96, 32, bc_mode=2)
    new = g.step_kernels()
    g.step(3)
    chain = g.step_kernels()
    g.step(AFTER)
    side = g.step_kernels()
    assert side < chain and new == chain  # the side-by-side form joins two phi transforms a vector
    g.set_dt(5e-7)
    assert g.step_kernels() == chain
    g.close()


def test_restored_start_bootstraps_again(gdb):
    import torch
    g = _model(gdb, 15, 24, 48, 12, bc_mode=2)
    buf = torch.empty((g.snapshot_bytes() + 7) // 8, dtype=torch.float64, device="cuda")
    g.snapshot(buf)
    out = []
    for _ in range(2):
        g.step(3)
        out.append(_all(g))
        g.step(AFTER + 2)
        out[-1] += _all(g)
        g.restore(buf)
    for x, y in zip(*out):
        assert np.array_equal(x, y, equal_nan=True)
    g.close()


def test_memory_of_the_branches_comes_with_them(gdb):
    lmax, nlat, nlon, nr = 31, 48, 96, 32
    g = _model(gdb, lmax, nlat, nlon, nr, bc_mode=2)
    h = gdb.SHTnsKitConfig(lmax, nlat, nlon, nr, dt=1e-6, bc_mode=2, composition=1)  # composition: always the chain
    components = 16 * nr * (lmax + 1) * nlat
    h.step(1)
    g.step(AFTER)
    before, other = g.device_bytes(), h.device_bytes()
    g.step(1)
    h.step(AFTER + 1)
    assert g.device_bytes() == before + 8 * components and h.device_bytes() == other
    g.step(4)
    assert g.device_bytes() == before + 8 * components
    g.close()
    h.close()
