"""Buffers of the checkpointed gradient: runs of other lengths and checkpoint
distances on one handle give what a new handle gives, and a large pullback's
scratch is not kept from the rest of the device.
"""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "geodynamo.jl_b200"))
import workloads  # noqa: E402

pytestmark = pytest.mark.gpu


def _start(g, seed=4):
    for k, (a, b) in workloads.seeded_state(g.lmax, g.lmax, g.nr, seed=seed, amp=0.3).items():
        g.set_field(k, a, b)


def _gradient(g, steps, every, full):
    g.temperature_forward(steps, every)
    lam = g.get_field("temp")
    return g.temperature_pullback_full(*lam) if full else g.temperature_pullback(*lam)


def _flat(x):
    return [x] if isinstance(x, np.ndarray) else [z for y in x for z in _flat(y)]


def test_runs_of_other_lengths_on_one_handle(gdb):
    import torch
    cfg = dict(lmax=15, nlat=24, nlon=48, nr=12, dt=1e-5)
    runs = [(7, 2, True), (3, 1, True), (9, 4, False), (1, 1, True), (9, 9, True), (9, 4, False), (7, 2, True)]
    g = gdb.SHTnsKitConfig(**cfg)
    _start(g)
    buf = torch.empty((g.snapshot_bytes() + 7) // 8, dtype=torch.float64, device="cuda")
    g.snapshot(buf)
    for run in runs:
        g.restore(buf)
        got = _flat(_gradient(g, *run))
        fresh = gdb.SHTnsKitConfig(**cfg)
        _start(fresh)
        want = _flat(_gradient(fresh, *run))
        fresh.close()
        assert len(got) == len(want) and np.any(want[0])  # (one step: no velocity gradient)
        for x, y in zip(got, want):
            assert np.array_equal(x, y), run
    g.close()


def test_large_scratch_is_given_back(gdb):
    import torch
    steps = 120  # four grids of 4.9 MB a step: 2.3 GB, more than is kept
    g = gdb.SHTnsKitConfig(63, 96, 192, 33, dt=1e-6)
    _start(g)
    g.step(70)  # everything a run itself makes
    _gradient(g, 2, 1, True)
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    first = _flat(_gradient(g, steps, steps, True))
    after = torch.cuda.mem_get_info()[0]
    assert before - after < 256 << 20
    assert all(np.all(np.isfinite(x)) for x in first)
    g.close()
