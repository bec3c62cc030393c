"""Allocation-free syntheses of several handles in flight at once: every handle
has a stream of its own and the call returns before its kernels end, so nothing
may pass between them.
"""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_two_handles_in_flight(gdb):
    import torch
    sizes = ((31, 48, 96, 32, 3), (63, 96, 192, 40, 4), (40, 62, 125, 17, 9))
    rng = np.random.default_rng(5)
    jobs = []
    for lmax, nlat, nlon, nr, nf in sizes:
        g = gdb.SHTnsKitConfig(lmax, nlat, nlon, nr)
        coef = torch.from_numpy(rng.standard_normal((nf, 2, nr, g.nlm))).cuda()
        want, got = (torch.empty((nf, nr, nlat, nlon), dtype=torch.float64, device="cuda") for _ in range(2))
        jobs.append((g, nf, coef, want, got))

    def run(job, out):
        g, nf, coef = job[:3]
        g._check(g.lib.gd_spectral_to_physical_noalloc(g.h, nf, ctypes.c_void_p(coef.data_ptr()),
                                                       ctypes.c_void_p(out.data_ptr())))

    for job in jobs:
        torch.cuda.synchronize()
        run(job, job[3])
        job[0].synchronize()
    for _ in range(30):
        for job in jobs:
            job[4].zero_()
        torch.cuda.synchronize()
        for job in jobs * 3:
            run(job, job[4])
        for job in jobs:
            job[0].synchronize()
        for job in jobs:
            assert torch.equal(job[3], job[4])
    for job in jobs:
        job[0].close()
