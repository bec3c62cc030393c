"""The tensor-core synthesis pipeline: repeated calls give the same bits (two
issuing warps, in-place splitting, slot rings), and every call agrees with the
FP64 kernels, at sizes around its tiles: one degree past a 32-deep chunk of a
parity, orders without odd degrees, column tiles with a remainder, a last
colatitude tile of a few rows.
"""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "geodynamo.jl_b200"))
import workloads  # noqa: E402

pytestmark = pytest.mark.gpu
TOL = 5e-6  # the bound of the mixed path's single transforms


@pytest.mark.parametrize("lmax,nlat,nlon,nr,nf", [
    (1, 4, 6, 3, 1),        # one chunk, one degree per parity
    (7, 10, 24, 33, 2),     # 33 shells: a second column tile of one
    (63, 66, 128, 5, 4),    # full chunks of 32 degrees
    (64, 262, 192, 32, 3),  # one degree past them; three rows in the second colatitude tile
    (130, 132, 288, 65, 4),
])
def test_synthesis_repeats_and_agrees(gdb, lmax, nlat, nlon, nr, nf):
    a = gdb.SHTnsKitConfig(lmax, nlat, nlon, nr, precision="mixed")
    b = gdb.SHTnsKitConfig(lmax, nlat, nlon, nr)
    re, im = workloads.transform_batch(lmax, lmax, nr, max(nf, 2), seed=lmax)
    s, v = a.synth_scalar(re[:nf], im[:nf]), a.synth_vector(re[0], im[0], re[1], im[1])
    for _ in range(20):
        assert np.array_equal(s, a.synth_scalar(re[:nf], im[:nf]))
        w = a.synth_vector(re[0], im[0], re[1], im[1])
        assert np.array_equal(v[0], w[0]) and np.array_equal(v[1], w[1])
    ref = b.synth_scalar(re[:nf], im[:nf])
    assert np.max(np.abs(s - ref)) <= TOL * np.max(np.abs(ref))
    rv = b.synth_vector(re[0], im[0], re[1], im[1])
    for x, y in zip(v, rv):
        assert np.max(np.abs(x - y)) <= TOL * max(np.max(np.abs(rv[0])), np.max(np.abs(rv[1])))
    a.close(); b.close()
