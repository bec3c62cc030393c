"""The field-struct transforms write into the caller's arrays when these are plain
(contiguous float64) and through a copy when not: same values either way, and
the caller's array objects stay the ones it has.
"""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "geodynamo.jl_b200"))
import workloads  # noqa: E402

pytestmark = pytest.mark.gpu


def _odd(a, how):
    """An array of a's shape that the library cannot write directly."""
    if how == "strided":
        return np.zeros(a.shape[:-1] + (2 * a.shape[-1],))[..., ::2]
    if how == "float32":
        return np.zeros(a.shape, dtype=np.float32)
    return np.zeros(a.shape[::-1]).T  # other order


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("how", ["strided", "float32", "order"])
def test_plain_and_other_arrays(gdb, precision, how):
    g = gdb.SHTnsKitConfig(20, 34, 48, 7, precision=precision)
    re, im = workloads.transform_batch(20, 20, 7, 2, seed=1)
    re[:, :, 0] = im[:, :, 0] = 0.0
    a, b = gdb.SHTnsSpectralField(g), gdb.SHTnsSpectralField(g)
    for f, k in ((a, 0), (b, 1)):
        f.data_real[...], f.data_imag[...] = re[k], im[k]
    out = []
    for plain in (True, False):
        vec, phys = gdb.SHTnsVectorField(g), gdb.SHTnsPhysicalField(g)
        tor, pol, s = (gdb.SHTnsSpectralField(g) for _ in range(3))
        if not plain:
            for o in (vec.theta_component, vec.phi_component, phys):
                o.data = _odd(o.data, how)
            for o in (tor, pol, s):
                o.data_real, o.data_imag = _odd(o.data_real, how), _odd(o.data_imag, how)
        held = [vec.theta_component.data, vec.phi_component.data, phys.data, tor.data_real, tor.data_imag,
                pol.data_real, pol.data_imag, s.data_real, s.data_imag]
        gdb.shtnskit_vector_synthesis(a, b, vec)
        gdb.shtnskit_spectral_to_physical(a, phys)
        if plain:
            grids = [x.copy() for x in held[:3]]
        for x, y in zip(held[:3], grids):
            x[...] = y  # the same analysis input for both
        gdb.shtnskit_vector_analysis(vec, tor, pol)
        gdb.shtnskit_physical_to_spectral(phys, s)
        out.append([np.array(x) for x in held])
    for x, y in zip(out[0][:3], out[1][:3]):
        assert np.array_equal(x.astype(y.dtype), y)
    if how != "float32":
        for x, y in zip(*out):
            assert np.array_equal(x, y)
    g.close()
