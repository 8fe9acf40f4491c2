"""The pupil far field (both sides) with fewer planes than the shares a block
cuts them into, exactly as many, and remainders: against the oracle's 2-D FFT.
Bound: N = nx ny nz terms of equal size per value, each with a few rounded
factors, squared for the Poynting vector: 16 N 2^-53 relative, at least 1e-13
for the angles' sines and cosines."""
import math

import numpy as np
import pytest

from cases import random_field, rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nz", [1, 5, 15, 16, 17, 33])
def test_farfield_fft_planes(gctx, orc, nz):
    nx, ny, d, k0 = 6, 4, 20e-9, 2 * math.pi / 632.8e-9
    n = nx * ny * nz
    k, j, i = np.meshgrid(np.arange(nz), np.arange(ny), np.arange(nx), indexing="ij")
    xs, ys, zs = ((a.ravel() + 0.5 - m / 2) * d for a, m in ((i, nx), (j, ny), (k, nz)))
    ff = random_field(3 * n, nz)
    args = (nx, ny, nz, d, xs, ys, zs, ff, k0, 1.0, 20.0, 30.0, 64, 20, 40)
    ref, got = orc.farfield_fft(*args), gctx.farfield_fft(*args)
    assert got["imaxk0"] == ref["imaxk0"]
    bound = max(16 * n * 2.0 ** -53, 1e-13)
    assert rel(got["kpos"], ref["kpos"]) < bound and rel(got["kneg"], ref["kneg"]) < bound
