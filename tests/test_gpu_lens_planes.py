"""The far fields behind the pupil (the lens's, and both sides without a lens) with every share of the planes a block
can take: few and many planes, even and uneven shares, small and large pupils, against the oracle's 2-D FFTs.

Bound: N = nx ny nz terms of equal size per value, each with a few rounded factors (16 N 2^-53 relative), at least
1e-12 for the phases, whose arguments reach some 50 radians and pass through sines, cosines and the lens's rotation."""
import math

import numpy as np
import pytest

from cases import random_field, rel

pytestmark = pytest.mark.gpu
K0 = 2 * math.pi / 632.8e-9


def _field(nx, ny, nz, d):
    k, j, i = np.meshgrid(np.arange(nz), np.arange(ny), np.arange(nx), indexing="ij")
    xs, ys, zs = ((a.ravel() + 0.5 - m / 2) * d for a, m in ((i, nx), (j, ny), (k, nz)))
    n = nx * ny * nz
    return xs, ys, zs, random_field(3 * n, nz), max(16 * n * 2.0 ** -53, 1e-12)


@pytest.mark.parametrize("nz,d,nfft2d", [(1, 20e-9, 64), (2, 20e-9, 64), (3, 20e-9, 64), (7, 20e-9, 64),
                                         (17, 20e-9, 64), (24, 20e-9, 64), (33, 20e-9, 64), (17, 200e-9, 256),
                                         (3, 200e-9, 512), (17, 200e-9, 512)])
def test_lens_far_field(gctx, orc, nz, d, nfft2d):
    nx, ny = 6, 4
    xs, ys, zs, ff, bound = _field(nx, ny, nz, d)
    E0, _ = orc.irradiance(1.0, 6328e-9)
    args = (nx, ny, nz, d, K0, xs, ys, zs, ff * 1e-22, E0, 10.0, 30.0, 0.3)
    ref = orc.holography(*args, nfft2d, 0.9, 100.0, 0.0, nside=0)
    got = gctx.holography(*args, nfft2d=nfft2d, numaper=0.9, gross=100.0, zlens=0.0, nside=0)
    assert got["nstop"] == ref["nstop"] == 0, (got["infostr"], ref["infostr"])
    assert rel(got["fourier"][:3], ref["fourier"][:3]) < bound


@pytest.mark.parametrize("nz,nfft2d", [(1, 512), (2, 512), (17, 256), (17, 512)])
def test_far_field_of_a_large_pupil(gctx, orc, nz, nfft2d):
    nx, ny, d = 6, 4, 200e-9
    xs, ys, zs, ff, bound = _field(nx, ny, nz, d)
    args = (nx, ny, nz, d, xs, ys, zs, ff, K0, 1.0, 20.0, 30.0, nfft2d, 20, 40)
    ref, got = orc.farfield_fft(*args), gctx.farfield_fft(*args)
    assert got["imaxk0"] == ref["imaxk0"]
    assert rel(got["kpos"], ref["kpos"]) < bound and rel(got["kneg"], ref["kneg"]) < bound
