"""The mat-vec at every compiled FFT length on every axis, with the other axes
small and uneven: tiles with a single pair of columns or a ragged remainder,
the unpaired frequencies 0 and n, every pass plan, both tile shapes.

Bound: an FFT of M points rounds to about u log2(M) relative in the 2-norm (u:
half a unit in the last place); there and back, with the 3x3 multiply between,
a factor 8 covers the constants."""
import math

import numpy as np
import pytest

from cases import random_field, rel
from ifdda import IFDDA_FP32, IFDDA_FP64

pytestmark = pytest.mark.gpu

SIDES = [1, 2, 3, 4, 5, 6, 8, 10, 12, 16, 20, 24, 32, 40, 48, 64, 80, 96, 128, 160, 192, 256, 320]


@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("n", SIDES)
def test_matvec_every_length_on_every_axis(gctx, orc, n, axis):
    dims = [(n, 3, 5), (5, n, 3), (10, 3, n)][axis]
    d, k0 = 11e-9, 2 * math.pi / 520e-9
    m = dims[0] * dims[1] * dims[2]
    x, b = random_field(3 * m, n), random_field(3 * m, n + 1)
    G = orc.greencalculfft(*dims, d, k0)
    conv = -orc.matvec(G, *dims, x, np.zeros_like(b))
    x /= np.linalg.norm(conv) / np.linalg.norm(b)  # the product as large as b
    ref = orc.matvec(G, *dims, x, b)
    g = gctx.green(*dims, d, k0)
    for prec, u in ((IFDDA_FP64, 2.0 ** -53), (IFDDA_FP32, 2.0 ** -24)):
        bound = 8 * u * math.log2(8 * m)
        for shape in (0, 1):
            zv, yv = (shape if 2 * s >= 64 else 0 for s in (dims[2], dims[1]))
            g.set_tiles(prec, zv, yv)
            assert rel(g.matvec(x, b, precision=prec), ref) < bound, (prec, shape)
    g.close()
