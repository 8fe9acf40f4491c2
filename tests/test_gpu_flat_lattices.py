"""The mat-vec on flat lattices, whose short axis has tiles and plans of its own: full tiles of columns and a remainder,
every z side up to 10 and every y side up to 8, in both precisions.

Bound: an FFT of M points rounds to about u log2(M) relative in the 2-norm (u: half a unit in the last place); there
and back, with the 3x3 multiply between, a factor 8 covers the constants."""
import math

import numpy as np
import pytest

from cases import random_field, rel
from ifdda import IFDDA_FP32, IFDDA_FP64

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(40, 3, n) for n in (1, 2, 3, 4, 5, 6, 8, 10)] +
                         [(40, n, 3) for n in (1, 2, 3, 4, 5, 6, 8)] + [(64, 2, 4), (33, 17, 1), (128, 1, 5)])
def test_matvec_flat(gctx, orc, dims):
    d, k0 = 11e-9, 2 * math.pi / 520e-9
    m = dims[0] * dims[1] * dims[2]
    x, b = random_field(3 * m, m), random_field(3 * m, m + 1)
    G = orc.greencalculfft(*dims, d, k0)
    conv = -orc.matvec(G, *dims, x, np.zeros_like(b))
    x /= np.linalg.norm(conv) / np.linalg.norm(b)  # the product as large as b
    ref = orc.matvec(G, *dims, x, b)
    g = gctx.green(*dims, d, k0)
    for prec, u in ((IFDDA_FP64, 2.0 ** -53), (IFDDA_FP32, 2.0 ** -24)):
        bound = 8 * u * math.log2(8 * m)
        assert rel(g.matvec(x, b, precision=prec), ref) < bound, prec
    g.close()
