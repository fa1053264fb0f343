"""The split-BF16 contraction at the edges of its r2 blocks and of its T and X buffers (one, two, three and more 64-point
blocks per work item, full and partly filled last ones), one and two grids, both column tiles, against the FP64 path.

A product carries the 24-bit rounding of psi1, psi2, X and Vt and the FP32 kernel value: below 8 x 2^-24 = 4.8e-7 of the
sum of magnitudes.  The bar is ten times that of the largest |G| element, the margin covering cancellation between
the Coulomb and exchange parts."""
import numpy as np
import pytest

from tcscf_b200 import api, ffi
from tcscf_b200 import basis as wl

from .test_gpu_fp64_tiles import _density, _grid

pytestmark = pytest.mark.gpu

TOL = 10 * 8 * 2.0 ** -24


@pytest.mark.parametrize("nb,nocc", [(5, 2), (64, 16), (65, 3), (128, 32)])
@pytest.mark.parametrize("n1,n2", [(64, 0), (128, 0), (129, 0), (320, 0), (65, 1), (128, 63), (128, 64), (130, 65), (257, 128), (31, 193), (128, 257)])
def test_blocks_and_buffers(ctx, nb, nocc, n1, n2):
    basis = wl.expand(0, [0.5 * 1.03 ** k for k in range(nb)])
    D = _density(basis, nocc, 7)
    h = np.zeros((nb, nb))
    A = api.QMCGrid(ctx, _grid(n1, n1))
    A.setBasisFunctions(basis)
    B = A
    if n2:
        B = api.QMCGrid(ctx, _grid(n2, 1000 + n2))
        B.setBasisFunctions(basis)
    G64 = api.fock_build(A, B, D, h, precision=ffi.PREC_FP64)[0]
    G = api.fock_build(A, B, D, h, precision=ffi.PREC_BF16X3)[0]
    A.close()
    if n2:
        B.close()
    assert np.abs(G - G64).max() <= TOL * np.abs(G64).max()
