"""Fji and Vji copied to the host in the reference's layout in pieces of at most 1 GiB: two whole pieces and a short one, whose rows
around the seams must be those of the same points computed by themselves (the same kernels on other tiles: 1e-13 of the
largest element)."""
import numpy as np
import pytest

from tcscf_b200 import api, ffi, grids
from tcscf_b200 import basis as wl

pytestmark = pytest.mark.gpu

BASIS = wl.expand(0, [0.5 * 1.3 ** k for k in range(16)]) + wl.expand(1, [0.6 * 1.4 ** k for k in range(6)]) + wl.expand(2, [0.8 * 1.5 ** k for k in range(6)])  # 64


@pytest.mark.parametrize("vector", [False, True])
def test_pieces_of_the_host_copy(ctx, vector):
    row = 64 * 64 * 16 * (3 if vector else 1)   # bytes of a point, complex
    piece = (1 << 30) // row
    n1 = 2 * piece + 5
    g1, g2 = grids.qmc_grid(3, n1, 5), grids.qmc_grid(3, 16, 6)
    u = ffi.ochi_struct(1.0, 1.0, [((1, 0, 0), -0.5, -0.25)])

    def compute(g):
        G1, G2 = api.QMCGrid(ctx, g), api.QMCGrid(ctx, g2)
        for G in (G1, G2):
            G.setBasisFunctions(BASIS)
        t = api.computeV(G1, G2, ffi.K_GRAD_U_SAME, u) if vector else api.computeF(G1, G2)
        G1.close()
        G2.close()
        return t

    rows = np.unique(np.concatenate([[0, piece - 1, piece, piece + 1, 2 * piece - 1, 2 * piece, n1 - 1], np.random.default_rng(1).integers(0, n1, 40)]))
    whole = compute(g1)[rows]
    part = compute(grids.subset(g1, rows))
    assert np.abs(whole - part).max() <= 1e-13 * np.abs(part).max()
