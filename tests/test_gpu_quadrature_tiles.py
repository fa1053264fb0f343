"""S and H by quadrature at the edges of the kernel's 32 x 32 tiles and 8-point groups, from context scratch and from the fixed
array, against the oracle.  Sums of at most 300 terms: rounding below 300 eps = 7e-14 of the sum of
magnitudes; the bar is 1e-11 of the largest element (cancellation between kinetic and nuclear terms)."""
import ctypes as C

import numpy as np
import pytest

import oracle
from tcscf_b200 import api, ffi, grids
from tcscf_b200 import basis as wl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,counts", [(1, (1, 0, 0)), (7, (3, 1, 1)), (8, (8, 8, 0)), (9, (2, 10, 0)), (33, (3, 10, 0)), (300, (5, 5, 9)), (257, (30, 10, 10))])
def test_overlap_core_tile_edges(ctx, n, counts):
    basis = [f for l, k in enumerate(counts) for f in wl.expand(l, [0.5 * 1.2 ** q for q in range(k)])]
    rng = np.random.default_rng(n)
    g = grids.QuadratureGrid(rng.normal(size=(3, n)) * 1.5, rng.uniform(0.5, 1.5, n) / n)
    v, gr = oracle.basis_values(g.points, basis, gradients=True)
    Sr, Hr = oracle.quadrature_overlap_core(g.points, g.weights, v, gr, 3)
    G = api.QMCGrid(ctx, g)
    G.setBasisFunctions(basis, storeGradients=True)
    nb = len(basis)
    S, H = api.overlap_core_quadrature(G, 3)
    Ss, Hs = np.empty((nb, nb), complex), np.empty((nb, nb), complex)
    ffi.check(ffi.lib().tcscf_overlap_core_quadrature_static(ctx.handle, G.id, 3, ffi.dptr(Ss), ffi.dptr(Hs)), ctx.handle)
    S0 = np.empty((nb, nb), complex)
    ffi.check(ffi.lib().tcscf_overlap_core_quadrature(ctx.handle, G.id, 3, ffi.dptr(S0), C.POINTER(C.c_double)()), ctx.handle)
    G.close()
    for a, r in ((S, Sr), (Ss, Sr), (S0, Sr), (H, Hr), (Hs, Hr)):
        assert np.abs(a - r).max() <= 1e-11 * np.abs(r).max()


# per-point tables: one function of the highest l (the largest tables, the most points a block would take), one point
# over a block's share, and many functions (fewest points a block)
@pytest.mark.parametrize("n,basis", [(3, [(0.8, 13, 12, 0)]), (129, [(0.8, 13, 12, 0)]), (65, wl.expand(0, [0.7])), (33, wl.expand(12, [0.9, 1.4])),
                                     (17, wl.expand(0, [0.5 * 1.02 ** k for k in range(150)]))])
def test_basis_values_and_gradients_by_block(ctx, n, basis):
    rng = np.random.default_rng(n)
    g = grids.QuadratureGrid(rng.normal(size=(3, n)) * 1.5, np.ones(n))
    v, gr = oracle.basis_values(g.points, basis, gradients=True)
    G = api.QMCGrid(ctx, g)
    G.setBasisFunctions(basis, storeGradients=True)
    a, b = G.basisValues, G.basisGradients
    G.close()
    # sums of a few dozen products of functions good to a few eps; the l = 12 recurrence loses another digit
    assert np.abs(a - v).max() <= 1e-12 * np.abs(v).max()
    assert np.abs(b - gr).max() <= 1e-12 * np.abs(gr).max()
