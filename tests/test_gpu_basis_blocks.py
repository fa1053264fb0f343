"""Basis values and gradients where the points a block takes change: one point a block, the first size with two, the most
points a block holds by its threads (1 function) and by its shared memory (l = 12), and a last block partly filled; against
the oracle with the bars of test_gpu_quadrature_tiles.py (1e-12 of the largest element)."""
import numpy as np
import pytest

import oracle
from tcscf_b200 import api, grids
from tcscf_b200 import basis as wl

pytestmark = pytest.mark.gpu

ONE, HIGH = wl.expand(0, [0.7]), wl.expand(0, [0.8]) + wl.expand(12, [0.9])
MANY = wl.expand(0, [0.5 * 1.02 ** k for k in range(150)])


@pytest.mark.parametrize("n,basis", [(1, ONE), (296, ONE), (297, ONE), (593, ONE), (75776, ONE), (75777, ONE), (1, HIGH), (297, HIGH), (9000, HIGH),
                                     (25000, HIGH), (296, MANY), (2369, MANY)])
def test_points_per_block(ctx, n, basis):
    rng = np.random.default_rng(n)
    g = grids.QuadratureGrid(rng.normal(size=(3, n)) * 1.5, np.ones(n))
    v, gr = oracle.basis_values(g.points, basis, gradients=True)
    G = api.QMCGrid(ctx, g)
    G.setBasisFunctions(basis)
    a = G.basisValues
    G.setBasisFunctions(basis, storeGradients=True)
    b, c = G.basisValues, G.basisGradients
    G.close()
    assert np.array_equal(a, b)
    assert np.abs(b - v).max() <= 1e-12 * np.abs(v).max()
    assert np.abs(c - gr).max() <= 1e-12 * np.abs(gr).max()
