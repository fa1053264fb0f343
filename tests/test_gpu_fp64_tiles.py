"""The FP64 contraction and its Coulomb row sums at the edges of their tiles, against the oracle: one grid as
r1 and r2 (the symmetric contraction, whose row sums come from kCoulombLowerFp64 in chunks of 64 points)
and two grids (the full one).  Every sum has at most 700 terms of one sign pattern, so FP64 rounding
stays below 700 eps = 1.6e-13 of the sum of magnitudes; the bar is 1e-11 of the largest element of G, the
margin covering cancellation between the Coulomb and exchange parts."""
import numpy as np
import pytest

import oracle
from tcscf_b200 import api, ffi, grids
from tcscf_b200 import basis as wl

pytestmark = pytest.mark.gpu

TOL = 1e-11


def _grid(n, seed):
    rng = np.random.default_rng(seed)
    return grids.QuadratureGrid(rng.normal(size=(3, n)) * 1.5, rng.uniform(0.5, 1.5, n) / n)


def _density(basis, nocc, seed):
    U = wl.real_harmonic_unitary(basis)
    C = U.T @ (np.random.default_rng(seed).normal(size=(len(basis), nocc)) * 0.3)
    return np.ascontiguousarray(C @ C.conj().T)


def _check(ctx, g1, g2, basis, nocc):
    D = _density(basis, nocc, 7)
    h = np.ones((len(basis),) * 2)
    A = api.QMCGrid(ctx, g1)
    A.setBasisFunctions(basis)
    B = A
    if g2 is not g1:
        B = api.QMCGrid(ctx, g2)
        B.setBasisFunctions(basis)
    G, _, E = api.fock_build(A, B, D, h, precision=ffi.PREC_FP64)
    A.close()
    if B is not A:
        B.close()
    F = oracle.compute_F(g1.points, g2.points, g2.weights, oracle.basis_values(g2.points, basis), len(basis))
    Gr, _, Er = oracle.fock_build(F, oracle.basis_values(g1.points, basis), g1.weights, D, h)
    assert np.abs(G - Gr).max() <= TOL * np.abs(Gr).max()
    assert abs(E - Er) <= TOL * max(abs(Er), 1.0)


@pytest.mark.parametrize("n", [2, 31, 63, 64, 65, 127, 128, 129, 191, 192, 193, 257, 700])
def test_symmetric_rows_at_tile_edges(ctx, n):
    g = _grid(n, n)
    _check(ctx, g, g, wl.expand(0, [0.7, 1.9]) + wl.expand(1, [1.1]), 2)
