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


# every column-tile count of the direct form (8-column tiles: 1 to 8, 10, 12 to 16) with full and partly filled
# last tiles, odd and even row lengths, and the ranks where the row-tile count changes
@pytest.mark.parametrize("nb,nocc", [(1, 1), (7, 2), (8, 3), (9, 4), (17, 5), (25, 9), (33, 6), (40, 5), (41, 21), (49, 3), (57, 13), (64, 64),
                                     (65, 8), (73, 30), (88, 20), (97, 12), (105, 17), (113, 33), (120, 18), (128, 47), (78, 78)])
def test_column_tiles_and_ranks(ctx, nb, nocc):
    basis = wl.expand(0, [0.5 * 1.03 ** k for k in range(nb)])
    g = _grid(193, nb)
    _check(ctx, g, g, basis, nocc)
    _check(ctx, g, _grid(97, nb + 1), basis, nocc)


@pytest.mark.parametrize("n1,n2", [(1, 1), (1, 70), (129, 31), (64, 33), (255, 257)])
def test_two_grids_at_tile_edges(ctx, n1, n2):
    _check(ctx, _grid(n1, n1), _grid(n2, 1000 + n2), wl.expand(0, [0.7, 1.9, 4.1]) + wl.expand(1, [1.1, 2.6]), 3)


# precompute form: one column group, several, and a partly filled last one, scalar and transcorrelated kernels
@pytest.mark.parametrize("ns", [3, 8, 15, 16, 23])
@pytest.mark.parametrize("kernel", [ffi.K_INV_R12, ffi.K_TC_SCALAR_SAME, ffi.K_GRAD_U_OPPO])
def test_precompute_column_groups(ctx, ns, kernel):
    basis = wl.expand(0, [0.4 * 1.1 ** k for k in range(ns)])
    terms = [((1, 0, 0), -0.4, -0.2), ((1, 1, 1), 0.1, 0.05)]
    g1, g2 = _grid(67, 3), _grid(101, 4)
    A, B = api.QMCGrid(ctx, g1), api.QMCGrid(ctx, g2)
    A.setBasisFunctions(basis)
    B.setBasisFunctions(basis)
    u, uo = ffi.ochi_struct(0.9, 0.8, terms), oracle.ochi(0.9, 0.8, terms)
    vals = oracle.basis_values(g2.points, basis)
    if kernel == ffi.K_GRAD_U_OPPO:
        got, ref = api.computeV(A, B, kernel, u), oracle.compute_V(g1.points, g2.points, g2.weights, vals, ns, kernel, uo)
    else:
        got, ref = api.computeF(A, B, kernel, u), oracle.compute_F(g1.points, g2.points, g2.weights, vals, ns, kernel, uo)
    A.close()
    B.close()
    assert np.abs(got - ref).max() <= TOL * np.abs(ref).max()
