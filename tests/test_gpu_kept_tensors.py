"""Builds from kept Fji / Vji tensors (real planes in the real-harmonic basis) at the edges of their kernels, against the
oracle: the transcorrelated build for every row-tile count (8 functions a tile), odd and even basis sizes,
unequal and zero spin counts, fewer points than blocks and densities that are not Hermitian; the
precompute-form Fock build around its two columns per lane; the reference layout on the host.  Bars:
1e-10 of the largest element (the transcorrelated sums chain five contractions of up to a few hundred terms
each), 1e-11 for the single-contraction builds."""
import numpy as np
import pytest

import oracle
from tcscf_b200 import api, ffi, grids
from tcscf_b200 import basis as wl

pytestmark = pytest.mark.gpu

U = dict(a=1.0, a12=1.0, terms=[((1, 0, 0), -0.5, -0.25)])


def _basis(s, p=0, d=0):
    return wl.expand(0, [0.5 * 1.5 ** k for k in range(s)]) + wl.expand(1, [0.7 * 1.6 ** k for k in range(p)]) + wl.expand(2, [1.1 * 1.7 ** k for k in range(d)])


def _complex(rng, *shape):
    return (rng.normal(size=shape) + 1j * rng.normal(size=shape)) * 0.3


def _grid(ctx, n, seed, basis, ndim=3, gradients=False):
    g = grids.qmc_grid(ndim, n, seed)
    G = api.QMCGrid(ctx, g)
    G.setBasisFunctions(basis, storeGradients=gradients)
    return g, G


@pytest.mark.parametrize("basis,nup,ndown,n1", [(_basis(1), 1, 1, 3), (_basis(2, 1), 1, 0, 1), (_basis(8), 0, 2, 40), (_basis(6, 1), 3, 2, 300),
                                                (_basis(7, 3), 2, 2, 64), (_basis(5, 4), 5, 4, 64), (_basis(12, 4), 2, 1, 700), (_basis(5, 5, 1), 1, 2, 64),
                                                (_basis(8, 6, 1), 4, 3, 200), (_basis(12, 5, 1), 20, 20, 20)])
def test_tc_build_row_tiles(ctx, basis, nup, ndown, n1):
    nb = len(basis)
    g1, G1 = _grid(ctx, n1, 61, basis, gradients=True)
    g2, G2 = _grid(ctx, 128, 62, basis)
    u, uo = ffi.ochi_struct(U["a"], U["a12"], U["terms"]), oracle.ochi(U["a"], U["a12"], U["terms"])
    ks = (ffi.K_TC_SCALAR_SAME, ffi.K_TC_SCALAR_OPPO, ffi.K_GRAD_U_SAME, ffi.K_GRAD_U_OPPO)
    t = [api.computeF(G1, G2, k, u, keep=True, copy=False)[1] for k in ks[:2]] + [api.computeV(G1, G2, k, u, keep=True, copy=False)[1] for k in ks[2:]]
    vals2 = oracle.basis_values(g2.points, basis)
    vals1, grads1 = oracle.basis_values(g1.points, basis, gradients=True)
    o = [oracle.compute_F(g1.points, g2.points, g2.weights, vals2, nb, k, uo) for k in ks[:2]]
    o += [oracle.compute_V(g1.points, g2.points, g2.weights, vals2, nb, k, uo) for k in ks[2:]]
    rng = np.random.default_rng(nb)
    occ = [_complex(rng, nup, nb), _complex(rng, ndown, nb)]
    D = _complex(rng, 2, nb, nb)   # any density, not that of the orbitals
    h = rng.normal(size=(nb, nb))
    got = api.tc_fock_build(G1, *t, nup, ndown, D, occ[0], occ[1], h)
    ref = oracle.tc_fock_build(*o, vals1, grads1, g1.weights, D, nup, ndown, occ[0], occ[1], h)
    for d in t + [G1, G2]:
        d.close()
    for a, b in zip(got[:3], ref[:3]):
        assert np.abs(a - b).max() <= 1e-10 * max(1.0, np.abs(b).max())
    assert abs(got[3] - ref[3]) <= 1e-10 * max(1.0, abs(ref[3]))


@pytest.mark.parametrize("dim2", [2, 3])
@pytest.mark.parametrize("nspin,basis,n1", [(1, _basis(1), 1), (2, _basis(4, 1), 5), (1, _basis(14, 6), 333), (2, _basis(12, 7), 65), (1, _basis(26, 11, 1), 129),
                                            (2, _basis(25, 13), 17)])
def test_precomputed_build_columns(ctx, nspin, basis, n1, dim2):
    nb = len(basis)
    g1, G1 = _grid(ctx, n1, 71, basis)
    g2, G2 = _grid(ctx, 96, 72, basis, ndim=dim2)
    F, t = api.computeF(G1, G2, keep=True)
    vals2 = oracle.basis_values(g2.points, basis)
    Fr = oracle.compute_F(g1.points, g2.points, g2.weights, vals2, nb)
    assert F.dtype == Fr.dtype and np.abs(F - Fr).max() <= 1e-11 * np.abs(Fr).max()
    rng = np.random.default_rng(nb)
    D = _complex(rng, nspin, nb, nb)
    h = rng.normal(size=(nb, nb))
    got = api.fock_build_precomputed(G1, t, D, h)
    ref = oracle.fock_build(Fr, oracle.basis_values(g1.points, basis), g1.weights, D, h)
    for d in (t, G1, G2):
        d.close()
    for a, b in zip(got[:2], ref[:2]):
        assert np.abs(a - np.reshape(b, a.shape)).max() <= 1e-11 * np.abs(b).max()
    assert abs(got[2] - ref[2]) <= 1e-11 * max(1.0, abs(ref[2]))
