"""FP64 Fock builds of bases whose functions do not fit one shared-memory panel of the orbital kernel (about 900 and more), with
factors that have one side or two (an indefinite density), against the oracle.  Sums over at most 1,500 functions and 20
points: 1e-11 of the largest element, the bar of the other FP64 builds."""
import numpy as np
import pytest

import oracle
from tcscf_b200 import api, grids

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nb,signs", [(909, (1, -1, 1, -1, 1, -1)), (1000, (1, 1, -1, -1, 1, -1)), (1023, (1, -1)), (1500, (1, 1, 1, 1))])
def test_bases_of_a_thousand_functions(ctx, nb, signs):
    basis = [(0.05 * 1.006 ** k, 1, 0, 0) for k in range(nb)]
    rng = np.random.default_rng(nb)
    gs = [grids.QuadratureGrid(rng.normal(size=(3, n)) * 1.5, rng.uniform(0.5, 1.5, n) / n) for n in (5, 20)]
    G1, G2 = [api.QMCGrid(ctx, g) for g in gs]
    for G in (G1, G2):
        G.setBasisFunctions(basis)
    C = np.linalg.qr(rng.normal(size=(nb, len(signs))))[0]
    D = ((C * np.array(signs) * rng.uniform(0.5, 1.5, len(signs))) @ C.T).astype(complex)
    h = rng.normal(size=(nb, nb))
    v = [oracle.basis_values(g.points, basis) for g in gs]
    F = oracle.compute_F(gs[0].points, gs[1].points, gs[1].weights, v[1], nb)
    Gr, Fr, Er = oracle.fock_build(F, v[0], gs[0].weights, D, h)
    Gg, Fg, Eg = api.fock_build(G1, G2, D, h)
    for G in (G1, G2):
        G.close()
    assert np.abs(Gg - np.reshape(Gr, Gg.shape)).max() <= 1e-11 * np.abs(Gr).max()
    assert abs(Eg - Er) <= 1e-11 * max(1.0, abs(Er))
