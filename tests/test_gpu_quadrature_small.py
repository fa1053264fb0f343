"""S and H by quadrature on both sides of the line between the block-per-element form (small sums) and the tiled one, against
the oracle; and the number of kernels a small call launches (one: a second launch is what such a call cannot
hide).  Sums of at most 86,000 terms of one scale: rounding below sqrt(n) eps to n eps = 2e-11 of the
largest element; the bar is that of test_gpu_quadrature_tiles.py, 1e-11."""
import ctypes as C

import numpy as np
import pytest
import torch

import oracle
from tcscf_b200 import api, ffi, grids
from tcscf_b200 import basis as wl

pytestmark = pytest.mark.gpu


def _basis(counts):
    return [f for l, k in enumerate(counts) for f in wl.expand(l, [0.5 * 1.2 ** q for q in range(k)])]


def _grid(n):
    rng = np.random.default_rng(n)
    return grids.QuadratureGrid(rng.normal(size=(3, n)) * 1.5, rng.uniform(0.5, 1.5, n) / n)


# the line: n (nb^2 + 100) = 610,000 with H, n (nb^2 + 20) = 1,800,000 without, and nb = 48
@pytest.mark.parametrize("counts", [(1,), (2, 1), (6, 2), (10, 5, 1), (10, 5, 3), (14, 8, 2), (15, 8, 2)])
@pytest.mark.parametrize("side", [0, 1])
@pytest.mark.parametrize("with_h", [True, False])
def test_both_forms_at_their_line(ctx, counts, side, with_h):
    basis = _basis(counts)
    nb = len(basis)
    n = (610000 // (nb * nb + 100) if with_h else 1800000 // (nb * nb + 20)) + side
    g = _grid(n)
    v, gr = oracle.basis_values(g.points, basis, gradients=True)
    Sr, Hr = oracle.quadrature_overlap_core(g.points, g.weights, v, gr, 3)
    G = api.QMCGrid(ctx, g)
    G.setBasisFunctions(basis, storeGradients=True)
    null = C.POINTER(C.c_double)()
    for entry in (ffi.lib().tcscf_overlap_core_quadrature, ffi.lib().tcscf_overlap_core_quadrature_static):
        S, H = np.full((nb, nb), np.nan, complex), np.full((nb, nb), np.nan, complex)
        ffi.check(entry(ctx.handle, G.id, 3, ffi.dptr(S), ffi.dptr(H) if with_h else null), ctx.handle)
        assert np.abs(S - Sr).max() <= 1e-11 * np.abs(Sr).max()
        if with_h:
            assert np.abs(H - Hr).max() <= 1e-11 * np.abs(Hr).max()
    G.close()


@pytest.mark.parametrize("n,counts", [(50, (1,)), (500, (8, 4)), (2500, (2, 1))])
def test_a_small_call_is_one_launch(ctx, n, counts):
    torch.zeros(1, device="cuda")
    G = api.QMCGrid(ctx, _grid(n))
    G.setBasisFunctions(_basis(counts), storeGradients=True)
    api.overlap_core_quadrature(G, 3)
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as p:
        api.overlap_core_quadrature(G, 3)
        torch.cuda.synchronize()
    G.close()
    names = [e.name for e in p.events() if "kQuad" in e.name]
    if not names:
        pytest.skip("no kernel activity records here")
    assert len(names) == 1, names
