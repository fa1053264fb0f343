"""Device memory of destroyed tensors: it is back with the device when the call returns, up to what the context's pool keeps
(4 GiB), and what the pool keeps does not starve the context's own scratch."""
import gc

import pytest
import torch

from tcscf_b200 import api, grids
from tcscf_b200 import basis as wl

pytestmark = pytest.mark.gpu

GIB, MIB = 1 << 30, 1 << 20
BASIS = wl.expand(0, [0.5 * 1.3 ** k for k in range(16)]) + wl.expand(1, [0.6 * 1.4 ** k for k in range(6)]) + wl.expand(2, [0.8 * 1.5 ** k for k in range(6)])  # 64


def _free():
    return torch.cuda.mem_get_info(0)[0]


def _grid(ctx, n, seed):
    G = api.QMCGrid(ctx, grids.qmc_grid(3, n, seed))
    G.setBasisFunctions(BASIS)
    return G


@pytest.fixture()
def fresh():
    gc.collect()
    torch.zeros(1, device="cuda")
    torch.cuda.empty_cache()
    with api.Context(0) as c:
        yield c


def test_destroyed_tensor_memory_is_back_at_once(fresh):
    n1 = 300000   # an Fji of 64 functions: 300,000 x 64 x 64 doubles at least, 9.2 GiB
    G1, G2 = _grid(fresh, n1, 1), _grid(fresh, 16, 2)
    _, t = api.computeF(G1, G2, keep=True, copy=False)
    held = _free()
    t.close()
    assert _free() - held >= n1 * 64 * 64 * 8 - 4 * GIB - 64 * MIB


def test_scratch_takes_the_memory_the_pool_keeps(fresh):
    # 3.5 GiB of a destroyed tensor stay in the pool; with 1 GiB free beside it and 1.8 GiB of old scratch, the next call's 3.1 GiB of
    # scratch fit only if the pool gives them back
    n1, n2 = 115000, 200000
    G1, G2, G3, G4 = _grid(fresh, n1, 1), _grid(fresh, 16, 2), _grid(fresh, n2, 3), _grid(fresh, 16, 4)
    _, t = api.computeF(G1, G2, keep=True, copy=False)
    t.close()
    fresh.synchronize()
    hog = (_free() - GIB) // (2 * MIB) * (2 * MIB)
    held = torch.empty(hog, dtype=torch.uint8, device="cuda")
    try:
        F = api.computeF(G4, G3)
    finally:
        del held
        torch.cuda.empty_cache()
    assert F.shape == (16, 64, 64)


@pytest.mark.parametrize("dim2", [2, 3])
def test_kept_tensor_above_32_functions_has_no_padding(fresh, dim2):
    # 33 functions: 1,089 doubles a point for either kind of r2 grid
    n1, basis = 400000, BASIS[:16] + BASIS[16:28] + BASIS[34:39]
    assert len(basis) == 33
    G1, G2 = api.QMCGrid(fresh, grids.qmc_grid(3, n1, 1)), api.QMCGrid(fresh, grids.qmc_grid(dim2, 16, 2))
    for G in (G1, G2):
        G.setBasisFunctions(basis)
    t = [api.computeF(G1, G2, keep=True, copy=False)[1]]   # the call's scratch is there from here on
    before = _free()
    t += [api.computeF(G1, G2, keep=True, copy=False)[1] for _ in range(2)]
    assert before - _free() <= 2 * n1 * 33 * 33 * 8 + 128 * MIB
    for x in t:
        x.close()
