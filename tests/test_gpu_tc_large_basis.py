"""Transcorrelated builds above the fused kernel's 32 functions: the per-intermediate kernels run over all points in one
pass (the launches do not grow with the points), and in chunks with the same result where the
intermediates do not fit the device's free memory.  Bars as in test_gpu_kept_tensors.py (1e-10 of the largest element
against the oracle); the chunks only regroup the sums over the points (1e-12)."""
import numpy as np
import pytest
import torch

import oracle
from tcscf_b200 import api, ffi, grids
from tcscf_b200 import basis as wl

pytestmark = pytest.mark.gpu

U = dict(a=1.0, a12=1.0, terms=[((1, 0, 0), -0.5, -0.25)])
BASIS = wl.expand(0, [0.5 * 1.7 ** k for k in range(11)]) + wl.expand(1, [0.8 * 1.8 ** k for k in range(4)]) + wl.expand(2, [1.0, 2.6])   # 33
KS = (ffi.K_TC_SCALAR_SAME, ffi.K_TC_SCALAR_OPPO, ffi.K_GRAD_U_SAME, ffi.K_GRAD_U_OPPO)
MIB = 1 << 20


class _Build:
    def __init__(self, ctx, n1, nel, dim2=3):
        self.g1, self.g2, g3 = grids.qmc_grid(3, n1, 61), grids.qmc_grid(dim2, 64, 62), grids.qmc_grid(3, 64, 63)
        self.own = [api.QMCGrid(ctx, g) for g in (self.g1, self.g2, g3)]
        for k, G in enumerate(self.own):
            G.setBasisFunctions(BASIS, storeGradients=k == 0)
        u = ffi.ochi_struct(U["a"], U["a12"], U["terms"])
        self.t = [api.computeF(self.own[0], self.own[1], k, u, keep=True, copy=False)[1] for k in KS[:2]]
        self.t += [api.computeV(self.own[0], self.own[2], k, u, keep=True, copy=False)[1] for k in KS[2:]]
        self.g3 = g3
        rng, nb = np.random.default_rng(5), len(BASIS)
        cx = lambda *s: (rng.normal(size=s) + 1j * rng.normal(size=s)) * 0.3  # noqa: E731
        self.nel, self.occ, self.D, self.h = nel, [cx(n, nb) for n in nel], cx(2, nb, nb), rng.normal(size=(nb, nb))

    def run(self):
        return api.tc_fock_build(self.own[0], *self.t, *self.nel, self.D, *self.occ, self.h)

    def close(self):
        for x in self.t + self.own:
            x.close()


def _oracle(b):
    uo, nb, g = oracle.ochi(U["a"], U["a12"], U["terms"]), len(BASIS), [b.g1, b.g2, b.g3]
    vals = [oracle.basis_values(x.points, BASIS) for x in g[1:]]
    o = [oracle.compute_F(g[0].points, g[1].points, g[1].weights, vals[0], nb, k, uo) for k in KS[:2]]
    o += [oracle.compute_V(g[0].points, g[2].points, g[2].weights, vals[1], nb, k, uo) for k in KS[2:]]
    v1, d1 = oracle.basis_values(g[0].points, BASIS, gradients=True)
    return oracle.tc_fock_build(*o, v1, d1, g[0].weights, b.D, *b.nel, *b.occ, b.h)


def _check(got, ref):
    for a, r in zip(got[:3], ref[:3]):
        assert np.abs(a - r).max() <= 1e-10 * max(1.0, np.abs(r).max())
    assert abs(got[3] - ref[3]) <= 1e-10 * max(1.0, abs(ref[3]))


def _kernels(f):
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as p:
        f()
        torch.cuda.synchronize()
    return sum(1 for e in p.events() if "kTc" in e.name)


def test_launches_do_not_grow_with_the_points(ctx):
    torch.zeros(1, device="cuda")
    counts = []
    for n1 in (64, 20000):
        b = _Build(ctx, n1, (2, 1))
        b.run()
        counts.append(_kernels(b.run))
        b.close()
    if not counts[0]:
        pytest.skip("no kernel activity records here")
    assert counts[0] == counts[1], counts


@pytest.mark.parametrize("dim2", [2, 3])
def test_chunks_under_memory_pressure(ctx, dim2):
    # 12 + 12 electrons at 2,501 points: about 220 MB of intermediates; with 80 MiB free they take several chunks, the last one short
    n1, nel = 2501, (12, 12)
    b = _Build(ctx, n1, nel, dim2)
    whole = b.run()
    b.close()
    with api.Context(0) as c2:
        b = _Build(c2, n1, nel, dim2)
        torch.cuda.empty_cache()
        hog = (torch.cuda.mem_get_info(0)[0] - 80 * MIB) // (2 * MIB) * (2 * MIB)
        held = torch.empty(hog, dtype=torch.uint8, device="cuda")
        try:
            parts = b.run()
        finally:
            del held
            torch.cuda.empty_cache()
        b.close()
    for a, w in zip(parts[:3], whole[:3]):
        assert np.abs(a - w).max() <= 1e-12 * max(1.0, np.abs(w).max())
    _check(parts, _oracle(b))


@pytest.mark.parametrize("nel", [(0, 2), (1, 0)])
def test_one_spin_empty(ctx, nel):
    b = _Build(ctx, 37, nel)
    got = b.run()
    b.close()
    _check(got, _oracle(b))
