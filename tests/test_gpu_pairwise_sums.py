"""The sums of the pairwise parameter gradients: weights far below one scale
every gradient as weights around one do, and many terms of both signs add up
as their FP64 sum does."""
import math

import numpy as np
import pytest

from test_gpu_pairwise_paths import _backward, _system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("exponent", [-60, -100, -113])
def test_small_weights(pkg, exponent):
    """A power of two on the weights scales the weights, and so every term,
    exactly: 2^-113 is 1e-34, the weights stay normal numbers.  What is left
    is the order of the additions: 1e-9 of the largest entry, as between two
    launches."""
    import torch
    sysm, d, *par = _system(pkg, 131, 32)
    w = torch.linspace(0.5, 2.0, len(d), device="cuda")
    a = _backward(sysm, d, *par, w)
    s = 2.0 ** exponent
    b = _backward(sysm, d, *par, w * s)
    for k in range(2, 6):
        assert np.abs(b[k] / s - a[k]).max() <= 1e-9 * np.abs(a[k]).max()
    sysm.ctx.close()


def test_terms_of_both_signs(pkg):
    """One bead against one: every pose adds one term to each of five cells.
    The poses' derivatives are read with a weight of one, the terms are their
    FP32 products with the weights, summed exactly on the host.  A sum of two
    floats takes an addition with an error of at most 2^-47 of the sum so far
    (Knuth's two-sum is exact, the low part and the renormalised one round
    once each), so the cells are off by at most n 2^-47 of the terms' total
    magnitude; FP64's own rounding is 64 times smaller.  Plain FP32 sums would
    be off by thousands of times as much."""
    import torch
    from gbattract.autograd import PairwiseSystem, _call
    from gbattract.context import GbaContext
    rng = np.random.default_rng(17)
    m = pkg.model
    one = lambda q: m.Protein(xyz=np.zeros((3, 1), np.float32), type=np.ones(1, np.uint32),
                              mapped=np.ones(1, np.uint32), charge=np.full(1, q, np.float32))
    table = m.ParamTable(table=m.attract_params(np.ones((1, 1)), np.ones((1, 1))))
    n, kinds = 1 << 16, 64
    r = rng.uniform(2.5, 9.5, kinds)
    u = rng.normal(size=(kinds, 3))
    u /= np.linalg.norm(u, axis=1, keepdims=True)
    poses = np.zeros((kinds, 6), np.float32)
    poses[:, :3] = u * r[:, None]
    with GbaContext(0) as ctx:
        rec, lig, par = ctx.upload_protein(one(1.0)), ctx.upload_protein(one(-1.0)), ctx.upload_params(table)
        grid = ctx.build_grid(rec, par, m.GridOptions(alphabet=[1]))
        t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
        sysm = PairwiseSystem(ctx=ctx, rec=rec, lig=lig, grid=grid, ipon=t(np.ones((1, 1), np.int32)),
                              ffelec=table.ffelec)
        # r0 = eps = 1: d/deps is drc + dac, d/dr0 is 8 drc + 6 dac
        ql, qr, r0, eps = t(np.full(1, -1.0, np.float32)), t(np.ones(1, np.float32)), *(t(np.ones((1, 1), np.float32)),) * 2

        def sums(d, w):
            g = [torch.zeros(1, dtype=torch.float64, device="cuda") for _ in range(4)]
            _call(sysm, d, ql, qr, r0, eps, gE=w, gd=torch.empty_like(d), gql=g[0], gqr=g[1], gr0=g[2], geps=g[3])
            q, p, a, b = (float(x[0]) for x in g)
            return q, p, (a - 6 * b) / 2, (8 * b - a) / 2

        unit = torch.ones(1, device="cuda")
        terms = np.float32([sums(t(p[None]), unit) for p in poses])      # FP32 values, exactly
        assert np.all(terms != 0)
        which = rng.integers(0, kinds, n)
        w = (rng.choice([-1.0, 1.0], n) * rng.lognormal(0, 3, n)).astype(np.float32)
        got = sums(t(poses[which]), t(w))
        for k in range(4):
            v = (w * terms[which, k]).astype(np.float64)
            bound = n * 2.0 ** -47 * np.abs(v).sum()
            # drc and dac come back from d/dr0 and d/deps: a few roundings of 8 drc + 6 dac
            bound += 2.0 ** -46 * np.abs(w.astype(np.float64)[:, None] * terms[which, 2:]).sum()
            assert abs(got[k] - math.fsum(v)) <= bound
