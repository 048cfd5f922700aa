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


def _one_pair(pkg, ctx):
    """One bead against one: a function of poses and weights that returns the
    sums in the five cells -- d/dq of either bead, and of the type pair
    d/drc and d/dac, which d/dr0 and d/deps hold together."""
    import torch
    from gbattract.autograd import PairwiseSystem, _call
    m = pkg.model
    one = lambda q: m.Protein(xyz=np.zeros((3, 1), np.float32), type=np.ones(1, np.uint32),
                              mapped=np.ones(1, np.uint32), charge=np.full(1, q, np.float32))
    table = m.ParamTable(table=m.attract_params(np.ones((1, 1)), np.ones((1, 1))))
    rec, lig, par = ctx.upload_protein(one(1.0)), ctx.upload_protein(one(-1.0)), ctx.upload_params(table)
    grid = ctx.build_grid(rec, par, m.GridOptions(alphabet=[1]))
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    sysm = PairwiseSystem(ctx=ctx, rec=rec, lig=lig, grid=grid, ipon=t(np.ones((1, 1), np.int32)), ffelec=table.ffelec)
    # r0 = eps = 1: d/deps is drc + dac, d/dr0 is 8 drc + 6 dac
    ql, qr, r0, eps = t(np.full(1, -1.0, np.float32)), t(np.ones(1, np.float32)), *(t(np.ones((1, 1), np.float32)),) * 2

    def sums(poses, w):
        d = t(poses)
        g = [torch.zeros(1, dtype=torch.float64, device="cuda") for _ in range(4)]
        _call(sysm, d, ql, qr, r0, eps, gE=t(w), gd=torch.empty_like(d), gql=g[0], gqr=g[1], gr0=g[2], geps=g[3])
        q, p, a, b = (float(x[0]) for x in g)
        return q, p, (a - 6 * b) / 2, (8 * b - a) / 2
    return sums


def _poses_around(rng, n):
    r = rng.uniform(2.5, 9.5, n)
    u = rng.normal(size=(n, 3))
    u /= np.linalg.norm(u, axis=1, keepdims=True)
    poses = np.zeros((n, 6), np.float32)
    poses[:, :3] = u * r[:, None]
    return poses


@pytest.mark.parametrize("exponent", [-100, -113, -126])
def test_small_weight_of_one_term(pkg, exponent):
    """One term a cell: a power of two on the weight scales it exactly, down to
    the smallest normal weight, although the derivatives are as small as 1e-8."""
    from gbattract.context import GbaContext
    with GbaContext(0) as ctx:
        sums = _one_pair(pkg, ctx)
        for p in _poses_around(np.random.default_rng(3), 32):
            a = np.array(sums(p[None], np.ones(1, np.float32)))
            b = np.array(sums(p[None], np.full(1, 2.0 ** exponent, np.float32)))
            assert np.all(a != 0) and np.array_equal(b / 2.0 ** exponent, a)


def test_terms_of_both_signs(pkg):
    """Every pose adds one term to each of the cells.  The poses' derivatives
    are read with a weight of one, the terms are their FP32 products with the
    weights, summed exactly on the host.  A sum of two floats takes an addition
    with an error of at most 2^-47 of the sum so far (Knuth's two-sum is exact,
    the low part and the renormalised one round once each), so the cells are
    off by at most n 2^-47 of the terms' total magnitude; FP64's own rounding
    is 64 times smaller.  Plain FP32 sums would be off by thousands of times as
    much."""
    from gbattract.context import GbaContext
    rng = np.random.default_rng(17)
    n, kinds = 1 << 16, 64
    poses = _poses_around(rng, kinds)
    with GbaContext(0) as ctx:
        sums = _one_pair(pkg, ctx)
        unit = np.ones(1, np.float32)
        terms = np.float32([sums(p[None], unit) for p in poses])      # FP32 values, exactly
        assert np.all(terms != 0)
        which = rng.integers(0, kinds, n)
        w = (rng.choice([-1.0, 1.0], n) * rng.lognormal(0, 3, n)).astype(np.float32)
        got = sums(poses[which], w)
        for k in range(4):
            v = (w * terms[which, k]).astype(np.float64)
            bound = n * 2.0 ** -47 * np.abs(v).sum()
            # drc and dac come back from d/dr0 and d/deps: a few roundings of 8 drc + 6 dac
            bound += 2.0 ** -46 * np.abs(w.astype(np.float64)[:, None] * terms[which, 2:]).sum()
            assert abs(got[k] - math.fsum(v)) <= bound


@pytest.mark.parametrize("n", [1, 15, 16, 17])
@pytest.mark.parametrize("T", [32, 60, 100])
def test_one_block_equals_several(pkg, n, T):
    """At most 16 poses of one round are one block (8 with 100 types, whose
    cells leave room for 256 threads), most of whose cells stay empty; four
    times the poses are several.  Each sum has some hundred terms: 2^-40 of the
    largest."""
    import torch
    sysm, d, *par = _system(pkg, 40, T)
    d = d[:n].contiguous()
    w = torch.linspace(0.5, 2.0, n, device="cuda")
    one = _backward(sysm, d, *par, w)
    four = _backward(sysm, d.repeat(4, 1), *par, w.repeat(4))
    assert np.array_equal(four[0].reshape(4, n), np.tile(one[0], (4, 1)))
    assert np.array_equal(four[1].reshape(4, n, 6), np.tile(one[1], (4, 1, 1)))
    for k in range(2, 6):
        assert np.abs(one[k]).max() > 0
        assert np.abs(four[k] / 4 - one[k]).max() <= 2.0 ** -40 * np.abs(one[k]).max()
    sysm.ctx.close()


@pytest.mark.parametrize("n_lig", [65, 200])
def test_sums_of_rounds_and_whole_poses(pkg, n_lig):
    """Forty times the poses, enough for launches of whole poses: the same
    terms, in other blocks and in another order, to 48 bits a block: 1e-9 of
    the largest."""
    import torch
    sysm, d, *par = _system(pkg, n_lig, 32)
    w = torch.linspace(0.5, 2.0, len(d), device="cuda")
    small = _backward(sysm, d, *par, w)
    big = _backward(sysm, d.repeat(40, 1), *par, w.repeat(40))
    for k in range(2, 6):
        assert np.abs(big[k] / 40 - small[k]).max() <= 1e-9 * np.abs(small[k]).max()
    sysm.ctx.close()
