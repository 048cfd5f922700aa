"""The pairwise kernels' launch forms against each other: poses split into
64-bead rounds and whole poses (bit for bit per pose), blocks of 512 and of
256 threads (a large type table), and parameter sums that leave a float's
range.  The values themselves are checked in test_gpu_adjoint.py."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _system(pkg, n_lig, T, seed=91):
    import torch
    from gbattract.autograd import PairwiseSystem
    from gbattract.context import GbaContext
    rng = np.random.default_rng(seed)
    wl = pkg.synth.make_pair(3, 220, n_lig, 700, (15.0, 30.0), seed=seed)
    r0 = np.full((T, T), 4.0, np.float32)
    eps = np.full((T, T), 1.0, np.float32)
    ipon = np.ones((T, T), np.int32)
    r0[:32, :32] = rng.uniform(3, 5, (32, 32))
    eps[:32, :32] = rng.uniform(0.1, 10, (32, 32))
    ipon[:32, :32] = rng.choice(np.array([1, 1, 1, 0, -1]), (32, 32))
    ctx = GbaContext(0)
    rec, lig, par = ctx.upload_protein(wl.rec), ctx.upload_protein(wl.lig), ctx.upload_params(wl.params)
    sysm = PairwiseSystem(ctx=ctx, rec=rec, lig=lig, grid=ctx.build_grid(rec, par),
                          ipon=torch.from_numpy(ipon).cuda(), ffelec=wl.params.ffelec)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a, np.float32)).cuda()
    ql, qr = (t(p.charge + rng.normal(0, 0.1, p.n)) for p in (wl.lig, wl.rec))
    return sysm, t(wl.dofs), ql, qr, t(r0), t(eps)


def _backward(sysm, d, ql, qr, r0, eps, w):
    """FP64 parameter gradients and the DOF gradient for upstream weights w."""
    import torch
    from gbattract.autograd import _call
    E = torch.empty(len(d), device="cuda")
    _call(sysm, d, ql, qr, r0, eps, E=E)
    gd = torch.empty_like(d)
    z = [torch.zeros(x.shape, dtype=torch.float64, device="cuda") for x in (ql, qr, r0, eps)]
    _call(sysm, d, ql, qr, r0, eps, gE=w, gd=gd, gql=z[0], gqr=z[1], gr0=z[2], geps=z[3])
    return [E.cpu().numpy(), gd.cpu().numpy()] + [x.cpu().numpy() for x in z]


@pytest.mark.parametrize("n_lig", [1, 64, 65, 200])
def test_rounds_equal_whole_poses(pkg, n_lig):
    import torch
    sysm, d, *par = _system(pkg, n_lig, 32)
    w = torch.linspace(0.5, 2.0, len(d), device="cuda")
    small = _backward(sysm, d, *par, w)
    reps = 40                     # 28,000 poses: more than four for every warp
    big = _backward(sysm, d.repeat(reps, 1), *par, w.repeat(reps))
    for k in (0, 1):
        whole = big[k].reshape(reps, *small[k].shape)
        for part in whole:
            assert np.array_equal(part, small[k])
    for k in range(2, 6):
        # the cells keep 48 bits; the sums differ in order alone
        scale = np.abs(small[k]).max()
        assert np.abs(big[k] / reps - small[k]).max() <= 1e-6 * scale
    sysm.ctx.close()


def test_large_type_table(pkg):
    """100 types leave shared memory for 256 threads only; the types of the
    beads are the first 32 of them."""
    import torch
    res = {}
    for T in (32, 100):
        sysm, d, *par = _system(pkg, 130, T)
        res[T] = _backward(sysm, d, *par, torch.ones(len(d), device="cuda"))
        sysm.ctx.close()
    assert np.array_equal(res[32][0], res[100][0]) and np.array_equal(res[32][1], res[100][1])
    for k in range(2, 6):
        a, b = res[32][k], res[100][k]
        if k >= 4:
            assert not b[32:].any() and not b[:, 32:].any()
            b = b[:32, :32]
        assert np.abs(a - b).max() <= 1e-9 * np.abs(a).max()


@pytest.mark.parametrize("T", [46, 47])
def test_copies_of_the_type_cells(pkg, T):
    """At 46 types the last blocks with two copies of the type pairs' cells, at
    47 the first with one; 32 types have two.  An odd number of charge cells
    lies between the copies.  48-bit sums that differ in order alone."""
    import torch
    res = {}
    for t in (32, T):
        sysm, d, *par = _system(pkg, 131, t)
        res[t] = _backward(sysm, d, *par, torch.linspace(0.5, 2.0, len(d), device="cuda"))
        sysm.ctx.close()
    assert np.array_equal(res[32][0], res[T][0]) and np.array_equal(res[32][1], res[T][1])
    for k in range(2, 6):
        a, b = res[32][k], res[T][k]
        if k >= 4:
            assert not b[32:].any() and not b[:, 32:].any()
            b = b[:32, :32]
        assert np.abs(a - b).max() <= 1e-9 * np.abs(a).max()


def test_sums_beyond_a_float(pkg):
    """A power of two on the weights scales every gradient exactly; the terms
    then pass 1e37 and are added up in double.  Only a sum one of whose terms
    is itself beyond FP32 is infinite."""
    import torch
    sysm, d, *par = _system(pkg, 65, 32)
    w = torch.linspace(0.5, 2.0, len(d), device="cuda")
    a = _backward(sysm, d, *par, w)
    s = 2.0 ** 118
    b = _backward(sysm, d, *par, w * s)
    top = float(np.finfo(np.float32).max)
    beyond = 0
    for k in range(2, 6):
        scale = np.abs(a[k]).max()
        fin = np.isfinite(b[k])
        assert np.all(np.abs(a[k][~fin]) * s > top)
        assert np.abs(b[k][fin] / s - a[k][fin]).max() <= 1e-9 * scale
        beyond += int((np.abs(b[k][fin]) > top).sum())
    assert beyond > 0
    sysm.ctx.close()
