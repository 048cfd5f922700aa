"""Pairwise calls of more poses than one launch takes (2^20): every pose's
result is that of a call by itself, the gradients are sums over all launches,
and the device memory that a call takes does not grow with its poses."""
import numpy as np
import pytest

from test_gpu_pairwise_paths import _system

pytestmark = pytest.mark.gpu

CHUNK = 1 << 20


def _run(sysm, d, par, w):
    import torch
    from gbattract.autograd import _call
    E, gd = torch.empty(len(d), device="cuda"), torch.empty_like(d)
    z = [torch.zeros(x.shape, dtype=torch.float64, device="cuda") for x in par]
    _call(sysm, d, *par, E=E)
    _call(sysm, d, *par, gE=w, gd=gd, gql=z[0], gqr=z[1], gr0=z[2], geps=z[3])
    torch.cuda.synchronize()
    return E, gd, z


def test_more_poses_than_a_launch(pkg):
    import torch
    sysm, d, *par = _system(pkg, 20, 32)
    reps = CHUNK // len(d) + 2
    many = d.repeat(reps, 1)[:CHUNK + 301].contiguous()
    k = len(d)
    w = torch.linspace(0.5, 2.0, k, device="cuda").repeat(reps)[:len(many)].contiguous()
    E1, gd1, _ = _run(sysm, d, par, w[:k].contiguous())
    E, gd, z = _run(sysm, many, par, w)
    assert torch.equal(E, E1.repeat(reps)[:len(many)]) and torch.equal(gd, gd1.repeat(reps, 1)[:len(many)])
    *_, a = _run(sysm, many[:CHUNK].contiguous(), par, w[:CHUNK].contiguous())
    *_, b = _run(sysm, many[CHUNK:].contiguous(), par, w[CHUNK:].contiguous())
    for x, y, v in zip(a, b, z):
        # the same FP32 terms; 48-bit sums of some thousand of them in a cell
        assert bool((x.abs() > 0).any()) and float((x + y - v).abs().max()) <= 2.0 ** -32 * float(v.abs().max())
    sysm.ctx.close()


def test_memory_does_not_grow(pkg):
    """6 M poses: records of 80 bytes for all of them would be 480 MB."""
    import torch
    sysm, d, *par = _system(pkg, 20, 32)
    n = 6_000_000
    many = d.repeat(n // len(d) + 1, 1)[:n].contiguous()
    w = torch.ones(n, device="cuda")
    E, gd = torch.empty(n, device="cuda"), torch.empty_like(many)
    z = [torch.zeros(x.shape, dtype=torch.float64, device="cuda") for x in par]
    from gbattract.autograd import _call
    _call(sysm, d, *par, E=E[:len(d)])           # what is built at first use
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    _call(sysm, many, *par, E=E)
    _call(sysm, many, *par, gE=w, gd=gd, gql=z[0], gqr=z[1], gr0=z[2], geps=z[3])
    torch.cuda.synchronize()
    assert free - torch.cuda.mem_get_info()[0] <= 256 << 20
    sysm.ctx.close()
