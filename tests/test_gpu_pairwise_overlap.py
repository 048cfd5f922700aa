"""Pairwise calls of few poses, whose launches overlap: calls in a row on one
stream, calls on several streams and calls replayed from a CUDA graph give the
results of a call by itself."""
import numpy as np
import pytest

from test_gpu_pairwise_paths import _system

pytestmark = pytest.mark.gpu


def _buffers(d, par):
    import torch
    return (torch.empty(len(d), device="cuda"), torch.empty_like(d),
            [torch.zeros(x.shape, dtype=torch.float64, device="cuda") for x in par])


def _both(sysm, d, par, w, out):
    from gbattract.autograd import _call
    E, gd, z = out
    _call(sysm, d, *par, E=E)
    _call(sysm, d, *par, gE=w, gd=gd, gql=z[0], gqr=z[1], gr0=z[2], geps=z[3])


def _same(a, b, calls=1):
    import torch
    assert torch.equal(a[0], b[0]) and torch.equal(a[1], b[1])
    for x, y in zip(a[2], b[2]):
        assert float((x / calls - y).abs().max()) <= 1e-11 * float(y.abs().max())


@pytest.mark.parametrize("n_lig,n", [(17, 40), (130, 60)])
def test_streams_and_rows(pkg, n_lig, n):
    import torch
    sysm, d, *par = _system(pkg, n_lig, 32)
    d = d[:n].contiguous()
    w = torch.linspace(0.5, 2.0, n, device="cuda")
    want = _buffers(d, par)
    _both(sysm, d, par, w, want)
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(4)]
    outs = [_buffers(d, par) for _ in range(40)]
    torch.cuda.synchronize()
    for k, o in enumerate(outs):
        with torch.cuda.stream(streams[k % 4]):
            _both(sysm, d, par, w, o)
    torch.cuda.synchronize()
    for o in outs:
        _same(o, want)
    # sums of calls in a row on one stream
    row = _buffers(d, par)
    torch.cuda.synchronize()
    for _ in range(50):
        _both(sysm, d, par, w, row)
    torch.cuda.synchronize()
    _same(row, want, calls=50)
    sysm.ctx.close()


def test_graph_replay(pkg):
    import torch
    sysm, d, *par = _system(pkg, 17, 32)
    d = d[:40].contiguous()
    w = torch.linspace(0.5, 2.0, 40, device="cuda")
    want, out = _buffers(d, par), _buffers(d, par)
    _both(sysm, d, par, w, want)              # what is built at first use, too
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        _both(sysm, d, par, w, out)
    for _ in range(20):
        g.replay()
    torch.cuda.synchronize()
    _same(out, want, calls=20)
    sysm.ctx.close()
