"""The parameter gradients that PairwiseEnergy.backward returns are tensors of
their own, on the CPU with the library call replaced: a caller may change one
in place while another is saved for a backward pass, multiply one in place by
a tensor that needs a gradient, and keep one without keeping the others."""
import ctypes as C

import numpy as np
import pytest
import torch


def _fill(ptr, value, n):
    if n:
        C.memmove(ptr, np.full(n, value, np.float64).ctypes.data, 8 * n)


@pytest.fixture
def grads(pkg, monkeypatch):
    from gbattract import autograd as ag

    def call(sysm, d, ql, qr, r0, eps, E=None, gE=None, gd=None, gql=None, gqr=None, gr0=None, geps=None):
        if gE is None:
            E.zero_()
            return
        gd.fill_(0.5)
        for k, (t, g) in enumerate(zip((ql, qr, r0, eps), (gql, gqr, gr0, geps))):
            _fill(g if isinstance(g, int) else g.data_ptr(), k + 1.0, t.numel())

    monkeypatch.setattr(ag, "_call", call)

    def run(n_lig=5, n_rec=7, T=3):
        leaves = [torch.ones(*s, requires_grad=True) for s in ((4, 6), (n_lig,), (n_rec,), (T, T), (T, T))]
        E = ag.PairwiseEnergy.apply(*leaves, None)
        return torch.autograd.grad(E, leaves, torch.ones(4))
    return run


@pytest.mark.parametrize("n_lig,n_rec", [(5, 7), (1, 1), (0, 3), (4, 8)])
def test_values_and_layout(grads, n_lig, n_rec):
    g = grads(n_lig, n_rec)
    for k, (t, shape) in enumerate(zip(g[1:], ((n_lig,), (n_rec,), (3, 3), (3, 3)))):
        assert tuple(t.shape) == shape and t.dtype is torch.float32 and t.is_contiguous()
        assert bool((t == k + 1.0).all())
    assert bool((g[0] == 0.5).all())


def test_each_has_its_own_memory(grads):
    g = grads()
    assert len({t.untyped_storage().data_ptr() for t in g}) == len(g)
    assert not any(t._is_view() for t in g)
    assert [t.untyped_storage().nbytes() for t in g] == [4 * t.numel() for t in g]


def test_one_changed_while_another_is_saved(grads):
    g = grads()
    w = torch.ones(7, requires_grad=True)
    loss = (w * g[2]).sum()                # saves g[2]
    g[1].mul_(2)
    g[3].zero_()
    loss.backward()
    assert bool((w.grad == 2.0).all())


def test_in_place_product_with_a_leaf(grads):
    g = grads()
    w = torch.full((5,), 3.0, requires_grad=True)
    g[1].mul_(w)
    g[1].sum().backward()
    assert bool((w.grad == 1.0).all())
