"""Flexible poses evaluated by a block of warps (few poses) against one warp
per pose (many), bit for bit: receptors and ligands of one round, just over
one and many, one to ten modes, poses in gentle contact and in deep clashes
(whose rounds have more pairs than a warp's buffer), and the minimizer's two
forms on the same poses."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MANY = 5000          # no GPU gives each of so many poses a block of its own


def _case(pkg, n_rec, n_lig, modes, n, shell, seed):
    import torch
    from gbattract.context import GbaContext
    wl = pkg.synth.make_pair(2, n_rec, n_lig, n, shell, n_modes=modes, seed=seed)
    ctx = GbaContext(0)
    rec, lig, par = ctx.upload_protein(wl.rec), ctx.upload_protein(wl.lig), ctx.upload_params(wl.params)
    grids = [ctx.build_grid(p, par) for p in (rec, lig)]
    for g in grids:
        ctx.grid_octets(g)
    return ctx, (rec, lig, *grids, par), torch.from_numpy(wl.dofs).cuda()


def _same(a, b):
    return np.array_equal(a.cpu().numpy(), b.cpu().numpy(), equal_nan=True)


@pytest.mark.parametrize("n_rec,n_lig,modes,n", [(64, 30, 1, 3), (65, 64, 5, 40), (130, 200, 6, 17), (513, 333, 10, 150),
                                                 (900, 65, 5, 300)])
@pytest.mark.parametrize("overlap", [0.6, 1.0])
def test_scoring(pkg, n_rec, n_lig, modes, n, overlap):
    reach = pkg.synth.receptor_radius(n_rec) + pkg.synth.ligand_radius(n_lig)
    ctx, ids, d = _case(pkg, n_rec, n_lig, modes, n, (overlap * reach, (overlap + 0.1) * reach), 800 + n)
    d[1, 0] = float("nan")
    few = ctx.energy_6d_modes(*ids, d)
    many = ctx.energy_6d_modes(*ids, d.repeat(MANY // n + 1, 1))
    for k in range(0, len(many) - n + 1, n):
        assert _same(many[k:k + n], few)
    ctx.close()


@pytest.mark.parametrize("modes", [2, 5, 8])
def test_minimizer(pkg, modes):
    n = 30
    reach = pkg.synth.receptor_radius(200) + pkg.synth.ligand_radius(130)
    ctx, ids, d = _case(pkg, 200, 130, modes, n, (0.8 * reach, 1.05 * reach), 820 + modes)
    few = ctx.minimize_6d_modes(*ids, d, max_evals=40)
    many = ctx.minimize_6d_modes(*ids, d.repeat(MANY // n + 1, 1), max_evals=40)
    for a, b in zip(few, many):
        assert _same(a, b[:n]) and _same(a, b[-n:])
    assert int(few[2].max()) > 5
    ctx.close()
