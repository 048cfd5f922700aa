"""Flexible scoring in the reference order: the kernel for launches whose
poses are all resident and the one for more poses give the same bits, on both
grid layouts, for the five- and the ten-mode kernels."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MANY = 5_000          # more than five blocks of four warps on every SM of the largest GPU hold


@pytest.mark.parametrize("modes", [1, 5, 6, 10])
def test_few_poses_equal_many(pkg, modes):
    import torch
    from gbattract.context import GbaContext
    wl = pkg.synth.make_pair(0, 90, 70, 60, (16.0, 40.0), n_modes=modes, seed=30 + modes)
    with GbaContext(0) as ctx:
        rec, lig, par = ctx.upload_protein(wl.rec), ctx.upload_protein(wl.lig), ctx.upload_params(wl.params)
        grids = [ctx.build_grid(rec, par), ctx.build_grid(lig, par)]
        ctx.set_kernel_options(31)
        d = torch.from_numpy(wl.dofs).cuda()
        many = d.repeat(MANY // len(d) + 1, 1)[:MANY].contiguous()
        for octets in (False, True):
            for g in grids:
                ctx.grid_octets(g, octets)
            few = ctx.energy_6d_modes(rec, lig, *grids, par, d).cpu().numpy()
            assert np.isfinite(few[:, 0]).all() and len(np.unique(few[:, 0])) > 30
            got = ctx.energy_6d_modes(rec, lig, *grids, par, many).cpu().numpy()
            want = np.tile(few, (MANY // len(d) + 1, 1))[:MANY]
            assert np.array_equal(got, want, equal_nan=True)
