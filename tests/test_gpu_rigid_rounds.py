"""Scoring launches split into 64-bead rounds against launches of whole poses:
a pose's result is the same bit for bit whichever it is part of, for ligands
of one round (never split), just over one, a partly filled last round and many
rounds, on both grid layouts, with and without the visiting order."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

WHOLE = 45_000          # more than four poses for every warp of the largest GPU


@pytest.mark.parametrize("n_lig", [1, 64, 65, 129, 700])
@pytest.mark.parametrize("octets", [False, True])
def test_split_equals_whole(pkg, n_lig, octets):
    import torch
    from gbattract.context import GbaContext
    wl = pkg.synth.make_pair(0, 300, n_lig, 5000, (14.0, 40.0), seed=700 + n_lig)
    wl.dofs[7, 0] = np.nan
    wl.dofs[8, 4] = np.inf
    with GbaContext(0) as ctx:
        rec, lig, par = ctx.upload_protein(wl.rec), ctx.upload_protein(wl.lig), ctx.upload_params(wl.params)
        grid = ctx.build_grid(rec, par)
        if octets:
            ctx.grid_octets(grid)
        ids = (rec, lig, grid, par)
        d = torch.from_numpy(wl.dofs).cuda()
        many = d.repeat(WHOLE // len(d), 1)
        whole = ctx.energy_6d(*ids, many).cpu().numpy().reshape(-1, len(d), 7)
        for part in whole:
            assert np.array_equal(part, whole[0], equal_nan=True)
        for n in (1, 5, 33, 1000, 5000):          # 4,096 and more are visited in the spatial order
            got = ctx.energy_6d(*ids, d[:n].contiguous()).cpu().numpy()
            assert np.array_equal(got, whole[0][:n], equal_nan=True)


def test_concurrent_streams(pkg):
    """Calls in flight on several streams keep their own scratch."""
    import torch
    from gbattract.context import GbaContext
    wl = pkg.synth.make_pair(0, 300, 200, 600, (14.0, 40.0), seed=71)
    with GbaContext(0) as ctx:
        rec, lig, par = ctx.upload_protein(wl.rec), ctx.upload_protein(wl.lig), ctx.upload_params(wl.params)
        ids = (rec, lig, ctx.build_grid(rec, par), par)
        d = torch.from_numpy(wl.dofs).cuda()
        want = ctx.energy_6d(*ids, d)
        torch.cuda.synchronize()
        streams = [torch.cuda.Stream() for _ in range(4)]
        outs = [torch.empty_like(want) for _ in range(40)]
        for k, o in enumerate(outs):
            ctx.energy_6d(*ids, d, out=o, stream=streams[k % 4].cuda_stream)
        torch.cuda.synchronize()
        for o in outs:
            assert torch.equal(o, want)
