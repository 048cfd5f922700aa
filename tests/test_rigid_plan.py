"""The launch shape of a rigid scoring batch: what gba_autotune or
gba_set_pair_shape chose for the pair is what is launched, in both forms --
poses split into 64-bead rounds and whole poses -- and every shape gives the
same bits."""
import ctypes as C
import subprocess
from pathlib import Path

import numpy as np
import pytest

HERE = Path(__file__).resolve().parent
SMS = 152


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    out = tmp_path_factory.mktemp("plan") / "libplan.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", str(HERE / "csrc" / "rigid_plan.cpp"), "-o", str(out)],
                   check=True)
    f = C.CDLL(str(out)).plan
    f.argtypes = [C.c_size_t] * 2 + [C.c_int] * 4 + [C.POINTER(C.c_int)]

    def run(n, beads, threads, bps, resident):
        o = (C.c_int * 3)()
        f(n, beads, SMS, threads, bps, resident, o)
        return tuple(o)
    return run


@pytest.mark.parametrize("threads,bps", [(32, 1), (64, 3), (128, 2), (128, 7), (256, 1), (256, 4)])
@pytest.mark.parametrize("n,beads,split", [(1, 1, 0), (1, 64, 0), (100, 700, 1), (19_456, 700, 1), (19_457, 700, 0),
                                           (5_000, 64, 0), (100_000, 700, 0), (1, 72, 0), (76, 73, 1), (77, 73, 0),
                                           (9_728, 200, 1), (9_729, 200, 0), (19_456, 328, 1), (19_456, 327, 0)])
def test_shape_asked_for_is_launched(plan, threads, bps, n, beads, split):
    units = n * -(-beads // 64) if split else n
    warps = threads // 32
    want = max(1, min(-(-units // warps), SMS * bps))
    assert plan(n, beads, threads, bps, 8) == (split, threads, want)
    # more blocks than are resident are not launched
    assert plan(n, beads, threads, 64, bps) == (split, threads, want)


def test_totals_stay_bounded(plan):
    """64 MiB of round totals at most: 16 floats per pose and round."""
    assert plan(1000, 64 * 1048, 256, 64, 4)[0] == 1
    assert plan(1000, 64 * 1048 + 1, 256, 64, 4)[0] == 0


@pytest.mark.gpu
@pytest.mark.parametrize("n", [7, 900])
def test_every_shape_gives_the_same_bits(pkg, n):
    import torch
    from gbattract.context import GbaContext
    wl = pkg.synth.make_pair(0, 300, 130, n, (14.0, 40.0), seed=77)
    with GbaContext(0) as ctx:
        rec, lig, par = ctx.upload_protein(wl.rec), ctx.upload_protein(wl.lig), ctx.upload_params(wl.params)
        grid = ctx.build_grid(rec, par)
        ctx.grid_octets(grid)
        ids = (rec, lig, grid, par)
        d = torch.from_numpy(wl.dofs).cuda()
        want = ctx.energy_6d(*ids, d).cpu().numpy()
        assert np.isfinite(want).all()
        for flags in (15, 11):                     # with and without the four-block instantiation
            ctx.set_kernel_options(flags)
            for threads, bps in ((32, 1), (64, 3), (128, 2), (224, 5), (256, 1), (256, 64)):
                ctx.set_pair_shape(*ids, energy_threads=threads, energy_blocks_per_sm=bps)
                assert np.array_equal(ctx.energy_6d(*ids, d).cpu().numpy(), want)
        ctx.set_kernel_options(15)
        r = ctx.autotune(*ids, wl.dofs, max_evals=2)
        assert r["energy_ms"] > 0
        assert np.array_equal(ctx.energy_6d(*ids, d).cpu().numpy(), want)
