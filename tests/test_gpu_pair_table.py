"""The pair table's one- and two-entry forms (ParamsItem::pair_table) against
the oracle: tables where every pair, some pairs or no pair reads the second
entry -- by its ipon, by a negative rc, by a zero rc with its sign bit set.
The bound is the rigid kernel's (test_gpu_rigid.py)."""
import numpy as np
import pytest

from test_gpu_rigid import RTOL, pose_errors, upload

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["plain", "mixed", "repulsive", "negative", "signed_zero"])
@pytest.mark.parametrize("shape", [0, 1])
def test_entries_against_oracle(pkg, oracle, kind, shape):
    wl = pkg.synth.make_pair(0, 150, 60, 96, (20.0, 28.0), seed=52)
    rng = np.random.default_rng(3)
    T = 32
    ipon = np.ones((T, T), np.int32)
    if kind == "mixed":
        ipon = rng.choice(np.array([1, -1, 0], np.int32), (T, T))
    elif kind == "repulsive":
        ipon[:] = -1
    table = pkg.model.attract_params(rng.uniform(3, 5, (T, T)), rng.uniform(0.1, 10, (T, T)), ipon=ipon,
                                     potshape=shape)
    if kind == "negative":
        table["rc"][::3] *= -1
    elif kind == "signed_zero":
        table["rc"][::3] = -0.0
    params = pkg.model.ParamTable(table=table, potshape=shape)
    grid = oracle.build_grid(wl.rec, params, pkg.GridOptions(alphabet=list(range(1, T + 1)), spacing=1.8, outer_ext=8))
    ref, st = oracle.energy_6d(wl.rec, wl.lig, grid, params, wl.dofs, stats=True)
    from gbattract.context import GbaContext
    with GbaContext(0) as ctx:
        ids = upload(ctx, wl.rec, wl.lig, grid, params)
        for octets in (False, True):
            ctx.grid_octets(ids[2], octets)
            got = ctx.energy_6d(*ids, wl.dofs)
            for e in pose_errors(got, ref, st):
                assert float(e.max()) <= RTOL
