"""Grids with a plateau so small that 1/d^6 overflows within it, bit for bit
against the CPU oracle's builder: dummy beads (and the ones that fill a chunk
up) on a voxel's centre add nothing, and a channel of ligand type 0 is zero,
however near a bead is."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("plateau", [1e-7, 1e-20])
@pytest.mark.parametrize("shape", [0, 1])
def test_dummies_on_a_voxel(pkg, oracle, plateau, shape):
    m = pkg.model
    rng = np.random.default_rng(3)
    # voxels at whole coordinates, the origin among them; beads between voxels
    # but for two dummies and, at the end, one real bead on a voxel
    xyz = (np.rint(rng.uniform(-4, 4, (3, 21))) + 0.37).astype(np.float32)
    xyz[:, 0] = 5.0
    xyz[:, 1] = -5.0
    typ = rng.integers(1, 4, 21).astype(np.uint32)
    typ[:2] = 0
    typ[5] = 0
    xyz[:, 5] = (1.0, 2.0, -3.0)
    xyz[:, 20] = (2.0, -1.0, 0.0)
    rec = m.Protein(xyz=xyz, type=typ, mapped=typ.copy(), charge=rng.choice([0.0, 1.0, -1.0], 21).astype(np.float32))
    params = m.ParamTable(table=m.attract_params(rng.uniform(3, 5, (3, 3)), rng.uniform(0.1, 10, (3, 3)), potshape=shape),
                          potshape=shape)
    opts = m.GridOptions(spacing=1.0, plateau=plateau, margin=3.0, outer_ext=4, alphabet=[1, 0, 3])
    from gbattract.context import GbaContext
    with GbaContext(0) as ctx:
        got = ctx.download_grid(ctx.build_grid(ctx.upload_protein(rec), ctx.upload_params(params), opts))
    want = oracle.build_grid(rec, params, opts)
    assert not np.isfinite(want.inner_data[[1, 3]]).all() and np.isfinite(want.inner_data[1]).mean() > 0.99
    assert not want.inner_data[2].any() and not want.outer_data[2].any()
    for a, b in ((got.inner_data, want.inner_data), (got.outer_data, want.outer_data)):
        assert np.array_equal(a, b, equal_nan=True)
