"""The device grid builder at the sizes where its tiling can go wrong, bit for
bit against the CPU oracle's builder: bead counts around the 256-bead tile,
dummy beads (type 0), voxel counts that leave bricks partly empty, and beads
far from the origin (where the FP32 neighbour test must leave more decisions
to FP64)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _receptor(pkg, n, offset, seed):
    rng = np.random.default_rng(seed)
    wl = pkg.synth.make_pair(0, max(n, 2), 2, 1, (10.0, 12.0), seed=seed)
    typ = wl.rec.type[:n].copy()
    typ[rng.random(n) < 0.15] = 0
    if n == 1:
        typ[:] = 3
    xyz = (wl.rec.xyz[:, :n].T + np.asarray(offset, np.float32)).T.astype(np.float32)
    return pkg.model.Protein(xyz=xyz, type=typ, mapped=typ.copy(), charge=wl.rec.charge[:n]), wl.params


@pytest.mark.parametrize("n,spacing,cutoff,offset", [
    (1, 0.9, 10.8, (0, 0, 0)),
    (31, 1.7, 6.5, (0.3, -0.2, 0.1)),
    (255, 0.9, 10.8, (700.0, -900.0, 35.0)),
    (256, 1.1, 10.8, (0, 0, 0)),
    (257, 1.3, 3.0, (-4000.0, 3.0, 2500.0)),
    (513, 2.3, 12.0, (0, 0, 0)),
])
def test_lists_at_tile_edges(pkg, oracle, n, spacing, cutoff, offset):
    rec, params = _receptor(pkg, n, offset, 40 + n)
    opts = pkg.GridOptions(spacing=spacing, nl_cutoff=cutoff, alphabet=[1, 2, 5])
    from gbattract.context import GbaContext
    with GbaContext(0) as ctx:
        got = ctx.download_grid(ctx.build_grid(ctx.upload_protein(rec), ctx.upload_params(params), opts))
    nl, ng, lst = oracle.build_grid_nl(rec, opts)
    assert tuple(got.nl.dimN) == tuple(nl.dimN) and got.nl.numEl == nl.numEl
    assert np.array_equal(got.nl_grid, ng)
    assert np.array_equal(got.nl_list, lst)


@pytest.mark.parametrize("n,n_types,shape,ipon,dielec,plateau,spacing", [
    (1, 3, 1, 1, 1, 10.0, 2.0),          # one bead: partial chunk and tile
    (16, 4, 1, 1, 0, 10.0, 1.9),         # exactly a chunk, a full channel warp, constant dielectric
    (17, 5, 1, 1, 1, 10.0, 2.1),         # one channel past a warp
    (31, 8, 1, 1, 1, 10.0, 2.0),         # a full eight-channel warp
    (48, 9, 1, 1, 0, 10.0, 2.2),         # one channel past it
    (256, 32, 1, 1, 1, 10.0, 3.1),       # exactly a tile and a block of channels
    (257, 33, 1, 1, 1, 10.0, 3.3),       # one past both
    (300, 32, 1, -1, 1, 10.0, 3.0),      # repulsive pairs: the general form
    (300, 7, 1, 1, 1, 3.0, 2.6),         # minima beyond the plateau
    (300, 9, 0, 1, 1, 10.0, 2.9),        # 12-6
    (40, 0, 1, 1, 1, 10.0, 2.0),         # the charge channel alone
])
def test_potentials_at_tile_edges(pkg, oracle, n, n_types, shape, ipon, dielec, plateau, spacing):
    rec, _ = _receptor(pkg, n, (0.0, 0.0, 0.0), 90 + n)
    rng = np.random.default_rng(7)
    T = max(n_types, 33)
    table = pkg.model.attract_params(rng.uniform(3, 5, (T, T)), rng.uniform(0.1, 10, (T, T)),
                                     ipon=np.where(rng.random((T, T)) < 0.3, ipon, 1).astype(np.int32), potshape=shape)
    params = pkg.model.ParamTable(table=table, potshape=shape, dielec=dielec)
    opts = pkg.GridOptions(spacing=spacing, plateau=plateau, outer_ext=9, alphabet=list(range(1, n_types + 1)))
    from gbattract.context import GbaContext
    with GbaContext(0) as ctx:
        got = ctx.download_grid(ctx.build_grid(ctx.upload_protein(rec), ctx.upload_params(params), opts))
    want = oracle.build_grid(rec, params, opts)
    assert np.array_equal(got.inner_data.view(np.uint32), want.inner_data.view(np.uint32))
    assert np.array_equal(got.outer_data.view(np.uint32), want.outer_data.view(np.uint32))
    assert np.array_equal(got.nl_grid, want.nl_grid) and np.array_equal(got.nl_list, want.nl_list)
