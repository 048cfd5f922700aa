"""The sizes that gba_pairwise_6d accepts: the host's check in 64 bits over
sizes whose cell count leaves 32 of them, and the entry point refusing such a
table before it launches anything."""
import ctypes as C
import subprocess
from pathlib import Path

import numpy as np
import pytest

HERE = Path(__file__).resolve().parent
CELL_BYTES = 200 * 1024 - 8 * 2624


@pytest.fixture(scope="module")
def refuses(tmp_path_factory):
    out = tmp_path_factory.mktemp("limits") / "libpairwiselimits.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", str(HERE / "csrc" / "pairwise_limits.cpp"),
                    "-o", str(out)], check=True)
    f = C.CDLL(str(out)).pairwise_refuses
    f.argtypes = [C.c_int] + [C.c_uint32] * 3
    return lambda *a: bool(f(*a))


def test_cell_count_in_full(refuses):
    rng = np.random.default_rng(5)
    types = [0, 1, 32, 99, 100, 108, 32768, 46340, 46341, 46342, 65535, 65536, 65537, 92682, 2**31, 2**32 - 1]
    types += [int(t) for t in rng.integers(0, 2**32, 200)]
    for T in types:
        for lig, rec in ((1, 1), (700, 2000), (1, 22984), (2**31, 2**31), (2**32 - 1, 2**32 - 1)):
            assert refuses(0, T, lig, rec) == (T > 65535)
            assert refuses(1, T, lig, rec) == (T > 65535 or 8 * (2 * T * T + lig + rec) > CELL_BYTES)


@pytest.mark.parametrize("n_rec,refused", [(CELL_BYTES // 8 - 2 * 32 * 32 - 5, False), (CELL_BYTES // 8 - 2 * 32 * 32 - 4, True)])
def test_last_size_that_fits(refuses, n_rec, refused):
    assert refuses(1, 32, 5, n_rec) == refused


@pytest.mark.gpu
def test_entry_point_refuses(pkg):
    import torch
    from gbattract import _lib
    from gbattract.autograd import PairwiseParamsC, _call, PairwiseSystem
    from gbattract.context import GbaContext
    wl = pkg.synth.make_pair(3, 60, 20, 8, (15.0, 30.0), seed=4)
    with GbaContext(0) as ctx:
        rec, lig, par = ctx.upload_protein(wl.rec), ctx.upload_protein(wl.lig), ctx.upload_params(wl.params)
        ones = torch.ones((32, 32), device="cuda")
        sysm = PairwiseSystem(ctx=ctx, rec=rec, lig=lig, grid=ctx.build_grid(rec, par), ipon=ones.to(torch.int32))
        d = torch.from_numpy(wl.dofs).cuda()
        ql, qr = (torch.ones(p.n, device="cuda") for p in (wl.lig, wl.rec))
        E = torch.full((len(d),), 7.0, device="cuda")
        _call(sysm, d, ql, qr, ones, ones, E=torch.empty_like(E))      # types the entry point
        outs = [torch.zeros(x.shape, dtype=torch.float64, device="cuda") for x in (ql, qr, ones, ones)]
        gd = torch.zeros_like(d)
        pp = PairwiseParamsC(r0=ones.data_ptr(), eps=ones.data_ptr(), ipon=sysm.ipon.data_ptr(), q_lig=ql.data_ptr(),
                             q_rec=qr.data_ptr(), potshape=1, dielec=1, ffelec=1.0, cutoff=10.0)
        grads = [E.data_ptr(), gd.data_ptr()] + [o.data_ptr() for o in outs]
        # refused on the host: the table's memory is that of 32 types
        for T, out in ((65536, [E.data_ptr()] + [None] * 6), (46341, [None] + grads), (65535, [None] + grads),
                       (65536, [None] + grads), (2**32 - 1, [None] + grads)):
            pp.num_types = T
            rc = _lib.load().gba_pairwise_6d(ctx.h, rec, lig, sysm.grid, C.byref(pp), d.data_ptr(), len(d), *out, None)
            assert rc != 0
        torch.cuda.synchronize()
        assert bool((E == 7.0).all()) and not any(bool(o.any()) for o in [*outs, gd])
