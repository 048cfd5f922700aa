"""The work that users of this library have it do, as cases to be measured.

Every case goes through the Python face of the C ABI (GbaContext) or the
autograd functions, on seeded synthetic complexes of the benchmark's
distributions (synth.make_pair): globules with 32 bead types, poses whose
ligand centre lies on a shell around contact, a 32 x 32 8-6 table.  Sizes are
those of the benchmark's workloads, of the reference server's work items (100
poses) and of uneven pairs between 300 and 3,000 receptor and 100 and 1,500
ligand beads.

  listed()              the cases
  draw(rng)             one more of the same ranges
  prepare(case, seed)   context, uploaded pair, grids, poses
  run(state)            one pass
  work(case)            bytes and floating-point operations of a pass
  exact(case, seed)     the pass's outputs in 64-bit torch, without this library
"""
import functools
import math

import numpy as np
import torch

import __graft_entry__

pkg = __graft_entry__.load_package()

from gbattract import synth                                      # noqa: E402
from gbattract.autograd import PairwiseEnergy, PairwiseSystem    # noqa: E402
from gbattract.context import GbaContext                         # noqa: E402

# Translation shells in units of the sum of the two globules' radii: from
# overlapping to just touching, as the scoring workloads have it (40-55 A for
# radii of 31.7 and 22.8 A), and from touching to a small gap for flexible
# docking, which refines poses that a rigid search has brought into contact
# (a deep clash takes the mode entries, fourth powers of a force, beyond FP32).
SHELL = (0.75, 1.0)
SHELL_MODES = (1.0, 1.12)
CUTOFF = 10.0            # pairwise cutoff of a refit, A
N_TYPES = 32


# ---- the cases ---------------------------------------------------------------

def listed():
    return [
        # one work item of the reference's server (100 poses), on the largest
        # benchmark pair: what a caller waits for who scores few poses at a time
        dict(name="score-item", kind="score", rec=2000, lig=700, poses=100, octets=True, host=False),
        # a systematic search: the benchmark's headline workload
        dict(name="score-search", kind="score", rec=2000, lig=700, poses=100_000, octets=True, host=False),
        # odd sizes on the grids as they are built, without the octet copy
        # that takes eight times their memory
        dict(name="score-lean", kind="score", rec=1237, lig=411, poses=9_999, octets=False, host=False),
        # a small pair scored from and to host arrays, as the server's item
        # processor does
        dict(name="score-host", kind="score", rec=500, lig=200, poses=1_000, octets=True, host=True),
        # flexible docking: scoring with five modes per protein, the
        # benchmark's pair
        dict(name="modes-search", kind="modes", rec=1500, lig=600, poses=20_000, modes=5, octets=True),
        # a work item of flexible poses with more modes than five
        dict(name="modes-item", kind="modes", rec=777, lig=333, poses=100, modes=7, octets=True),
        # one step of a scoring-function refit: energies and every gradient
        dict(name="refit-step", kind="refit", rec=2000, lig=700, poses=10_000, dielec="variable"),
        # the same on a small mini-batch of a small pair, constant dielectric
        dict(name="refit-small", kind="refit", rec=500, lig=200, poses=500, dielec="constant"),
        # a small job of rigid minimizations (the benchmark's smallest workload)
        dict(name="minimize-job", kind="minimize", rec=500, lig=200, poses=1_000, evals=100, pairs=1),
        # many pairs of uneven sizes minimized in one call
        dict(name="minimize-pairs", kind="minimize", rec=1500, lig=600, poses=12_000, evals=40, pairs=4),
        # flexible minimization of a docking run's best poses
        dict(name="minimize-modes", kind="minimize-modes", rec=700, lig=300, poses=500, evals=50, modes=5),
        # a new receptor: its grids built on the device, then poses scored
        dict(name="new-receptor", kind="receptor", rec=1500, lig=500, poses=2_000, octets=True),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["score", "score", "modes", "refit", "minimize", "receptor"])
    rec, lig = _log_int(rng, 300, 2500), _log_int(rng, 100, 1000)
    if kind == "score":
        poses = _log_int(rng, 50, min(100_000, 60_000_000 // lig))
        octets, host = rng.random() < 0.6, rng.random() < 0.25
        if not octets:
            poses = min(poses, max(50, 25_000_000 // lig))
        return dict(kind=kind, rec=rec, lig=lig, poses=poses, octets=octets, host=host)
    if kind == "modes":
        rec, lig = _log_int(rng, 300, 1500), _log_int(rng, 100, 700)
        modes = rng.randint(1, 10)
        poses = _log_int(rng, 50, max(51, 25_000_000 // ((rec + lig) * (1 if modes <= 5 else 3))))
        return dict(kind=kind, rec=rec, lig=lig, poses=min(poses, 20_000), modes=modes, octets=True)
    if kind == "refit":
        rec, lig = _log_int(rng, 300, 2000), _log_int(rng, 100, 700)
        return dict(kind=kind, rec=rec, lig=lig, poses=_log_int(rng, 200, 10_000),
                    dielec=rng.choice(["variable", "constant"]))
    if kind == "minimize":
        pairs = rng.choice([1, 1, 3])
        rec, lig = _log_int(rng, 300, 1500), _log_int(rng, 100, 600)
        poses = _log_int(rng, 200, 6_000)
        return dict(kind=kind, rec=rec, lig=lig, poses=poses, evals=rng.randint(20, 60), pairs=pairs)
    return dict(kind=kind, rec=_log_int(rng, 300, 1500), lig=lig, poses=_log_int(rng, 100, 5_000),
                octets=rng.random() < 0.7)


# ---- inputs --------------------------------------------------------------------

def _shell(case):
    lo, hi = SHELL_MODES if "modes" in case else SHELL
    reach = synth.receptor_radius(case["rec"]) + synth.ligand_radius(case["lig"])
    return lo * reach, hi * reach


def _pair(case, seed):
    return synth.make_pair(0, case["rec"], case["lig"], case["poses"], _shell(case),
                           n_modes=case.get("modes", 0), seed=seed)


def _pairs(case, seed):
    """The uneven pairs of a batch: the case's sizes, then smaller ones, the
    poses shared out in uneven parts."""
    k = case["pairs"]
    share = [1.0 + 0.5 * i for i in range(k)]
    out = []
    for i in range(k):
        c = dict(case, rec=max(300, int(case["rec"] / (1 + 0.45 * i))), lig=max(100, int(case["lig"] / (1 + 0.6 * i))),
                 poses=max(1, int(case["poses"] * share[i] / sum(share))))
        out.append(_pair(c, seed + 1009 * i))
    return out


def _refit_params(case, seed):
    """Per-bead charges and type-pair (r0, eps) as a refit moves them."""
    rng = np.random.default_rng(seed + 77)
    wl = _pair(case, seed)
    r0 = rng.uniform(3.0, 5.0, (N_TYPES, N_TYPES)).astype(np.float32)
    eps = rng.uniform(0.1, 10.0, (N_TYPES, N_TYPES)).astype(np.float32)
    q_lig = (wl.lig.charge + rng.normal(0, 0.1, wl.lig.n)).astype(np.float32)
    q_rec = (wl.rec.charge + rng.normal(0, 0.1, wl.rec.n)).astype(np.float32)
    weight = rng.uniform(0.1, 1.0, case["poses"]).astype(np.float32)
    return wl, r0, eps, q_lig, q_rec, weight


def _cuda(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _upload(ctx, wl, octets, lig_grid=False):
    rec, lig, par = ctx.upload_protein(wl.rec), ctx.upload_protein(wl.lig), ctx.upload_params(wl.params)
    grids = [ctx.build_grid(rec, par)] + ([ctx.build_grid(lig, par)] if lig_grid else [])
    if octets:
        for g in grids:
            ctx.grid_octets(g)
    return (rec, lig, *grids, par)


def prepare(case, seed):
    ctx = GbaContext(torch.cuda.current_device())
    s = dict(kind=case["kind"], ctx=ctx)
    kind = case["kind"]
    if kind == "score":
        wl = _pair(case, seed)
        s["ids"] = _upload(ctx, wl, case["octets"])
        s["host"] = case["host"]
        s["dofs"] = wl.dofs if case["host"] else _cuda(wl.dofs)
    elif kind == "modes":
        wl = _pair(case, seed)
        s["ids"] = _upload(ctx, wl, case["octets"], lig_grid=True)
        s["dofs"] = _cuda(wl.dofs)
    elif kind == "refit":
        wl, r0, eps, ql, qr, w = _refit_params(case, seed)
        rec, lig, grid, _ = _upload(ctx, wl, False)
        s["system"] = PairwiseSystem(ctx=ctx, rec=rec, lig=lig, grid=grid,
                                     ipon=torch.ones((N_TYPES, N_TYPES), dtype=torch.int32, device="cuda"),
                                     dielec=0 if case["dielec"] == "constant" else 1,
                                     ffelec=wl.params.ffelec, cutoff=CUTOFF)
        s["leaves"] = [_cuda(a).requires_grad_(True) for a in (wl.dofs, ql, qr, r0, eps)]
        s["weight"] = _cuda(w)
    elif kind == "minimize":
        s["evals"] = case["evals"]
        wls = _pairs(case, seed)
        s["pairs"] = [(*_upload(ctx, wl, True), _cuda(wl.dofs)) for wl in wls]
    elif kind == "minimize-modes":
        wl = _pair(case, seed)
        s["evals"] = case["evals"]
        s["ids"] = _upload(ctx, wl, True, lig_grid=True)
        s["dofs"] = _cuda(wl.dofs)
    else:
        wl = _pair(case, seed)
        s["ids"] = (ctx.upload_protein(wl.rec), ctx.upload_protein(wl.lig), ctx.upload_params(wl.params))
        s["octets"] = case["octets"]
        s["dofs"] = _cuda(wl.dofs)
    return s


def run(s):
    ctx, kind = s["ctx"], s["kind"]
    stream = torch.cuda.current_stream().cuda_stream
    if kind == "score":
        return ctx.energy_6d(*s["ids"], s["dofs"], stream=stream)
    if kind == "modes":
        return ctx.energy_6d_modes(*s["ids"], s["dofs"], stream=stream)
    if kind == "refit":
        E = PairwiseEnergy.apply(*s["leaves"], s["system"])
        return [E.detach(), *torch.autograd.grad(E, s["leaves"], s["weight"])]
    if kind == "minimize":
        if len(s["pairs"]) == 1:
            return list(ctx.minimize_6d(*s["pairs"][0], max_evals=s["evals"], stream=stream))
        return [list(r) for r in ctx.batch_minimize_6d(s["pairs"], max_evals=s["evals"], stream=stream)]
    if kind == "minimize-modes":
        return list(ctx.minimize_6d_modes(*s["ids"], s["dofs"], max_evals=s["evals"], stream=stream))
    rec, lig, par = s["ids"]
    grid = ctx.build_grid(rec, par)
    if s["octets"]:
        ctx.grid_octets(grid)
    out = ctx.energy_6d(rec, lig, grid, par, s["dofs"], stream=stream)
    ctx.release(grid)
    return out


# ---- what a pass cannot do without ------------------------------------------------

@functools.lru_cache(maxsize=None)
def _pairs_per_pose(rec, lig, modes):
    """Bead pairs within 10 A of a pose, averaged over 16 seeded poses."""
    case = dict(rec=rec, lig=lig, poses=16)
    if modes:
        case["modes"] = modes
    wl = _pair(case, 1)
    R = torch.from_numpy(wl.rec.xyz.T.copy()).double()
    X = torch.from_numpy(wl.lig.xyz.T.copy()).double()
    rot, _ = _rotation(torch.from_numpy(wl.dofs[:, 3:6].copy()).double())
    n = 0
    for k in range(16):
        p = X @ rot[k].T + torch.from_numpy(wl.dofs[k, :3].copy()).double()
        n += int((torch.cdist(p, R) <= 10.0).sum())
    return n / 16


def _voxels(beads, radius):
    inner = (math.ceil(2 * (radius + 10.8) / 0.9) + 1) ** 3
    outer = (math.ceil((2 * (radius + 10.8) + 57.6) / 1.8) + 1) ** 3
    return inner + outer


def work(case):
    rec, lig, n = case["rec"], case["lig"], case["poses"]
    kind, M = case["kind"], case.get("modes", 0)
    vox = _voxels(rec, synth.receptor_radius(rec))
    grid_bytes = 16 * (N_TYPES + 1) * vox
    if kind == "minimize" and case["pairs"] > 1:
        shares = [1.0 + 0.5 * i for i in range(case["pairs"])]
        parts = [work(dict(case, pairs=1, rec=max(300, int(rec / (1 + 0.45 * i))), lig=max(100, int(lig / (1 + 0.6 * i))),
                           poses=int(n * f / sum(shares)))) for i, f in enumerate(shares)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    pairs = _pairs_per_pose(rec, lig, M)
    # 1.2 lookups per bead (a fifth carry a charge), 8 corners of 4 floats
    lookups = 1.2 * lig + (1.2 * rec if M else 0)
    per_pose = lookups * 80 + pairs * (45 + 24 * M) + (lig + (rec if M else 0)) * (40 + 12 * M)
    touched = min(grid_bytes, n * lookups * 128)
    if kind in ("score", "modes"):
        io = (104 + 108) if M else 52
        return dict(bytes=n * io + touched + 20 * (rec + lig), flops=n * per_pose)
    if kind == "refit":
        return dict(bytes=n * (24 + 4 + 4 + 4 + 24) + 4 * n * min(pairs, 64) + 40 * (rec + lig) + 24 * N_TYPES ** 2,
                    flops=n * (pairs * 130 + lig * 60))
    if kind in ("minimize", "minimize-modes"):
        # about half of the evaluation budget is used; a VA13 step is ~ 3 dof^2
        dof = 6 + 2 * M
        ev = 0.5 * case["evals"] * n
        return dict(bytes=n * (104 + 104 + 108 if M else 80) + min(grid_bytes, ev * lookups * 128),
                    flops=ev * (per_pose + 6 * dof * dof))
    build = vox * rec * ((N_TYPES + 1) * 13 + 20)
    return dict(bytes=grid_bytes * (10 if case["octets"] else 1) + n * 52, flops=build + n * per_pose)


# ---- 64-bit restatement ------------------------------------------------------------

def _rotation(ang):
    """(n, 3) Euler angles phi, ssi, rot -> R (n, 3, 3) and dR (n, angle, 3, 3)."""
    c, s = torch.cos(ang), torch.sin(ang)
    cp, cs, cr = c.unbind(1)
    sp, ss, sr = s.unbind(1)
    z = torch.zeros_like(cp)
    R = [cr * cs * cp + sr * sp, sr * cs * cp - cr * sp, ss * cp,
         cr * cs * sp - sr * cp, sr * cs * sp + cr * cp, ss * sp,
         -cr * ss, -sr * ss, cs]
    dphi = [-cr * cs * sp + sr * cp, -sr * cs * sp - cr * cp, -ss * sp,
            cr * cs * cp + sr * sp, sr * cs * cp - cr * sp, ss * cp, z, z, z]
    dssi = [-cr * ss * cp, -sr * ss * cp, cs * cp, -cr * ss * sp, -sr * ss * sp, cs * sp, -cr * cs, -sr * cs, -ss]
    drot = [-sr * cs * cp + cr * sp, cr * cs * cp + sr * sp, z, -sr * cs * sp - cr * cp, cr * cs * sp - sr * cp, z,
            sr * ss, -cr * ss, z]
    to = lambda m: torch.stack(m, 1).reshape(-1, 3, 3)      # noqa: E731
    return to(R), torch.stack([to(dphi), to(dssi), to(drot)], 1)


def _d(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda().double()


class _Protein64:
    def __init__(self, p):
        self.x = _d(p.xyz.T)
        self.type = torch.from_numpy(p.type.astype(np.int64)).cuda()
        self.q = _d(p.charge)
        self.modes = None if p.modes is None else _d(p.modes.transpose(1, 2, 0))     # (n, M, 3)
        self.force = None if p.modes is None else _d(p.mode_force)


class _Grid64:
    """Both potential grids of a protein on the builder's layout, in 64 bits:
    per voxel and channel the pair force and energy of every bead at
    max(r, 10 A)."""

    def __init__(self, p, params):
        self.params = params
        self.table = {k: _d(params.table[k].astype(np.float64)).reshape(N_TYPES, N_TYPES) for k in ("rc", "ac")}
        # every type pair is attractive (ipon 1) with its minimum inside the
        # plateau: 8-6 energy rc r^-8 - ac r^-6 at every grid distance
        assert (params.table["ipon"] == 1).all() and float(params.table["rmin2"].max()) < 100.0
        sp = float(np.float32(0.9))
        lo = p.xyz.astype(np.float64).min(1) - float(np.float32(10.8))
        hi = p.xyz.astype(np.float64).max(1) + float(np.float32(10.8))
        n = np.ceil((hi - lo) / sp).astype(int) + 1
        pos = lo.astype(np.float32).astype(np.float64)
        opos = (pos - 32 * sp).astype(np.float32).astype(np.float64)
        on = np.ceil(((n - 1) * sp + 64 * sp) / (2 * sp)).astype(int) + 1
        b = _Protein64(p)
        self.boxes = [(_d(pos), sp, [int(v) for v in n]), (_d(opos), 2 * sp, [int(v) for v in on])]
        self.data = [self._fill(b, *box) for box in self.boxes]

    def _fill(self, b, pos, sp, n):
        C, N = N_TYPES + 1, n[0] * n[1] * n[2]
        out = torch.empty(C, N, 4, dtype=torch.float64, device="cuda")
        hot = torch.nn.functional.one_hot(b.type - 1, N_TYPES).double()
        q = b.q * self.params.ffelec
        q = torch.where(q.abs() > 0.001, q, torch.zeros_like(q))
        step = max(1, 8_000_000 // len(b.q))
        for v0 in range(0, N, step):
            v = torch.arange(v0, min(N, v0 + step), device="cuda")
            at = torch.stack([v % n[0], (v // n[0]) % n[1], v // (n[0] * n[1])], 1).double() * sp + pos
            e = at[:, None, :] - b.x[None]
            r2 = (e * e).sum(-1)
            near = (r2 < 100.0) & (r2 > 0)
            e = e * torch.where(near, 10.0 / r2.sqrt(), torch.ones_like(r2))[..., None]
            ir2 = 1.0 / r2.clamp(min=100.0)
            u = e * ir2[..., None]
            u[r2 == 0] = 0
            ir6 = ir2 ** 3
            ir8 = ir6 * ir2
            s8, s6 = ir8 @ hot, ir6 @ hot
            rc, ac = self.table["rc"], self.table["ac"]
            out[1:, v, 3] = (s8 @ rc - s6 @ ac).T
            # distance-dependent dielectric, zero beyond 50 A
            dd = (ir2 - 4.0e-4).clamp(min=0.0)
            on = (dd > 0).double()
            out[0, v, 3] = dd @ q
            for a in range(3):
                out[1:, v, a] = (((ir8 * u[..., a]) @ hot) @ (8 * rc) - ((ir6 * u[..., a]) @ hot) @ (6 * ac)).T
                out[0, v, a] = (on * 2 * ir2 * u[..., a]) @ q
        return out

    def at(self, x, typ, q):
        """Force (n, 3) and energy (n,) of beads at x (n, 3): the inner grid's
        trilinear value, else the outer's, else zero."""
        f = torch.zeros(len(x), 4, dtype=torch.float64, device="cuda")
        left = torch.ones(len(x), dtype=torch.bool, device="cuda")
        for (pos, sp, n), data in zip(self.boxes, self.data):
            nn = torch.tensor(n, device="cuda")
            inside = left & ((x >= pos) & (x <= pos + (nn - 1) * sp)).all(1)
            left &= ~inside
            k = inside.nonzero()[:, 0]
            g = (x[k] - pos) / sp
            i = torch.minimum(g.floor().long(), nn - 2)
            w = g - i
            for c in range(8):
                bit = [(c >> a) & 1 for a in range(3)]
                wc = math.prod((w[:, a] if bit[a] else 1 - w[:, a]) for a in range(3))
                v = (i[:, 0] + bit[0]) + n[0] * ((i[:, 1] + bit[1]) + n[1] * (i[:, 2] + bit[2]))
                d = data[typ[k], v]
                charged = (q[k].abs() > 0.001).double() * q[k]
                f[k] += wc[:, None] * (d + charged[:, None] * data[0, v])
        return f[:, :3], f[:, 3]

    def near(self, x):
        pos, sp, n = self.boxes[0]
        return ((x >= pos) & (x <= pos + (torch.tensor(n, device="cuda") - 1) * sp)).all(1)


def _close(x, rx, reach):
    """(ligand index, receptor index) of the pairs within reach; x (n, 3), rx
    (m, 3) or, with a receptor of its own per pose, (poses, m, 3)."""
    if rx.dim() == 2:
        d = torch.cdist(x.float(), rx.float(), compute_mode="donot_use_mm_for_euclid_dist")
        return (d <= reach + 0.01).nonzero().unbind(1)
    P = rx.shape[0]
    d = torch.cdist(x.float().reshape(P, -1, 3), rx.float(), compute_mode="donot_use_mm_for_euclid_dist")
    p, i, j = (d <= reach + 0.01).nonzero().unbind(1)
    return p * (len(x) // P) + i, p * rx.shape[1] + j


def _nl64(grid, L, x, tl, ql, R, rx, P):
    """Neighbour-list pair terms within the 10 A plateau: per-pair indices,
    energies and forces on the ligand bead."""
    i, j = _close(x, rx, 10.0)
    keep = grid.near(x)[i]
    i, j = i[keep], j[keep]
    flat = rx.reshape(-1, 3)
    m = len(R.q)
    d = x[i] - flat[j]
    r2 = (d * d).sum(1)
    keep = r2 <= 100.0
    i, j, d, r2 = i[keep], j[keep], d[keep], r2[keep]
    tr, tt = R.type[j % m] - 1, tl[i] - 1
    rc, ac = grid.table["rc"][tr, tt], grid.table["ac"][tr, tt]
    ir2 = 1.0 / r2
    ratio = ((torch.floor(r2 * 10000.0) + 0.5) * 1e-4 / 100.0).sqrt()
    e = rc * ir2 ** 4 - ac * ir2 ** 3 - (rc * 1e-8 - ac * 1e-6)
    s = 8 * rc * ir2 ** 4 - 6 * ac * ir2 ** 3 - (8 * rc * 1e-8 - 6 * ac * 1e-6) * ratio
    qq = ql[i] * R.q[j % m] * grid.params.ffelec
    qq = torch.where(qq.abs() > 0.001, qq, torch.zeros_like(qq))
    e = e + qq * (ir2 - 0.01)
    s = s + qq * 2 * ir2 - qq * 2 * 0.01 * ratio
    return i, j, e, (s * ir2)[:, None] * d


def _limit(F):
    for _ in range(3):
        F = torch.where((F * F).sum(1, keepdim=True) > 1e18, F * 0.01, F)
    return F


def _score64(wl, grid):
    """(n, 7) energies, forces and Euler gradients of rigid poses."""
    L, R = _Protein64(wl.lig), _Protein64(wl.rec)
    m, out = len(L.q), []
    dofs = _d(wl.dofs)
    step = max(1, 60_000_000 // (m * len(R.q)))
    for p0 in range(0, len(dofs), step):
        t, ang = dofs[p0:p0 + step, :3], dofs[p0:p0 + step, 3:6]
        rot, drot = _rotation(ang)
        P = len(t)
        x = (torch.einsum("pab,ib->pia", rot, L.x) + t[:, None]).reshape(-1, 3)
        tl, ql = L.type.repeat(P), L.q.repeat(P)
        f, e = grid.at(x, tl, ql)
        i, _, pe, pf = _nl64(grid, L, x, tl, ql, R, R.x, P)
        e.index_add_(0, i, pe)
        f.index_add_(0, i, pf)
        f = f.reshape(P, m, 3)
        T = torch.einsum("pia,ib->pab", f, L.x)
        out.append(torch.cat([e.reshape(P, m).sum(1, keepdim=True), _limit(f.sum(1)),
                              torch.einsum("pkab,pab->pk", drot, T)], 1))
    return torch.cat(out)


def _modes64(wl, grid, lgrid):
    """(n, 27) results of flexible poses."""
    L, R = _Protein64(wl.lig), _Protein64(wl.rec)
    M, out = wl.rec.n_modes, []
    dofs = _d(wl.dofs)
    m = len(L.q)
    step = max(1, 40_000_000 // (m * len(R.q)))
    for p0 in range(0, len(dofs), step):
        d = dofs[p0:p0 + step]
        P = len(d)
        t, aR, aL = d[:, :3], d[:, 6:6 + M], d[:, 16:16 + M]
        rot, drot = _rotation(d[:, 3:6])
        inv, _ = _rotation(-d[:, 3:6])
        xr = R.x + torch.einsum("pm,imc->pic", aR, R.modes)
        xl = L.x + torch.einsum("pm,imc->pic", aL, L.modes)
        # receptor in the ligand frame of the inverted record: R(-ang) x + R^T (-t)
        back = torch.einsum("pab,pib->pia", inv, xr) - torch.einsum("pba,pb->pa", rot, t)[:, None]
        fr, _ = lgrid.at(back.reshape(-1, 3), R.type.repeat(P), R.q.repeat(P))
        fr = torch.einsum("pab,pib->pia", rot, fr.reshape(P, -1, 3)).reshape(-1, 3)
        x = (torch.einsum("pab,pib->pia", rot, xl) + t[:, None]).reshape(-1, 3)
        tl, ql = L.type.repeat(P), L.q.repeat(P)
        f, e = grid.at(x, tl, ql)
        i, j, pe, pf = _nl64(grid, L, x, tl, ql, R, xr, P)
        e.index_add_(0, i, pe)
        f.index_add_(0, i, pf)
        fr.index_add_(0, j, -pf)
        f, fr = f.reshape(P, m, 3), fr.reshape(P, -1, 3)
        gL = -torch.einsum("pia,pab,imb->pm", f, rot, L.modes)
        gR = -torch.einsum("pia,ima->pm", fr, R.modes)
        gL, gR = gL + 4 * L.force * gL ** 4, gR + 4 * R.force * gR ** 4
        T = torch.einsum("pia,ib->pab", f, L.x)
        r = torch.zeros(P, 27, dtype=torch.float64, device="cuda")
        r[:, 0], r[:, 1:4] = e.reshape(P, m).sum(1), _limit(f.sum(1))
        r[:, 4:7] = torch.einsum("pkab,pab->pk", drot, T)
        r[:, 7:7 + M], r[:, 17:17 + M] = gR, gL
        out.append(r)
    r = torch.cat(out)
    top = torch.finfo(torch.float32).max          # the results are FP32 records
    return torch.where(r.abs() > top, torch.sign(r) * math.inf, r)


def _refit64(case, seed):
    wl, r0, eps, ql, qr, w = _refit_params(case, seed)
    L, R = _Protein64(wl.lig), _Protein64(wl.rec)
    r0, eps, ql, qr, w, dofs = map(_d, (r0, eps, ql, qr, w, wl.dofs))
    pos = _d((wl.rec.xyz.astype(np.float64).min(1) - float(np.float32(10.8))).astype(np.float32))
    n = np.ceil((np.ptp(wl.rec.xyz.astype(np.float64), axis=1) + 2 * float(np.float32(10.8))) / float(np.float32(0.9)))
    end = pos + _d(n * float(np.float32(0.9)))
    m, kr = len(L.q), len(R.q)
    E, gd = [], []
    gql, gqr = torch.zeros_like(ql), torch.zeros_like(qr)
    g0, ge = torch.zeros_like(r0).reshape(-1), torch.zeros_like(eps).reshape(-1)
    step = max(1, 60_000_000 // (m * kr))
    for p0 in range(0, len(dofs), step):
        t, ang, wp = dofs[p0:p0 + step, :3], dofs[p0:p0 + step, 3:6], w[p0:p0 + step]
        P = len(t)
        rot, drot = _rotation(ang)
        x = (torch.einsum("pab,ib->pia", rot, L.x) + t[:, None]).reshape(-1, 3)
        i, j = _close(x, R.x, CUTOFF)
        keep = ((x >= pos) & (x <= end)).all(1)[i]
        i, j = i[keep], j[keep]
        d = x[i] - R.x[j]
        r2 = (d * d).sum(1)
        keep = r2 < CUTOFF * CUTOFF
        i, j, d, r2 = i[keep], j[keep], d[keep], r2[keep]
        b, p = i % m, i // m
        tp = (R.type[j] - 1) * N_TYPES + (L.type[b] - 1)
        a, ep = r0.reshape(-1)[tp], eps.reshape(-1)[tp]
        ir2 = 1.0 / r2
        ir6, ir8 = ir2 ** 3, ir2 ** 4
        if case["dielec"] == "constant":
            dd, fc = ir2.sqrt() - 0.02, ir2.sqrt()
        else:
            dd, fc = ir2 - 4.0e-4, 2 * ir2
        fc = torch.where(dd > 0, fc, torch.zeros_like(fc))
        dd = dd.clamp(min=0.0)
        ff, qi, qj = wl.params.ffelec, ql[b], qr[j]
        e = ep * (a ** 8 * ir8 - a ** 6 * ir6) + ff * qi * qj * dd
        f = ((ep * (8 * a ** 8 * ir8 - 6 * a ** 6 * ir6) + ff * qi * qj * fc) * ir2)[:, None] * d
        add = lambda k, v, size: torch.zeros(size, dtype=torch.float64, device="cuda").index_add_(0, k, v)  # noqa: E731
        E.append(add(p, e, P))
        T = add(p, (f[:, :, None] * L.x[b][:, None, :]).reshape(-1, 9), (P, 9)).reshape(P, 3, 3)
        gd.append(-wp[:, None] * torch.cat([add(p, f, (P, 3)), torch.einsum("pkab,pab->pk", drot, T)], 1))
        gql += add(b, wp[p] * ff * qj * dd, m)
        gqr += add(j, wp[p] * ff * qi * dd, kr)
        g0 += add(tp, wp[p] * ep * (8 * a ** 7 * ir8 - 6 * a ** 5 * ir6), N_TYPES ** 2)
        ge += add(tp, wp[p] * (a ** 8 * ir8 - a ** 6 * ir6), N_TYPES ** 2)
    return [torch.cat(E), torch.cat(gd), gql, gqr, g0.reshape(r0.shape), ge.reshape(eps.shape)]


def exact(case, seed):
    kind = case["kind"]
    if kind == "refit":
        return _refit64(case, seed)
    if kind in ("minimize", "minimize-modes"):
        return None          # hundreds of dependent evaluations: no 64-bit counterpart
    wl = _pair(case, seed)
    grid = _Grid64(wl.rec, wl.params)
    if kind == "modes":
        return _modes64(wl, grid, _Grid64(wl.lig, wl.params))
    r = _score64(wl, grid)
    return r.cpu().numpy() if case.get("host") else r
