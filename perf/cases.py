"""What the performance of this framework is measured on: its public entry
points over the sizes and options a flow solver calls them with.

A case is a dict of plain values.  ``kind`` names the entry point:

* ``solve``     one pressure projection (``Projection.newsolv_mg_device``), the
                fields resident on the device;
* ``host``      the same through the host-array drop-in (``newsolv_mg``);
* ``batch``     many independent domains in one call (``Batch.solve_device``);
* ``predictor`` one Runge-Kutta stage of the velocity predictor
                (``mf3d_rungek_2nd_device``);
* ``restart``   a restart file image written and read back
                (``mf3d_tecbin_encode_device`` / ``mf3d_tecbin_decode_device``).

A solve starts from p = 0, so every pass does the same iterations.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from multiflow3d_b200 import abi
from multiflow3d_b200.abi import RkFields
from multiflow3d_b200.problems import PERIODIC, WALL, Problem, domain_desc, domain_problem, random_batch
from multiflow3d_b200.solver import Batch, Projection

_DP = C.POINTER(C.c_double)
_SMOOTHER = {"lexicographic": 1, "line": 2, "redblack": 3}
_SOLVE_KEYS = ("ustar", "vstar", "wstar", "u", "v", "w", "p")


# ---------------------------------------------------------------------------
# The cases.
# ---------------------------------------------------------------------------
def _solve(name, blocks, cells, levels, **kw):
    """One projection on blocks[0] x blocks[1] x blocks[2] blocks of
    cells[0] x cells[1] x cells[2] cells; ``iterations`` is what the stopping
    test gives (a count, used by ``work`` alone)."""
    c = {"kind": "solve", "px": blocks[0], "py": blocks[1], "pz": blocks[2], "nx": cells[0], "ny": cells[1],
         "nz": cells[2], "levels": levels, "smoother": "redblack", "precision": "fp64", "stretch": 0.0,
         "tol": 1e-8, "maxcy": 200, "density": False, "sip": 0, "bounds": False, "pl": 2, "pl_ex": 0,
         "spacing": 1.0 / (blocks[0] * cells[0]), "iterations": 30}
    c.update(kw)
    if name:
        c["name"] = name
    return c


def _predictor(name, scheme, blocks, cells, **kw):
    c = {"kind": "predictor", "scheme": scheme, "px": blocks[0], "py": blocks[1], "pz": blocks[2],
         "nx": cells[0], "ny": cells[1], "nz": cells[2], "spacing": 1.0 / (blocks[0] * cells[0]), "dt": 1e-3,
         "alfapr": 0.5, "forcing": True}
    c.update(kw)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest channel a user checks the solver with: one block, four
        # levels, launches and latency
        _solve("channel_64x32x32", (1, 1, 1), (64, 32, 32), 4, pl=1, spacing=1.0 / 32, iterations=15),
        # the production channel of the benchmark: eight blocks, wall-normal
        # stretching, six levels, a tight tolerance
        _solve("channel_256_blocks8", (2, 2, 2), (128, 128, 128), 6, stretch=2.0, tol=1e-10, maxcy=400, iterations=91),
        # a Fortran time loop on host arrays: ragged blocks whose edges are no
        # powers of two, a spacing that is none either, boundary values too
        _solve("host_ragged_blocks6", (3, 1, 2), (60, 44, 72), 3, kind="host", bounds=True, spacing=0.0107,
               tol=1e-6, maxcy=40, iterations=40),
        # mixed precision (FP32 V-cycle in the FP64 loop) on one large block
        _solve("mixed_512x256x256", (1, 1, 1), (512, 256, 256), 7, precision="fp32", stretch=2.0, spacing=1.0 / 256,
               maxcy=400, iterations=69),
        # many small domains of uneven sizes in one call, mixed precision
        {"name": "batch_64_uneven", "kind": "batch", "domains": 64, "low": 32, "high": 192, "sizes_seed": 2024,
         "precision": "fp32", "tol": 1e-8, "maxcy": 300, "iterations": 77},
        # the reference's default smoother (line Gauss-Seidel) on the
        # stretched channel at half resolution
        _solve("lines_128_blocks8", (2, 2, 2), (64, 64, 64), 5, smoother="line", stretch=2.0, tol=1e-8, maxcy=100,
               iterations=18),
        # two-phase flow: variable density, the time step's budget of cycles
        _solve("density_128_blocks8", (2, 2, 2), (64, 64, 64), 5, density=True, tol=1e-8, maxcy=60, iterations=60),
        # solver 1 (Stone's SIP), four sweeps per call, a bounded number of calls
        _solve("sip_64_blocks8", (2, 2, 2), (32, 32, 32), 1, sip=4, pl=1, tol=1e-8, maxcy=50, iterations=50),
        # one predictor stage, 2nd-order convection, the benchmark's channel
        _predictor("predictor_2nd_256_blocks8", 1, (2, 2, 2), (128, 128, 128)),
        # 4th-order convection on ragged blocks, a spacing that is no power of two
        _predictor("predictor_4th_ragged", 2, (2, 1, 2), (90, 117, 75), spacing=0.0113),
        # WENO convection (required with the level set), a mid-size channel
        _predictor("predictor_weno_128_blocks8", 3, (2, 2, 2), (64, 64, 64)),
        # one block's restart file (ttc 132^3) written and read back
        {"name": "restart_132", "kind": "restart", "ti": 132, "tj": 132, "tk": 132},
    ]


def draw(rng):
    def logu(lo, hi):
        return math.exp(rng.uniform(math.log(lo), math.log(hi)))

    kind = rng.choice(("solve", "solve", "solve", "host", "batch", "line", "density", "sip", "predictor", "predictor",
                       "restart"))
    blocks = rng.choice(((1, 1, 1), (2, 1, 1), (2, 2, 1), (1, 2, 2), (2, 2, 2), (3, 1, 2)))
    if kind == "restart":
        return {"kind": "restart", **{k: int(logu(12, 160)) for k in ("ti", "tj", "tk")}}
    if kind == "batch":
        return {"kind": "batch", "domains": rng.randint(3, 40), "low": 16, "high": rng.choice((48, 96, 160)),
                "sizes_seed": rng.randrange(1 << 20), "precision": rng.choice(("fp32", "fp64")), "tol": 1e-8,
                "maxcy": 60, "iterations": 25}
    if kind == "predictor":
        cells = [int(logu(17, 110)) for _ in range(3)]
        return _predictor(None, rng.choice((1, 1, 2, 3)), blocks, cells, dt=rng.choice((1e-3, 0.0137)),
                          alfapr=rng.choice((0.5, 1.0 / 3.0)), forcing=rng.random() < 0.5,
                          spacing=rng.choice((1.0 / 128, logu(0.004, 0.05))))
    if kind == "sip":
        return _solve(None, blocks, [int(logu(10, 56)) for _ in range(3)], 1, sip=rng.choice((2, 4, 10)), pl=1, tol=1e-8,
                      maxcy=rng.randint(5, 30), iterations=20)
    levels = rng.randint(2, 5)
    unit = 1 << (levels - 1)
    top = {"solve": 144, "host": 72, "line": 72, "density": 80}[kind]
    cells = [max(1, round(logu(max(12, 2 * unit), top) / unit)) * unit for _ in range(3)]
    kw = {"maxcy": rng.randint(10, 40), "iterations": 25, "tol": 10.0 ** -rng.randint(5, 9), "pl": rng.choice((1, 2)),
          "spacing": rng.choice((1.0 / 128, logu(0.004, 0.05)))}
    if kind == "solve":
        kw["precision"] = rng.choice(("fp64", "fp64", "fp32"))
        kw["stretch"] = rng.choice((0.0, 1.5, 2.0))
    elif kind == "host":
        kw.update(kind="host", bounds=True)
    elif kind == "line":
        kw["smoother"] = rng.choice(("line", "line", "lexicographic"))
        kw["stretch"] = rng.choice((0.0, 2.0))
        kw["maxcy"] = rng.randint(5, 15)
    else:
        kw["density"] = True
    return _solve(None, blocks, cells, levels, **kw)


# ---------------------------------------------------------------------------
# Inputs: one global field cut into blocks.
# ---------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _wrap(a, pr):
    """Ghost layers made periodic along the periodic axes (in place)."""
    pl = pr.pl
    for ax, bc in ((2, pr.bc[0]), (1, pr.bc[2]), (0, pr.bc[4])):
        if bc == PERIODIC:
            n = a.shape[ax] - 2 * pl
            idx = pl + torch.remainder(torch.arange(a.shape[ax], device=a.device) - pl, n)
            a = a.index_select(ax, idx)
    return a


def _walls(vel, pr, mirror):
    """Wall values of the three global components: the normal velocity is 0
    on a wall; with ``mirror`` its deeper ghosts too, and the tangential
    ghosts are minus the cells inside, as boundu/v/w leave them."""
    pl = pr.pl
    for ax, bc, comp in ((2, pr.bc[0], 0), (1, pr.bc[2], 1), (0, pr.bc[4], 2)):
        if bc == PERIODIC:
            continue
        for c, a in enumerate(vel):
            n = a.shape[ax] - 2 * pl
            v = a.movedim(ax, 0)
            if c == comp:
                if mirror:
                    v[:pl] = 0.0
                    v[pl + n - 1:] = 0.0
                else:
                    v[pl - 1] = 0.0
                    v[pl + n - 1] = 0.0
            elif mirror:
                v[:pl] = -v[pl:2 * pl].flip(0)
                v[pl + n:] = -v[n:pl + n].flip(0)
    return vel


def _velocity(pr, seed, mirror=False):
    """Uniform [-1, 1] noise plus four smooth modes of amplitude 0.1, mean
    removed, ghosts periodic where the box is."""
    g, rng, pl = _gen(seed), np.random.default_rng(seed), pr.pl
    shp = (pr.NZ + 2 * pl, pr.NY + 2 * pl, pr.NX + 2 * pl)
    out = []
    for _ in range(3):
        a = torch.rand(shp, generator=g, device="cuda", dtype=torch.float64).mul_(2.0).sub_(1.0)
        for _m in range(4):
            k, ph = rng.integers(1, 4, size=3), rng.uniform(0, 2 * np.pi, size=3)
            w = [torch.sin(2 * np.pi * int(k[q]) * (torch.arange(s, device="cuda", dtype=torch.float64) - pl + 0.5)
                           / (s - 2 * pl) + ph[q]) for q, s in enumerate(shp)]
            a.addcmul_(w[0][:, None, None] * w[1][None, :, None], w[2][None, None, :], value=0.1)
        a -= a[pl:-pl, pl:-pl, pl:-pl].mean()
        out.append(_wrap(a, pr))
    out = _walls(out, pr, mirror)
    return [_wrap(a, pr) for a in out] if mirror else out


class _Store:
    """One array of a field over all blocks; block b is a view of it."""

    def __init__(self, shapes):
        self.at, n = [], 0
        for s in shapes:
            self.at.append((n, s))
            n += -(-int(np.prod(s)) // 32) * 32  # every block 256-byte aligned
        self.flat = torch.zeros(n, dtype=torch.float64, device="cuda")

    def block(self, b):
        o, s = self.at[b]
        return self.flat[o:o + int(np.prod(s))].view(s)


def _cut(pr, glob):
    """A global field's blocks, ghost layers included, in one store."""
    st = _Store([pr.ttc] * pr.nblocks)
    for b in range(pr.nblocks):
        bx, by, bz = pr.block_pos(b)
        z, y, x = bz * pr.nz, by * pr.ny, bx * pr.nx
        st.block(b).copy_(glob[z:z + pr.ttc[0], y:y + pr.ttc[1], x:x + pr.ttc[2]])
    return st


def _problem(case):
    pl, h = case.get("pl", 2), case["spacing"]
    if case["kind"] == "predictor":
        pl = {1: 2, 2: 3, 3: 4}[case["scheme"]]
    return Problem(case["px"], case["py"], case["pz"], case["nx"], case["ny"], case["nz"], dx=h, dy=h, dz=h, pl=pl,
                   ngrid=case.get("levels", 1), stretch_y=case.get("stretch", 0.0))


def _density(pr, seed):
    """Cell densities uniform in [0.5, 2], every block seeing its neighbours'."""
    pl = pr.pl
    shp = (pr.NZ + 2 * pl, pr.NY + 2 * pl, pr.NX + 2 * pl)
    return _wrap(torch.rand(shp, generator=_gen(seed + 77), device="cuda", dtype=torch.float64).mul_(1.5).add_(0.5), pr)


def _params(pr, case):
    prec = abi.MF3D_PREC_FP32 if case["precision"] == "fp32" else abi.MF3D_PREC_FP64
    return pr.params(mg_itrsch=_SMOOTHER[case["smoother"]], irestr=2, iproln=1, maxcy=case["maxcy"], eps=case["tol"],
                     eps_relative=1, precision=prec, pl_ex=case["pl_ex"], lsm=int(case["density"]),
                     bounds=int(case["bounds"]), solver=1 if case["sip"] else 0, nswp=case["sip"])


# ---------------------------------------------------------------------------
# prepare / run
# ---------------------------------------------------------------------------
def _batch_problems(case):
    lib = abi.load()
    return [domain_problem(nx, ny, nz, bc, lib.mf3d_max_levels(nx, ny, nz))
            for nx, ny, nz, bc in random_batch(case["domains"], case["sizes_seed"], lo=case["low"], hi=case["high"])]


def prepare(case, seed):
    lib = abi.load()
    kind = case["kind"]
    if kind == "restart":
        n = (case["tk"], case["tj"], case["ti"])
        fields = torch.randn((16, *n), generator=_gen(seed), dtype=torch.float64, device="cuda")
        xyz = [(torch.arange(m, dtype=torch.float64, device="cuda") - 2) / 256.0 for m in reversed(n)]
        size = int(lib.mf3d_tecbin_size(*reversed(n)))
        info = abi.TecbinInfo(toti=n[2], totj=n[1], totk=n[0], pl=2, inind=0, jnind=-1, knind=0,
                              records=n[0] * n[1] * n[2], data_offset=52)
        return {"kind": kind, "lib": lib, "n": n, "xyz": xyz, "fields": fields, "info": info,
                "image": torch.empty(size, dtype=torch.uint8, device="cuda"), "out": torch.empty_like(fields)}
    if kind == "batch":
        prs = _batch_problems(case)
        vel = [_velocity(pr, seed * 1000 + i) for i, pr in enumerate(prs)]
        store = {k: _Store([pr.ttc for pr in prs]) for k in _SOLVE_KEYS}
        for i, v in enumerate(vel):
            for k, a in zip(("ustar", "vstar", "wstar", "u", "v", "w"), v + v):
                store[k].block(i).copy_(a)
        prec = abi.MF3D_PREC_FP32 if case["precision"] == "fp32" else abi.MF3D_PREC_FP64
        prm = prs[0].params(mg_itrsch=3, maxcy=case["maxcy"], eps=case["tol"], precision=prec)
        prm.ngrid = 1
        return {"kind": kind, "store": store, "call": Batch([domain_desc(pr) for pr in prs], prm, lib),
                "blocks": [{k: s.block(i) for k, s in store.items()} for i in range(len(prs))]}
    pr = _problem(case)
    if kind == "predictor":
        store = {k: _cut(pr, a) for k, a in zip("uvw", _velocity(pr, seed, mirror=True))}
        g = _gen(seed + 5)
        for k, src in (("uoo", "u"), ("voo", "v"), ("woo", "w")):
            store[k] = _Store([pr.ttc] * pr.nblocks)
            store[k].flat.copy_(store[src].flat)
            store[k].flat += 0.1 * torch.randn(store[k].flat.shape, generator=g, device="cuda", dtype=torch.float64)
        store["vis"] = _cut(pr, 1e-3 * (1.0 + torch.rand((pr.NZ + 2 * pr.pl, pr.NY + 2 * pr.pl, pr.NX + 2 * pr.pl),
                                                         generator=g, device="cuda", dtype=torch.float64)))
        for k in ("ustar", "vstar", "wstar", "p"):
            store[k] = _Store([pr.ttc] * pr.nblocks)
        prm = pr.params(bounds=1, alfabc=1, pl_ex=pr.pl - 2, differencing=case["scheme"])
        proj = Projection(pr.descriptors(lib), prm, lib)
        fa, ra = (abi.Fields * pr.nblocks)(), (RkFields * pr.nblocks)()
        for b in range(pr.nblocks):
            for arr, keys in ((fa, _SOLVE_KEYS), (ra, ("uoo", "voo", "woo", "vis"))):
                for k in keys:
                    setattr(arr[b], k, C.cast(C.c_void_p(store[k].block(b).data_ptr()), _DP))
        return {"kind": kind, "lib": lib, "store": store, "proj": proj, "fields": fa, "rk": ra, "dt": case["dt"],
                "alfapr": case["alfapr"], "forcing": int(case["forcing"]), "problem": pr}
    vel = _velocity(pr, seed, mirror=case["bounds"])
    store = {k: _cut(pr, a) for k, a in zip(("ustar", "vstar", "wstar", "u", "v", "w"), vel + vel)}
    store["p"] = _Store([pr.ttc] * pr.nblocks)
    if case["density"]:
        store["dens"] = _cut(pr, _density(pr, seed))
    blocks = [{k: s.block(b) for k, s in store.items()} for b in range(pr.nblocks)]
    state = {"kind": kind, "problem": pr, "call": Projection(pr.descriptors(lib), _params(pr, case), lib)}
    if kind == "host":
        blocks = [{k: f[k].cpu().numpy() for k in _SOLVE_KEYS} | {"su": np.zeros(pr.ttc)} for f in blocks]
    else:
        state["store"] = store
    state["blocks"] = blocks
    return state


def _course(state, r):
    """A solve's residual history (zeros after its last iteration) and count."""
    hist = np.zeros(state["call"].params.maxcy)
    hist[:len(r.history)] = r.history
    return {"history": hist, "iterations": r.iter}


def run(state):
    kind = state["kind"]
    if kind == "solve":
        state["store"]["p"].flat.zero_()
        r = state["call"].newsolv_mg_device(state["blocks"])
        return {**_course(state, r), **{k: state["store"][k].flat for k in ("p", "u", "v", "w")}}
    if kind == "host":
        for f in state["blocks"]:
            f["p"].fill(0.0)
        r = state["call"].newsolv_mg(state["blocks"])
        return {**_course(state, r),
                **{k: [f[k] for f in state["blocks"]] for k in ("p", "u", "v", "w")}}
    if kind == "batch":
        state["store"]["p"].flat.zero_()
        res, _ = state["call"].solve_device(state["blocks"])
        return {"rmax": np.array([r.rmax for r in res]), "iterations": np.array([r.iter for r in res]),
                **{k: state["store"][k].flat for k in ("p", "u", "v", "w")}}
    lib = state["lib"]
    if kind == "predictor":
        st = lib.mf3d_rungek_2nd_device(state["proj"].ctx, state["fields"], state["rk"], state["dt"],
                                        state["alfapr"], 1, state["forcing"], 0.31)
        abi.check(lib, st, "mf3d_rungek_2nd_device")
        return {k: state["store"][k].flat for k in ("ustar", "vstar", "wstar", "u", "v", "w")}
    n, vp = state["n"], C.c_void_p
    fields = (vp * 16)(*[f.data_ptr() for f in state["fields"]])
    outs = (vp * 16)(*[f.data_ptr() for f in state["out"]])
    img = vp(state["image"].data_ptr())
    st = lib.mf3d_tecbin_encode_device(n[2], n[1], n[0], 2, 0, -1, 0, *[vp(x.data_ptr()) for x in state["xyz"]], fields,
                                       img, 0)
    abi.check(lib, st, "mf3d_tecbin_encode_device")
    st = lib.mf3d_tecbin_decode_device(img, C.byref(state["info"]), outs, 0)
    abi.check(lib, st, "mf3d_tecbin_decode_device")
    return {"image": state["image"], "fields": state["out"]}


# ---------------------------------------------------------------------------
# work
# ---------------------------------------------------------------------------
def work(case):
    """Bytes: the inputs once and the outputs once - a solve's ustar, vstar,
    wstar, p in and u, v, w, p out (density in, where it varies).  Flops: the
    arithmetic of the outer iterations, whose number is a result."""
    kind = case["kind"]
    if kind == "restart":
        n = case["ti"] * case["tj"] * case["tk"]
        return {"bytes": 2.0 * n * (160 + 16 * 8), "flops": 0.0}
    if kind == "batch":
        n = sum(pr.nx * pr.ny * pr.nz for pr in _batch_problems(case))
        return {"bytes": 64.0 * n, "flops": 130.0 * n * case["iterations"]}
    n = case["px"] * case["py"] * case["pz"] * case["nx"] * case["ny"] * case["nz"]
    if kind == "predictor":
        return {"bytes": 80.0 * n, "flops": {1: 165.0, 2: 480.0, 3: 1150.0}[case["scheme"]] * n}
    # per cell and iteration: calvel/calmas and the update 30; three sweeps,
    # residual, restriction and prolongation over all levels (8/7), or SIP's
    # residual and two substitutions per sweep
    flops = 30.0 + (8 / 7 * (3 * 14 * (3 if case["smoother"] == "line" else 1) + 45) if not case["sip"]
                    else case["sip"] * 28.0)
    return {"bytes": (72.0 if case["density"] else 64.0) * n, "flops": flops * n * case["iterations"]}


# ---------------------------------------------------------------------------
# exact: plain torch in 64 bits
# ---------------------------------------------------------------------------
def _axis_modes(h, periodic):
    """Eigen-decomposition of (1/h) d(1/df d) along one axis: (T, Tinv, lam)
    with the operator = Tinv diag(lam) T."""
    n = h.numel()
    s = torch.zeros((n, n), dtype=torch.float64, device=h.device)
    for a in range(n if periodic else n - 1):
        b = (a + 1) % n
        g = 1.0 / (0.5 * (h[a] + h[b]))
        s[a, a] -= g
        s[b, b] -= g
        s[a, b] += g
        s[b, a] += g
    r = h.sqrt()
    lam, q = torch.linalg.eigh(s.cpu() / torch.outer(r, r).cpu())
    q = q.to(h.device)
    return q.T * r[None, :], q / r[:, None], lam.to(h.device)


def _projected(pr, vel):
    """The discretely divergence-free velocity nearest the given global one:
    u - grad p with div(u - grad p) = 0, by the axes' eigenvectors."""
    pl = pr.pl
    hs = []
    for ax, (n, d) in enumerate(((pr.NZ, pr.dz), (pr.NY, pr.dy), (pr.NX, pr.dx))):
        hy = pr.hy_global() if ax == 1 else None
        hs.append(torch.from_numpy(hy.copy()).cuda() if hy is not None else
                  torch.full((n,), d, dtype=torch.float64, device="cuda"))
    per = (pr.bc[4] == PERIODIC, pr.bc[2] == PERIODIC, pr.bc[0] == PERIODIC)
    comp = (2, 1, 0)  # the component normal to array axis 0, 1, 2
    div = 0.0
    sl = [slice(pl, -pl)] * 3
    for ax in range(3):
        a = vel[comp[ax]]
        low = list(sl)
        low[ax] = slice(pl - 1, -pl - 1)
        shape = [1, 1, 1]
        shape[ax] = -1
        div = div + (a[tuple(sl)] - a[tuple(low)]) / hs[ax].view(shape)
    modes = [_axis_modes(h, p) for h, p in zip(hs, per)]
    p = div
    for ax in range(3):
        p = torch.tensordot(modes[ax][0], p.movedim(ax, 0), dims=1).movedim(0, ax)
    lam = modes[0][2][:, None, None] + modes[1][2][None, :, None] + modes[2][2][None, None, :]
    small = lam.abs() < 1e-9 * lam.abs().max()
    p = torch.where(small, torch.zeros_like(p), p / torch.where(small, torch.ones_like(lam), lam))
    for ax in range(3):
        p = torch.tensordot(modes[ax][1], p.movedim(ax, 0), dims=1).movedim(0, ax)
    out = []
    for c in range(3):
        ax = 2 - c
        h = hs[ax]
        shape = [1, 1, 1]
        shape[ax] = -1
        grad = (torch.roll(p, -1, ax) - p) / (0.5 * (h + torch.roll(h, -1))).view(shape)
        if not per[ax]:
            grad.movedim(ax, 0)[-1] = 0.0
        a = vel[c].clone()
        a[tuple(sl)] -= grad
        out.append(_wrap(a, pr))
    return out


def _weno5(v1, v2, v3, v4, v5):
    e = 1.0e-6 * torch.stack([v * v for v in (v1, v2, v3, v4, v5)]).amax(0) + 1.0e-99
    s1 = 13.0 / 12.0 * (v1 - 2 * v2 + v3) ** 2 + 0.25 * (v1 - 4 * v2 + 3 * v3) ** 2
    s2 = 13.0 / 12.0 * (v2 - 2 * v3 + v4) ** 2 + 0.25 * (v2 - v4) ** 2
    s3 = 13.0 / 12.0 * (v3 - 2 * v4 + v5) ** 2 + 0.25 * (3 * v3 - 4 * v4 + v5) ** 2
    a1, a2, a3 = 0.1 / (e + s1) ** 2, 0.6 / (e + s2) ** 2, 0.3 / (e + s3) ** 2
    return (a1 * (v1 / 3 - 7 * v2 / 6 + 11 * v3 / 6) + a2 * (-v2 / 6 + 5 * v3 / 6 + v4 / 3)
            + a3 * (v3 / 3 + 5 * v4 / 6 - v5 / 6)) / (a1 + a2 + a3)


def _stage(pr, case, f, b, comp):
    """The predicted component of block b over its faces, from the block's
    own arrays (ghosts included); returns (values, slices)."""
    pl, h, scheme = pr.pl, case["spacing"], case["scheme"]
    pos, num = pr.block_pos(b), (pr.px, pr.py, pr.pz)
    size = [pr.nx, pr.ny, pr.nz]
    for ax in range(3):
        if ax == comp and pos[ax] == num[ax] - 1 and pr.bc[2 * ax + 1] != PERIODIC:
            size[ax] -= 1
    sl = tuple(slice(pl, pl + size[2 - q]) for q in range(3))

    def at(a, *shifts):
        m = [0, 0, 0]
        for ax, s in shifts:
            m[ax] += s
        return a[tuple(slice(sl[q].start + m[2 - q], sl[q].stop + m[2 - q]) for q in range(3))]

    vel = (f["u"], f["v"], f["w"])
    c = vel[comp]
    conv = 0.0
    for ax in range(3):
        if scheme == 1:
            if ax == comp:
                t = ((0.5 * (at(c) + at(c, (ax, 1)))) ** 2 - (0.5 * (at(c) + at(c, (ax, -1)))) ** 2) / h
            else:
                w = vel[ax]
                t = 0.25 * ((at(w) + at(w, (comp, 1))) * (at(c) + at(c, (ax, 1)))
                            - (at(w, (ax, -1)) + at(w, (ax, -1), (comp, 1))) * (at(c) + at(c, (ax, -1)))) / h
        elif scheme == 2:
            def mid(a, x, *base):
                return (-at(a, *base, (x, 1)) + 9 * at(a, *base) + 9 * at(a, *base, (x, -1))
                        - at(a, *base, (x, -2))) / 16
            if ax == comp:
                q = [mid(c, ax, (ax, m)) ** 2 for m in (2, 1, 0, -1)]
            else:
                q = [mid(c, ax, (ax, m + 1)) * mid(vel[ax], comp, (ax, m), (comp, 1)) for m in (1, 0, -1, -2)]
            t = (-q[0] + 27 * q[1] - 27 * q[2] + q[3]) / (24 * h)
        else:
            adv = at(c) if ax == comp else 0.25 * (at(vel[ax]) + at(vel[ax], (comp, 1)) + at(vel[ax], (ax, -1))
                                                   + at(vel[ax], (ax, -1), (comp, 1)))
            d = [(at(c, (ax, m + 1)) - at(c, (ax, m))) / h for m in range(-3, 3)]
            up, down = _weno5(*d[:5]), _weno5(d[5], d[4], d[3], d[2], d[1])
            der = torch.where(adv > 0, up, torch.where(adv < 0, down, torch.zeros_like(up)))
            lim = size[ax] + pl + (pl - 2) + 1  # derivatives exist on cells 4 .. lim-3 (1-based)
            idx = torch.arange(size[ax], device=der.device) + pl + 1
            shape = [1, 1, 1]
            shape[2 - ax] = -1
            t = adv * der * ((idx >= 4) & (idx <= lim - 3)).view(shape)
        conv = conv + t
    vis = at(f["vis"]) if scheme == 2 and comp == 0 else at(f["vis"], (comp, 1))
    lap = 0.0
    for ax in range(3):
        if scheme == 2:
            lap = lap + (-at(c, (ax, 2)) + 16 * at(c, (ax, 1)) - 30 * at(c) + 16 * at(c, (ax, -1))
                         - at(c, (ax, -2))) / (12 * h * h)
        else:
            lap = lap + (at(c, (ax, 1)) - 2 * at(c) + at(c, (ax, -1))) / (h * h)
    oo = f[("uoo", "voo", "woo")[comp]]
    da = case["dt"] * case["alfapr"]
    return at(oo) - da * conv + da * vis * lap + (da * 0.31 if comp == 0 and case["forcing"] else 0.0), sl


def exact(case, seed):
    kind = case["kind"]
    if kind == "restart":
        s = prepare(case, seed)
        n, nrec = s["n"], s["info"].records
        rec = torch.empty((nrec, 19), dtype=torch.float64, device="cuda")
        z, y, x = torch.meshgrid(*[s["xyz"][q] for q in (2, 1, 0)], indexing="ij")
        for q, a in enumerate((x, y, z)):
            rec[:, q] = a.reshape(-1)
        rec[:, 3:] = s["fields"].reshape(16, -1).T
        words = torch.full((nrec, 40), 152, dtype=torch.int32, device="cuda")
        words[:, 1:39] = rec.view(torch.int32).view(nrec, 38)
        head = torch.tensor([12, n[2], n[1], n[0], 12, 4, 2, 4, 12, 0, -1, 0, 12], dtype=torch.int32, device="cuda")
        return {"image": torch.cat([head, words.reshape(-1)]).view(torch.uint8), "fields": s["fields"]}
    if kind == "predictor":
        s = prepare(case, seed)
        pr, store = s["problem"], s["store"]
        out = {k: _Store([pr.ttc] * pr.nblocks) for k in ("ustar", "vstar", "wstar")}
        for b in range(pr.nblocks):
            f = {k: v.block(b) for k, v in store.items()}
            for comp, k in enumerate(out):
                val, sl = _stage(pr, case, f, b, comp)
                out[k].block(b)[sl] = val
        # the inputs' ghosts are already what boundu/v/w give
        return {**{k: v.flat for k, v in out.items()}, **{k: store[k].flat for k in "uvw"}}
    if kind == "batch":
        prs = _batch_problems(case)
        out = {k: _Store([pr.ttc for pr in prs]) for k in "uvw"}
        for i, pr in enumerate(prs):
            vel = _velocity(pr, seed * 1000 + i)
            for k, a, given in zip("uvw", _projected(pr, vel), vel):
                o = out[k].block(i)
                o.copy_(given)
                _face_ghosts(o, a, pr.pl)
        return {"rmax": None, "iterations": None, "p": None, **{k: v.flat for k, v in out.items()}}
    if case["density"] or case["sip"]:
        return None  # the fixed number of cycles ends before convergence: no value but the iteration's own
    pr = _problem(case)
    vel = _velocity(pr, seed, mirror=case["bounds"])
    new = _projected(pr, vel)
    if case["bounds"]:
        new = [_wrap(a, pr) for a in _walls(new, pr, True)]
    out = {"history": None, "iterations": None, "p": None}
    # ghost layers past 0..pl_ex are no exchange's: as given.  (Where several
    # blocks meet, some ghost edges hold an earlier iteration's value or a
    # neighbour's; they have no value of their own and stay as formed here.)
    deep = [(d < pr.pl - 1 - case["pl_ex"]) for d in
            (torch.minimum(torch.arange(n, device="cuda"), torch.arange(n - 1, -1, -1, device="cuda")) for n in pr.ttc)]
    keep = deep[0][:, None, None] | deep[1][None, :, None] | deep[2][None, None, :]
    for k, a, given in zip("uvw", new, vel):
        st, old = _cut(pr, a), _cut(pr, given)
        for b in range(pr.nblocks):
            st.block(b).copy_(torch.where(keep, old.block(b), st.block(b)))
        out[k] = st.flat if kind == "solve" else [st.block(b).cpu().numpy() for b in range(pr.nblocks)]
    return out


def _face_ghosts(o, a, pl):
    """A batch domain's velocity: interior cells and the first ghost layer
    over the faces (ghost edges stay as given)."""
    s = slice(pl, -pl)
    o[s, s, s] = a[s, s, s]
    for ax in range(3):
        for g in (pl - 1, -pl):
            at = [s, s, s]
            at[ax] = g
            o[tuple(at)] = a[tuple(at)]
