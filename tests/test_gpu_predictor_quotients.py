"""The predictor's quotients without a division each, and its periodic copies
with a partner behind every face, bit for bit against the oracle: spacings
that are powers of two, are not, or are outside the reciprocal's range;
velocities that make numerators zero, subnormal and huge; ragged tiles; and
two blocks along every axis, all ghost layers compared."""
import ctypes as C

import numpy as np
import pytest

from multiflow3d_b200 import abi
from multiflow3d_b200.abi import RkFields
from multiflow3d_b200.problems import Problem, PERIODIC, WALL
from multiflow3d_b200.solver import Projection
from test_rungek import rk_inputs, orc_rk

pytestmark = pytest.mark.gpu
P, W = PERIODIC, WALL
PL = {1: (2, 1), 2: (3, 1), 3: (4, 2)}  # differencing: pl, pl_ex


def run(lib, oracle, cuda, pr, differencing, edit):
    import torch
    pl_ex = PL[differencing][1]
    blocks, rk = rk_inputs(pr, 31)
    edit(blocks, rk)
    dt, alfapr, forcn = 0.0137, 1.0 / 3.0, 0.31
    gpu = [{k: torch.from_numpy(v.copy()).to(cuda) for k, v in f.items()} for f in blocks]
    grk = [{k: torch.from_numpy(v.copy()).to(cuda) for k, v in r.items()} for r in rk]
    assert orc_rk(oracle, pr, blocks, rk, dt, alfapr, pforce=1, forcn=forcn, pl_ex=pl_ex,
                  differencing=differencing) == 0
    proj = Projection(pr.descriptors(lib), pr.params(pl_ex=pl_ex, bounds=1, differencing=differencing), lib)
    fa, ra = (abi.Fields * pr.nblocks)(), (RkFields * pr.nblocks)()
    dp = C.POINTER(C.c_double)
    for b in range(pr.nblocks):
        for arr, src, keys in ((fa, gpu, ("ustar", "vstar", "wstar", "u", "v", "w", "p")),
                               (ra, grk, ("uoo", "voo", "woo", "vis"))):
            for k in keys:
                setattr(arr[b], k, C.cast(C.c_void_p(src[b][k].data_ptr()), dp))
    st = lib.mf3d_rungek_2nd_device(proj.ctx, fa, ra, dt, alfapr, 1, 1, forcn)
    abi.check(lib, st, "mf3d_rungek_2nd_device")
    proj.close()
    for b in range(pr.nblocks):
        for k in ("ustar", "vstar", "wstar", "u", "v", "w"):
            got = gpu[b][k].cpu().numpy()
            assert np.array_equal(got, blocks[b][k], equal_nan=True), (b, k, np.argwhere(got != blocks[b][k])[:4])


def scale(s):
    def edit(blocks, rk):
        for f, r in zip(blocks, rk):
            for k in ("u", "v", "w"):
                f[k] *= s
            for k in ("uoo", "voo", "woo"):
                r[k] *= s
    return edit


def patches(blocks, rk):
    """Zero, tiny and huge cells side by side, a cell without viscosity."""
    for f, r in zip(blocks, rk):
        for k in ("u", "v", "w"):
            f[k][:, :, ::3] = 0.0
            f[k][:, 1::4, :] *= 1e-170
            f[k][2::5, :, :] *= 1e120
        r["vis"][::2, ::2, ::2] = 0.0


FIELDS = {"as drawn": scale(1.0), "zero": scale(0.0), "1e-160": scale(1e-160), "1e+140": scale(1e140), "patches": patches}


@pytest.mark.parametrize("differencing", [1, 2, 3])
@pytest.mark.parametrize("spacing", [1 / 64, 0.0107, 2.0 ** -60])
@pytest.mark.parametrize("field", sorted(FIELDS))
def test_quotients(lib, oracle, cuda, differencing, spacing, field):
    pr = Problem(1, 1, 1, 35, 9, 10, bc=(P, P, W, W, P, P), ngrid=1, pl=PL[differencing][0], dx=spacing, dy=spacing,
                 dz=spacing)
    with np.errstate(all="ignore"):
        run(lib, oracle, cuda, pr, differencing, FIELDS[field])


@pytest.mark.parametrize("differencing", [1, 2, 3])
@pytest.mark.parametrize("bc", [(P,) * 6, (P, P, W, W, P, P), (W, W, P, P, W, W)])
def test_periodic_partners(lib, oracle, cuda, differencing, bc):
    pr = Problem(2, 2, 2, 9, 7, 8, bc=bc, ngrid=1, pl=PL[differencing][0], dx=0.02, dy=0.03, dz=1 / 32)
    run(lib, oracle, cuda, pr, differencing, scale(1.0))
