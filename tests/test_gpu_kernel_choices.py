"""Kernels that a rule on sizes keeps away from small grids, on small grids: the
half-sweep with copies (k_rbgs) on odd, thin and ragged blocks, and calvel and
calmas with 4, 8 and 16 planes a CTA and a short last run, bit for bit against
the oracle; the FP32 V-cycle's two half-sweep kernels bit for bit against each
other."""
import numpy as np
import pytest

from multiflow3d_b200 import abi
from multiflow3d_b200.problems import Problem, PERIODIC, WALL
from multiflow3d_b200.solver import Projection
from test_gpu_edges import run_both, assert_same, ragged_blocks

pytestmark = pytest.mark.gpu
P, W = PERIODIC, WALL

# nx, ny, nz, blocks, levels, boundaries
SWEEPS = {
    "7x5x3": (7, 5, 3, (1, 1, 1), 1, (P, P, W, W, P, P)),
    "one cell wide": (1, 9, 6, (1, 1, 1), 1, (W,) * 6),
    "past a tile each way": (65, 17, 9, (1, 1, 1), 1, (P, P, W, W, W, W)),
    "thin in z": (66, 34, 2, (1, 1, 1), 1, (W,) * 6),
    "thin in x and y": (4, 4, 72, (1, 1, 1), 3, (P, P, P, P, W, W)),
    "odd halves": (10, 14, 6, (2, 1, 2), 2, (P, P, W, W, P, P)),
    "blocks of 21x33x17": (21, 33, 17, (2, 2, 1), 1, (W, W, P, P, W, W)),
}


@pytest.mark.parametrize("shape", sorted(SWEEPS))
def test_copy_sweep_matches_oracle(lib, oracle, cuda, shape, monkeypatch):
    monkeypatch.setenv("MF3D_SMALL_LEVEL_CELLS", "0")
    nx, ny, nz, (px, py, pz), levels, bc = SWEEPS[shape]
    pr = Problem(px, py, pz, nx, ny, nz, bc=bc, ngrid=levels, pl=1, dx=0.017, dy=0.017, dz=0.017)
    prm = pr.params(mg_itrsch=3, maxcy=6, eps=1e-12)
    seen = []
    o, g = run_both(lib, oracle, cuda, pr.descriptors(lib), pr.descriptors(oracle), pr.nblocks, prm,
                    pr.block_fields(seed=61, fourier_modes=0), prepare=lambda proj: seen.append(proj.tuning(1)))
    assert seen[0]["small_sweep"] == 0
    assert_same(o, g, pr.pl)


def test_copy_sweep_ragged_blocks(lib, oracle, cuda, monkeypatch):
    monkeypatch.setenv("MF3D_SMALL_LEVEL_CELLS", "0")
    bc = (P, P, W, W, W, W)
    args = ([18, 34, 7], 12, 10, 1 / 32, 1, bc, 62)
    arr, blocks = ragged_blocks(lib, *args)
    arr_o, _ = ragged_blocks(oracle, *args)
    pr = Problem(1, 1, 1, 59, 12, 10, bc=bc, ngrid=1, pl=1)
    prm = pr.params(mg_itrsch=3, maxcy=6, eps=1e-12)
    o, g = run_both(lib, oracle, cuda, arr, arr_o, 3, prm, blocks)
    assert_same(o, g, 1)


@pytest.mark.parametrize("shape", ["odd halves", "thin in x and y", "past a tile each way"])
def test_fp32_sweeps_agree(lib, cuda, shape, monkeypatch):
    import torch
    nx, ny, nz, (px, py, pz), levels, bc = SWEEPS[shape]
    pr = Problem(px, py, pz, nx, ny, nz, bc=bc, ngrid=max(levels, 1), pl=1, dx=0.017, dy=0.017, dz=0.017)
    prm = pr.params(mg_itrsch=3, maxcy=6, eps=1e-12, precision=abi.MF3D_PREC_FP32)
    out = []
    for limit in ("0", "100000000"):
        monkeypatch.setenv("MF3D_SMALL_LEVEL_CELLS", limit)
        d = [{k: torch.from_numpy(v).to(cuda) for k, v in f.items()} for f in pr.block_fields(seed=63)]
        proj = Projection(pr.descriptors(lib), prm, lib)
        res = proj.newsolv_mg_device(d)
        proj.close()
        out.append((res.history, [f["p"].cpu().numpy() for f in d]))
    assert np.array_equal(out[0][0], out[1][0])
    assert all(np.array_equal(a, b) for a, b in zip(out[0][1], out[1][1]))


def planes_per_cta(blocks, nx, ny, nz, resident):
    """The library's choice: the shortest of the marches that fill the device."""
    cost = {}
    for kc in (2, 4, 8, 16):
        tiles = blocks * -(-nx // 32) * -(-ny // 8) * -(-nz // kc)
        cost[kc] = -(-tiles // resident) * (kc + 3)
    return max(k for k in cost if cost[k] == min(cost.values()))


# blocks, spacing, y stretching, density, boundaries, x cells (34: the kernel
# with copies, 33: rows of odd length, plain loads), planes a CTA
MARCHES = {
    "4 planes": ((5, 3, 2), 0.02, 0.0, False, (P, P, W, W, P, P), 34, 4),
    "4 planes, stretched": ((5, 3, 2), 1 / 64, 1.5, False, (W,) * 6, 34, 4),
    "8 planes": ((5, 4, 3), 1 / 64, 0.0, False, (W, W, P, P, W, W), 34, 8),
    "8 planes, stretched": ((5, 4, 3), 0.02, 1.5, False, (P, P, W, W, W, W), 34, 8),
    "16 planes": ((5, 5, 4), 0.02, 0.0, False, (W,) * 6, 34, 16),
    "16 planes, powers of two": ((5, 5, 4), 1 / 64, 0.0, False, (P, P, W, W, P, P), 34, 16),
    "16 planes, stretched": ((5, 5, 4), 0.02, 1.5, False, (P, P, W, W, P, P), 34, 16),
    "16 planes, plain loads": ((5, 5, 4), 0.02, 1.5, False, (P, P, W, W, P, P), 33, 16),
    "4 planes, density": ((5, 5, 4), 0.02, 0.0, True, (P, P, W, W, P, P), 34, 4),
}


@pytest.mark.parametrize("march", sorted(MARCHES))
def test_calvel_march_matches_oracle(lib, oracle, cuda, march):
    import torch
    (px, py, pz), h, stretch, density, bc, nx, planes = MARCHES[march]
    pr = Problem(px, py, pz, nx, 9, 17, bc=bc, ngrid=1, pl=1, dx=h, dy=h, dz=h, stretch_y=stretch)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert planes_per_cta(pr.nblocks, nx, 9, 17, sms * (4 if density else 6)) == planes
    blocks = pr.block_fields(seed=64, fourier_modes=2)
    if density:
        for f, d in zip(blocks, pr.block_density(65)):
            f["dens"] = d
    prm = pr.params(mg_itrsch=3, maxcy=3, eps=1e-12, lsm=int(density))
    o, g = run_both(lib, oracle, cuda, pr.descriptors(lib), pr.descriptors(oracle), pr.nblocks, prm, blocks)
    assert_same(o, g, pr.pl)
