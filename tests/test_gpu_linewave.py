"""Line relaxation (mg_itrsch 2) at the edges of its launch shapes, bit for
bit against the oracle: one CTA and clusters, slices with a short last CTA,
ragged line lengths in the three directions, diagonals shorter than a slice,
more lines than a warp's lanes a CTA (the staged kernel), two blocks of one
level side by side, and the FP32 V-cycle within rounding."""
import numpy as np
import pytest

from multiflow3d_b200 import abi
from multiflow3d_b200.problems import Problem, PERIODIC, WALL
from multiflow3d_b200.solver import Projection
from test_gpu_edges import run_both, assert_same

pytestmark = pytest.mark.gpu
P, W = PERIODIC, WALL

# nx, ny, nz, blocks, levels
SHAPES = {
    "one line": (1, 1, 9, (1, 1, 1), 1),
    "one CTA": (5, 7, 3, (1, 1, 1), 1),
    "one CTA, 31 lines": (31, 30, 9, (1, 1, 1), 1),
    "a cluster of four": (33, 32, 20, (1, 1, 1), 1),
    "short last slice": (37, 33, 50, (1, 1, 1), 1),
    "long j": (8, 64, 16, (1, 1, 1), 3),
    "long k": (40, 6, 90, (1, 1, 1), 1),
    "25 lines a CTA": (200, 8, 8, (1, 1, 1), 2),
    "past 32 lines a CTA": (300, 4, 6, (1, 1, 1), 1),
    "two blocks, three levels": (32, 16, 24, (2, 1, 2), 3),
}


@pytest.mark.parametrize("shape", sorted(SHAPES))
def test_line_relaxation_matches_oracle(lib, oracle, cuda, shape):
    nx, ny, nz, (px, py, pz), levels = SHAPES[shape]
    pr = Problem(px, py, pz, nx, ny, nz, bc=(P, P, W, W, P, P), ngrid=levels, pl=1, stretch_y=1.5 if ny > 8 else 0.0,
                 dx=0.017, dy=0.017, dz=0.017)
    prm = pr.params(mg_itrsch=2, maxcy=4, eps=1e-12)
    o, g = run_both(lib, oracle, cuda, pr.descriptors(lib), pr.descriptors(oracle), pr.nblocks, prm,
                    pr.block_fields(seed=51, fourier_modes=2))
    assert_same(o, g, pr.pl)


def test_line_relaxation_fp32_converges(lib, cuda):
    """The FP32 V-cycle with line smoothing reaches the FP64 pressure: both
    solves stop at 1e-9 of the initial rmax, so they differ by a small multiple
    of that."""
    import torch
    pr = Problem(2, 1, 1, 32, 40, 24, ngrid=3, pl=1, stretch_y=1.5, dx=1 / 64, dy=1 / 64, dz=1 / 64)
    out = []
    for prec in (abi.MF3D_PREC_FP64, abi.MF3D_PREC_FP32):
        d = [{k: torch.from_numpy(v).to(cuda) for k, v in f.items()} for f in pr.block_fields(seed=52)]
        proj = Projection(pr.descriptors(lib), pr.params(mg_itrsch=2, maxcy=100, eps=1e-9, precision=prec), lib)
        res = proj.newsolv_mg_device(d)
        proj.close()
        assert res.status == 0
        p = pr.gather([{k: t.cpu().numpy() for k, t in f.items()} for f in d], "p")
        out.append(p - p.mean())
    assert np.linalg.norm(out[1] - out[0]) / np.linalg.norm(out[0]) < 1e-6


# levels of one and two planes, where a line is shorter than a batch of the
# recurrences and its coefficients are the last of the shared memory
THIN = {
    "one plane": (9, 6, 1, (1, 1, 1), 1),
    "two planes, clusters": (40, 33, 2, (1, 1, 1), 1),
    "a line of seven": (16, 12, 7, (1, 1, 1), 1),
    "coarsest 4x4x1": (64, 64, 16, (1, 1, 1), 5),
    "coarsest 4x4x2": (32, 32, 16, (1, 1, 1), 4),
    "coarsest 8x8x2, two blocks": (32, 32, 8, (2, 1, 1), 3),
    "coarsest 1x2x4": (16, 32, 64, (1, 1, 1), 5),
}


@pytest.mark.parametrize("shape", sorted(THIN))
def test_thin_levels_match_oracle(lib, oracle, cuda, shape):
    nx, ny, nz, (px, py, pz), levels = THIN[shape]
    pr = Problem(px, py, pz, nx, ny, nz, bc=(P, P, W, W, W, W), ngrid=levels, pl=1, dx=0.017, dy=0.017, dz=0.017)
    prm = pr.params(mg_itrsch=2, maxcy=3, eps=1e-12)
    o, g = run_both(lib, oracle, cuda, pr.descriptors(lib), pr.descriptors(oracle), pr.nblocks, prm,
                    pr.block_fields(seed=53, fourier_modes=0))
    assert_same(o, g, pr.pl)
