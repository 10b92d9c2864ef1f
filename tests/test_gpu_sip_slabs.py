"""solver 1 (Stone's SIP) at the edges of its substitution launches, bit for
bit against the oracle: a warp per segment of 32 columns, slabs of rows over
up to 8 CTAs (a short last one, an empty one, full ones, two blocks), lines
longer and shorter than the rings, 16 and 32 warps a CTA, and planes past
that (a launch per hyperplane)."""
import pytest

from multiflow3d_b200.problems import Problem, WALL
from test_gpu_edges import run_both, assert_same

pytestmark = pytest.mark.gpu

# (nx, ny, nz, blocks, nswp)
PLANES = {
    "one column": (1, 1, 2, (1, 1, 1), 3),
    "one row, long lines": (31, 1, 70, (1, 1, 1), 2),
    "full segments": (32, 32, 5, (1, 1, 1), 4),
    "lines past the shared memory": (40, 30, 150, (1, 1, 1), 2),
    "an empty slab": (20, 33, 6, (1, 1, 1), 4),
    "two segments, the second one lane": (33, 17, 18, (1, 1, 1), 9),
    "two blocks, short last slab": (45, 50, 4, (1, 2, 1), 17),
    "128 segments": (128, 32, 3, (1, 1, 1), 2),
    "32 warps": (200, 20, 9, (1, 1, 1), 2),
    "256 segments": (1000, 8, 3, (1, 1, 1), 2),
    "past 256 segments": (129, 65, 3, (1, 1, 1), 2),
    "a row past 1024 columns": (1030, 2, 3, (1, 1, 1), 2),
}


@pytest.mark.parametrize("plane", sorted(PLANES))
def test_substitution_launches_match_oracle(lib, oracle, cuda, plane):
    nx, ny, nz, (px, py, pz), nswp = PLANES[plane]
    pr = Problem(px, py, pz, nx, ny, nz, bc=(WALL,) * 6, ngrid=1, pl=1, dx=0.013, dy=0.013, dz=0.013)
    prm = pr.params(maxcy=5, eps=1e-9, solver=1, nswp=nswp)
    o, g = run_both(lib, oracle, cuda, pr.descriptors(lib), pr.descriptors(oracle), pr.nblocks, prm,
                    pr.block_fields(seed=44, fourier_modes=0))
    assert o[0] in (0, 1)
    assert_same(o, g, pr.pl)
