"""solver 1 (Stone's SIP) at the edges of its substitution launches, bit for
bit against the oracle: a warp per segment of 32 columns, slabs of rows over
up to 8 CTAs (a short last one, an empty one, full ones, two blocks), lines
longer and shorter than the rings, 16 and 32 warps a CTA, and planes past
that (a launch per hyperplane)."""
import pytest

from multiflow3d_b200 import abi
from multiflow3d_b200.problems import Problem, PERIODIC, WALL
from multiflow3d_b200.solver import Projection
from test_gpu_edges import run_both, assert_same, ragged_blocks
from test_gpu_failures import _dev, _solve

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


@pytest.mark.parametrize("plane", ["full segments", "32 warps", "lines past the shared memory",
                                   "two segments, the second one lane", "two blocks, short last slab"])
def test_withheld_value_times_out(lib, cuda, plane):
    """The first row segment withholds its values: the warps that wait for them,
    or for room in a ring, give up within their limit (2 s), each as a whole, the
    call returns MF3D_E_TIMEOUT, and the next call on the context equals a fresh
    context's."""
    nx, ny, nz, (px, py, pz), nswp = PLANES[plane]
    pr = Problem(px, py, pz, nx, ny, nz, bc=(WALL,) * 6, ngrid=1, pl=1, dx=0.013, dy=0.013, dz=0.013)
    prm = pr.params(maxcy=3, eps=1e-9, solver=1, nswp=nswp)
    host = pr.block_fields(seed=45, fourier_modes=0)
    proj = Projection(pr.descriptors(lib), prm, lib)
    assert lib.mf3d_test_stall_copy(0, 16) == abi.MF3D_OK
    st, _, _ = _solve(lib, proj, _dev(pr, host, cuda), prm.maxcy)
    lib.mf3d_test_stall_copy(0, 0)
    assert st == abi.MF3D_E_TIMEOUT, st
    assert "time limit" in abi.last_error(lib)
    out = []
    for call in (proj, Projection(pr.descriptors(lib), prm, lib)):
        d = _dev(pr, host, cuda)
        st, info, hist = _solve(lib, call, d, prm.maxcy)
        call.close()
        out.append((st, info.iter, hist.tolist(), [f["p"].cpu() for f in d]))
    assert out[0][:3] == out[1][:3]
    for a, b in zip(out[0][3], out[1][3]):
        assert a.equal(b)


def _launches(lib, cuda, cells, blocks, nswp):
    pr = Problem(*blocks, *cells, bc=(WALL,) * 6, ngrid=1, pl=1, dx=0.013, dy=0.013, dz=0.013)
    prm = pr.params(maxcy=2, eps=1e-30, solver=1, nswp=nswp)
    proj = Projection(pr.descriptors(lib), prm, lib)
    proj.newsolv_mg_device(_dev(pr, pr.block_fields(seed=46, fourier_modes=0), cuda))
    n = proj.launches
    proj.close()
    return n


# planes that one CTA walks: past 256 segments, and where the rows' warps would
# mostly wait (nx, ny, nz, blocks, nswp)
CTA_PLANES = {
    "a thread per column": (3, 300, 4, (1, 1, 1), 3),
    "1024 columns": (4, 256, 2, (1, 1, 1), 2),
    "a column of 1000 rows": (1, 1000, 3, (1, 1, 1), 2),
    "several columns a thread": (5, 300, 3, (1, 1, 1), 3),
    "4096 columns": (2, 2048, 2, (1, 1, 1), 2),
    "a wide row": (1100, 2, 3, (1, 1, 1), 2),
    "few lanes, tall": (2, 200, 8, (1, 1, 1), 9),
    "two tall blocks": (3, 140, 5, (1, 2, 1), 2),
    "many blocks": (4, 130, 2, (4, 2, 2), 2),
}


@pytest.mark.parametrize("plane", sorted(CTA_PLANES))
def test_cta_planes_match_oracle(lib, oracle, cuda, plane):
    nx, ny, nz, (px, py, pz), nswp = CTA_PLANES[plane]
    pr = Problem(px, py, pz, nx, ny, nz, bc=(WALL,) * 6, ngrid=1, pl=1, dx=0.013, dy=0.013, dz=0.013)
    prm = pr.params(maxcy=4, eps=1e-9, solver=1, nswp=nswp)
    o, g = run_both(lib, oracle, cuda, pr.descriptors(lib), pr.descriptors(oracle), pr.nblocks, prm,
                    pr.block_fields(seed=47, fourier_modes=0))
    assert_same(o, g, pr.pl)
    # one launch for both substitutions, which adds to pp as well (k_sip_subst
    # leaves that to a second launch)
    if pr.nblocks == 1:
        rows = _launches(lib, cuda, (32, 32, 5), (1, 1, 1), 2) - _launches(lib, cuda, (32, 32, 5), (1, 1, 1), 1)
        here = _launches(lib, cuda, (nx, ny, nz), (1, 1, 1), 2) - _launches(lib, cuda, (nx, ny, nz), (1, 1, 1), 1)
        assert here == rows - 2  # two calls


def test_no_launches_past_the_stop(lib, cuda):
    """A call whose sweeps stop before their budget queues no hyperplane launches
    for the rest: the launches tell the sweeps run, the pressure is that of
    exactly so many, and one sweep less gives another."""
    pr = Problem(1, 1, 1, 129, 65, 2, bc=(WALL,) * 6, ngrid=1, pl=1, dx=0.013, dy=0.013, dz=0.013)
    host = pr.block_fields(seed=48, fourier_modes=0)

    def call(nswp):
        proj = Projection(pr.descriptors(lib), pr.params(maxcy=1, eps=1e-30, solver=1, nswp=nswp), lib)
        d = _dev(pr, host, cuda)
        proj.newsolv_mg_device(d)
        n = proj.launches
        proj.close()
        return n, d[0]["p"].cpu()

    one, two, (many, p) = call(1)[0], call(2)[0], call(400)
    sweeps, rest = divmod(many - one, two - one)
    assert rest == 0 and 1 < sweeps < 399
    assert p.equal(call(sweeps + 1)[1])
    assert not p.equal(call(sweeps)[1])


def test_a_timeout_ends_the_call(lib, cuda):
    """After a wait gave up the call ends with its round, says which wait it was,
    and runs no further sweeps or rounds on what is left."""
    pr = Problem(1, 1, 1, 32, 32, 5, bc=(WALL,) * 6, ngrid=1, pl=1, dx=0.013, dy=0.013, dz=0.013)
    prm = pr.params(maxcy=200, eps=1e-30, solver=1, nswp=20)
    host = pr.block_fields(seed=49, fourier_modes=0)
    proj = Projection(pr.descriptors(lib), prm, lib)
    _solve(lib, proj, _dev(pr, host, cuda), prm.maxcy)
    whole = proj.launches
    assert lib.mf3d_test_stall_copy(0, 16) == abi.MF3D_OK
    st, _, _ = _solve(lib, proj, _dev(pr, host, cuda), prm.maxcy)
    lib.mf3d_test_stall_copy(0, 0)
    stalled = proj.launches
    proj.close()
    assert st == abi.MF3D_E_TIMEOUT and "SIP" in abi.last_error(lib)
    assert stalled < whole / 100


# lines past a CTA's shared memory with 12, 16 and more than 16 warps a CTA: the
# rings are used again and again, across the slabs of a cluster
RINGS = {
    "12 warps": (48, 48, 48, 2),
    "16 warps": (64, 64, 40, 2),
    "16 warps, one segment": (20, 128, 60, 2),
    "32 warps, many rounds": (200, 20, 60, 2),
    "32 warps, short last slab": (32, 235, 40, 1),
}


@pytest.mark.parametrize("plane", sorted(RINGS))
def test_rings_match_oracle(lib, oracle, cuda, plane):
    nx, ny, nz, nswp = RINGS[plane]
    pr = Problem(1, 1, 1, nx, ny, nz, bc=(WALL,) * 6, ngrid=1, pl=1, dx=0.013, dy=0.013, dz=0.013)
    prm = pr.params(maxcy=3, eps=1e-9, solver=1, nswp=nswp)
    o, g = run_both(lib, oracle, cuda, pr.descriptors(lib), pr.descriptors(oracle), pr.nblocks, prm,
                    pr.block_fields(seed=50, fourier_modes=0))
    assert_same(o, g, pr.pl)
    rows = _launches(lib, cuda, (32, 32, 5), (1, 1, 1), 2) - _launches(lib, cuda, (32, 32, 5), (1, 1, 1), 1)
    here = _launches(lib, cuda, (nx, ny, nz), (1, 1, 1), 2) - _launches(lib, cuda, (nx, ny, nz), (1, 1, 1), 1)
    assert here == rows


def test_rings_ragged_blocks(lib, oracle, cuda):
    bc = (PERIODIC, PERIODIC, WALL, WALL, WALL, WALL)
    args = ([40, 64, 21], 48, 70, 1 / 32, 1, bc, 51)
    arr, blocks = ragged_blocks(lib, *args)
    arr_o, _ = ragged_blocks(oracle, *args)
    pr = Problem(1, 1, 1, 125, 48, 70, bc=bc, ngrid=1, pl=1)
    o, g = run_both(lib, oracle, cuda, arr, arr_o, 3, pr.params(maxcy=3, eps=1e-9, solver=1, nswp=3), blocks)
    assert_same(o, g, 1)
