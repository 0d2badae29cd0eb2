"""Which meshes take the multigrid preconditioner: host rule."""
import pytest


@pytest.mark.parametrize("lmin", range(0, 13))
@pytest.mark.parametrize("gap", range(0, 6))
def test_levels(lib, lmin, gap):
    """Level 2 (a 4^3 grid) at least, three levels of leaves under the coarsest
    grid at most, and grids whose kernels number their threads in 32 bits: an
    entry has three edges a point and eight pairs of right-hand sides."""
    ok = lib.m3d_test_multigrid_levels(lmin, lmin + gap)
    assert ok == (2 <= lmin <= 8 and gap <= 3)
    if ok:
        assert 3 * (2 ** lmin + 1) ** 3 * 8 + 256 < 2 ** 31
