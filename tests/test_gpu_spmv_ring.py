"""The sparse product's ring of matrix tiles fits the shared memory there is:
fewer 32-row slices per tile, then fewer stages."""
import numpy as np
import pytest

from conftest import rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_rhs", [1, 4, 8, 16])
@pytest.mark.parametrize("precision", [0, 1])
def test_small_shared_memory(lib, n_rhs, precision):
    """201 k edges (up to 24 slices a tile).  Limits from two slices (the least, 8 KB
    in FP32) upwards: the same systems solved to 1e-10, 1e-6 apart at most as in
    the oracle comparisons; the ring's shape changes the order of the sums alone."""
    from maple3dmt_gb300 import mesh
    from maple3dmt_gb300.solver import solver_for_survey
    sv = mesh.layered_block_survey(min_level=5, max_level=6, n_side=5, freqs=np.array([10.0]))
    s = solver_for_survey(sv, bicgstab_tol=1e-10, bicgstab_maxiter=5000, precision=precision)
    s.factorize_frequency(10.0)
    rng = np.random.default_rng(n_rhs)
    b = rng.normal(size=(n_rhs, s.ne)) + 1j * rng.normal(size=(n_rhs, s.ne))
    want = s.solve_rhs_batch(b)
    for limit in (1, 17 * 1024, 30 * 1024, 65 * 1024, 120 * 1024):
        s.test_set_smem_limit(limit)
        got = s.solve_rhs_batch(b)
        assert s.stats()["status"][:n_rhs] == [1] * n_rhs
        assert rel(got, want) < 1e-6
    s.test_set_smem_limit(0)
    assert np.array_equal(s.solve_rhs_batch(b), want)
