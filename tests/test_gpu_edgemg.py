"""The geometric multigrid preconditioner of the mixed-precision solve: meshes
at the edges of its rule (coarsest grid only, one and two grids in the bottom
kernel, grids above it, zero to three levels of leaves under the uniform
grid), every batch width, against the all-FP64 solver, which the oracle tests
pin.  Both stop at the 1e-10 FP64 true residual, so fields and impedances
agree to 1e-6 as in the oracle comparisons."""
import numpy as np
import pytest

from conftest import rel

pytestmark = pytest.mark.gpu

TOL = 1e-6


def _survey(lo, hi, freqs):
    from maple3dmt_gb300 import mesh
    return mesh.small_survey(min_level=lo, max_level=hi, freqs=freqs)


@pytest.mark.parametrize("lo,hi", [(2, 2), (2, 4), (2, 5), (3, 3), (3, 5), (3, 6), (4, 4), (4, 5), (1, 4), (2, 6)])
@pytest.mark.parametrize("nf", [1, 3])
def test_multigrid_matches_fp64_solver(lib, lo, hi, nf):
    """(1, 4) and (2, 6) are outside the rule and run SSOR."""
    from maple3dmt_gb300.solver import solver_for_survey
    sv = _survey(lo, hi, np.logspace(-1, 2, 3)[:nf])
    out = {}
    for precision in (0, 1):
        s = solver_for_survey(sv, bicgstab_tol=1e-10, bicgstab_maxiter=5000, precision=precision)
        out[precision] = s.forward_batch(sv.freqs, with_fields=True)
        st = s.stats()
        assert all(t <= 1e-8 for t in st["true_residual"][:2 * nf]), st
        s.close()
    for a, b in zip(out[1], out[0]):
        assert rel(a, b) < TOL


@pytest.mark.parametrize("n_rhs", [1, 3, 5, 16])
def test_multigrid_batch_widths(lib, n_rhs):
    """2, 4, 8 and 16 lanes, with sources on identity rows too: each column as
    the FP64 solver gives it alone."""
    from maple3dmt_gb300.solver import solver_for_survey
    sv = _survey(4, 5, (0.5,))
    rng = np.random.default_rng(n_rhs)
    s = solver_for_survey(sv, bicgstab_tol=1e-10, bicgstab_maxiter=5000, precision=1)
    b = rng.normal(size=(n_rhs, s.ne)) + 1j * rng.normal(size=(n_rhs, s.ne))
    s.factorize_frequency(0.5)
    x = s.solve_rhs_batch(b)
    f = solver_for_survey(sv, bicgstab_tol=1e-10, bicgstab_maxiter=5000, precision=0)
    f.factorize_frequency(0.5)
    for k in {0, n_rhs - 1}:
        assert rel(x[k], f.solve_rhs_complex(b[k])) < TOL


def test_multigrid_needs_fewer_iterations(lib):
    """On a grid of 32^3 cells and a level of leaves under it, the multigrid
    preconditioner takes less than half of the SSOR preconditioner's
    iterations (a relaxation factor other than 1 asks for SSOR)."""
    from maple3dmt_gb300 import mesh
    from maple3dmt_gb300.solver import solver_for_survey
    sv = mesh.layered_block_survey(min_level=5, max_level=6, freqs=np.array([0.1, 1.0]))
    it, Z = {}, {}
    for relax in (1.0, 1.0001):
        s = solver_for_survey(sv, bicgstab_tol=1e-9, bicgstab_maxiter=5000, precision=1, ssor_relax=relax)
        Z[relax] = s.forward_batch(sv.freqs)
        it[relax] = s.stats()["total_iterations"]
    assert 2 * it[1.0] < it[1.0001], it
    assert rel(Z[1.0], Z[1.0001]) < TOL


@pytest.mark.parametrize("precision,lo,hi,nf", [(0, 3, 5, 1), (1, 3, 5, 1), (1, 5, 6, 3), (1, 2, 6, 3)])
def test_dependent_launches_give_the_same_bits(lib, precision, lo, hi, nf):
    """Replayed graphs hold plain launches, everything else dependent ones
    that start while their predecessor runs: a value read before it was
    written would change the iteration, so all bits agree, run after run.
    (2, 6) runs SSOR in mixed precision."""
    from maple3dmt_gb300.solver import solver_for_survey
    sv = _survey(lo, hi, np.logspace(-1, 2, 3)[:nf])
    ref = None
    for graphs in (1, 0, 0, 0):
        s = solver_for_survey(sv, bicgstab_tol=1e-10, bicgstab_maxiter=5000, precision=precision, cuda_graphs=graphs)
        got = s.forward_batch(sv.freqs, with_fields=True)
        s.close()
        if ref is None:
            ref = got
        for a, b in zip(got, ref):
            assert np.array_equal(a, b)


def test_solvers_of_different_meshes_at_once(lib):
    """Four handles, four threads: each mesh and batch width launches the same
    kernels with its own amount of shared memory, and each solve gives the
    bits that it gives alone."""
    from concurrent.futures import ThreadPoolExecutor
    from maple3dmt_gb300.solver import solver_for_survey
    freqs = np.logspace(-1, 2, 5)
    surveys = [_survey(*l, freqs[:n]) for l, n in (((3, 5), 1), ((4, 5), 5), ((5, 6), 3), ((2, 4), 4))]
    solvers = [solver_for_survey(sv, bicgstab_tol=1e-8, bicgstab_maxiter=5000, precision=1) for sv in surveys]
    run = lambda k: solvers[k].forward_batch(surveys[k].freqs)
    want = [run(k) for k in range(4)]
    with ThreadPoolExecutor(4) as pool:
        for got in pool.map(lambda k: [run(k) for _ in range(25)] + [k], range(4)):
            for z in got[:-1]:
                assert np.array_equal(z, want[got[-1]])
