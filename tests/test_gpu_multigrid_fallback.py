"""From the multigrid preconditioner to SSOR: with the coarse grids' cell sizes
scaled, their corrections spoil the multigrid steps of every right-hand side, and
each goes on with SSOR."""
import numpy as np
import pytest

from conftest import rel

pytestmark = pytest.mark.gpu

CONVERGED, MAXITER = 1, 3
FREQS = np.array([0.1, 1.0, 10.0])


def _solver(**par):
    from maple3dmt_gb300 import mesh
    from maple3dmt_gb300.solver import solver_for_survey
    sv = mesh.small_survey(min_level=4, max_level=5, freqs=FREQS)
    return solver_for_survey(sv, **(dict(bicgstab_tol=1e-10, bicgstab_maxiter=5000, precision=1) | par))


@pytest.mark.parametrize("scale", [1 / 32, 0.25, 32.0])
@pytest.mark.parametrize("opts", [dict(), dict(cuda_graphs=1), dict(residual_replacement=1)])
def test_every_lane_falls_back(lib, scale, opts):
    """All six right-hand sides converge, to the impedances of the sound
    preconditioner within the oracle comparisons' 1e-6 (two 1e-10 solves), and the
    residual reported is that of the returned solution.  With the cell sizes
    restored (powers of two, exactly) the handle gives its first bits again."""
    s = _solver(**opts)
    want = s.forward_batch(FREQS)
    s.test_set_multigrid_scale(scale)
    got = s.forward_batch(FREQS)
    st = s.stats()
    assert st["status"][:6] == [CONVERGED] * 6, st
    assert all(t <= 1e-10 for t in st["true_residual"][:6]), st
    assert rel(got, want) < 1e-6
    s.test_set_multigrid_scale(1.0 / scale)
    assert np.array_equal(s.forward_batch(FREQS), want)


def test_last_refinement_step(lib):
    """max_refinements = 0: two correction steps of a relative 3e-5 in FP32, then
    as many with SSOR.  Every right-hand side ends with one of the two statuses, in
    accord with its residual."""
    s = _solver(max_refinements=0)
    s.test_set_multigrid_scale(1 / 32)
    s.forward_batch(FREQS)
    st = s.stats()
    for status, res in zip(st["status"][:6], st["true_residual"][:6]):
        assert status == (CONVERGED if res <= 1e-10 else MAXITER), st
        assert res < 1e-4, st


def test_iteration_cap_with_a_spoiled_preconditioner(lib):
    """Seven iterations: no right-hand side runs more, and each reports the cap."""
    s = _solver(bicgstab_maxiter=7)
    s.test_set_multigrid_scale(1 / 32)
    s.forward_batch(FREQS)
    st = s.stats()
    assert st["status"][:6] == [MAXITER] * 6, st
    assert all(1 <= it <= 7 for it in st["iterations"][:6]), st


def test_one_column_alone_and_among_others(lib):
    """A right-hand side's fallback does not depend on its place in the batch."""
    s = _solver()
    s.factorize_frequency(1.0)
    rng = np.random.default_rng(1)
    b = rng.normal(size=(5, s.ne)) + 1j * rng.normal(size=(5, s.ne))
    want = s.solve_rhs_batch(b)
    s.test_set_multigrid_scale(1 / 32)
    got = s.solve_rhs_batch(b)
    alone = [s.solve_rhs_complex(b[k]) for k in (0, 4)]
    assert s.stats()["status"][0] == CONVERGED
    for k in range(5):
        assert rel(got[k], want[k]) < 1e-6
    assert rel(alone[0], want[0]) < 1e-6 and rel(alone[1], want[4]) < 1e-6


@pytest.mark.parametrize("model", ["sea", "salt", "sheet", "random", "conductive"])
def test_strong_contrasts(lib, model):
    """Sea water over a resistive basement, a resistive body in a conductive
    earth, a conductive sheet in a resistive one, three decades from cell to cell,
    sea water throughout: impedances of the mixed and of the FP64 solve.  At a
    residual of 1e-9 either's error is up to 6e-5 (sheet); it goes with the
    residual, so 1e-12 leaves 1e-7 and a factor of ten."""
    from maple3dmt_gb300 import mesh
    from maple3dmt_gb300.solver import solver_for_survey
    freqs = np.array([0.01, 1.0, 100.0])
    sv = mesh.layered_block_survey(min_level=4, max_level=5, n_side=5, freqs=freqs)
    x, y, z = sv.leaves.cx, sv.leaves.cy, sv.leaves.cz
    earth = {"sea": np.where(z > -2000, 3.3, np.where(z > -30000, 1e-3, 0.1)),
             "salt": np.where((abs(x) < 5000) & (abs(y) < 5000) & (z > -6000) & (z < -1000), 1e-6, 1.0),
             "sheet": np.where((z < -3000) & (z > -4500), 100.0, 1e-4),
             "random": 10.0 ** np.random.default_rng(3).normal(-2, 1.0, len(x)),
             "conductive": np.full_like(x, 3.3)}[model]
    sigma = np.where(sv.leaves.cell_type == 0, earth, sv.sigma)
    Z = []
    for precision in (0, 1):
        s = solver_for_survey(sv, bicgstab_tol=1e-12, bicgstab_maxiter=20000, precision=precision)
        s.set_sigma(sigma)
        Z.append(s.forward_batch(freqs))
        st = s.stats()
        assert st["status"][:6] == [CONVERGED] * 6, st
        s.close()
    for f in range(3):
        assert rel(Z[1][f], Z[0][f]) < 1e-6


def test_setup_without_memory_for_the_grids(lib):
    """Set-up succeeds, solves run SSOR: more iterations, the same impedances, no
    multigrid to scale; set up again with memory, the handle has it."""
    from maple3dmt_gb300 import mesh
    from maple3dmt_gb300.solver import ForwardSolverFV, SolverError, solver_for_survey
    sv = mesh.small_survey(min_level=4, max_level=5, freqs=FREQS)
    par = dict(bicgstab_tol=1e-10, bicgstab_maxiter=5000, precision=1)
    m = solver_for_survey(sv, **par)
    want = m.forward_batch(FREQS)
    s = ForwardSolverFV(0)
    for fail in (True, False):
        s.test_fail_multigrid_alloc(fail)
        s.setup(sv.leaves, sigma_bg=sv.sigma_bg, **par)
        s.set_sigma(sv.sigma)
        s.set_stations(sv.stations)
        got = s.forward_batch(FREQS)
        st = s.stats()
        assert st["status"][:6] == [CONVERGED] * 6
        if fail:
            assert rel(got, want) < 1e-6
            assert sum(st["iterations"][:6]) > 1.5 * sum(m.stats()["iterations"][:6])
            with pytest.raises(SolverError):
                s.test_set_multigrid_scale(1.0)
        else:
            assert np.array_equal(got, want)
