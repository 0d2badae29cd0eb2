"""Every row that a solve carries is its own: the memory of a narrow batch holds
what wider batches left on the rows that the batch does not write (identity rows
in the mixed-precision solve), and rows that pad the sweeps must be swept too."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("opts", [dict(), dict(gradcorr=0), dict(gradcorr=0, ssor_form=0),
                                  dict(gradcorr=0, row_kernels=0), dict(gradcorr=0, coop_sweep=1, ssor_form=0),
                                  dict(gradcorr=0, sweep_rows=16384), dict(ssor_relax=1.0001),
                                  dict(gradcorr=0, residual_replacement=1, ssor_form=0), dict(krylov=1),
                                  dict(precision=0), dict(precision=0, row_kernels=0)])
def test_narrow_batch_after_a_wide_one(lib, opts):
    """Eight frequencies (16 lanes, narrowing as they converge), then one, on one
    handle: the bits and the iterations of a fresh handle."""
    from maple3dmt_gb300 import mesh
    from maple3dmt_gb300.solver import solver_for_survey
    freqs = np.logspace(-1, 3, 8)
    sv = mesh.small_survey(min_level=4, max_level=5, freqs=freqs)
    par = dict(bicgstab_tol=1e-10, bicgstab_maxiter=5000, precision=1) | opts
    used = solver_for_survey(sv, **par)
    used.forward_batch(freqs)
    for f in (freqs[1], freqs[6]):
        fresh = solver_for_survey(sv, **par)
        want = fresh.forward_batch([f], with_fields=True)
        got = used.forward_batch([f], with_fields=True)
        for a, b in zip(got, want):
            assert np.array_equal(a, b)
        a, b = used.stats(), fresh.stats()
        assert a["iterations"][:2] == b["iterations"][:2] and a["status"][:2] == [1, 1]
        fresh.close()


@pytest.mark.parametrize("opts", [dict(), dict(ssor_form=0), dict(row_kernels=0), dict(coop_sweep=1, ssor_form=0),
                                  dict(ssor_relax=1.0001), dict(krylov=1), dict(precision=0),
                                  dict(precision=0, row_kernels=0)])
def test_solve_after_a_failed_one(lib, opts):
    """A conductivity beyond the FP32 range and a right-hand side whose square
    overflows in FP64 leave infinities and NaN in the solver's vectors; the next
    solve (without divergence correction) gives the bits of a fresh handle."""
    from maple3dmt_gb300 import mesh
    from maple3dmt_gb300.solver import solver_for_survey
    freqs = np.logspace(-1, 1, 2)
    sv = mesh.small_survey(min_level=4, max_level=5, freqs=freqs)
    par = dict(bicgstab_tol=1e-10, bicgstab_maxiter=2000, precision=1, div_correction=0) | opts
    fresh = solver_for_survey(sv, **par)
    want = fresh.forward_batch(freqs, with_fields=True)
    s = solver_for_survey(sv, **par)
    s.set_sigma(np.where(sv.leaves.cell_type == 0, 1e40, sv.sigma))
    s.forward_batch(freqs)
    s.set_sigma(sv.sigma)
    s.factorize_frequency(freqs[0])
    rng = np.random.default_rng(2)
    s.solve_rhs_batch(1e200 * (rng.normal(size=(4, s.ne)) + 1j * rng.normal(size=(4, s.ne))))
    got = s.forward_batch(freqs, with_fields=True)
    assert s.stats()["status"][:4] == fresh.stats()["status"][:4]
    for a, b in zip(got, want):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("precision", [0, 1])
def test_copy_wait_timeout_with_reused_stages(lib, precision):
    """On 201 k edges with 16 lanes each block of the product runs its ring of
    stages through more than once.  With the hook on, warps that find a copy not
    landed skip it, in step with the others; the call reports the timeout, and with
    the hook off the handle solves as a fresh one does."""
    from maple3dmt_gb300 import mesh
    from maple3dmt_gb300.solver import SolverError, solver_for_survey
    freqs = np.logspace(0, 2, 8)
    sv = mesh.layered_block_survey(min_level=5, max_level=6, n_side=5, freqs=freqs)
    par = dict(bicgstab_tol=1e-6, bicgstab_maxiter=30, precision=precision)
    s = solver_for_survey(sv, **par)
    s.test_set_consume_no_wait(True)
    with pytest.raises(SolverError) as e:
        s.forward_batch(freqs)
    assert e.value.code == 3 and "timed out" in str(e.value)
    s.test_set_consume_no_wait(False)
    assert np.array_equal(s.forward_batch(freqs), solver_for_survey(sv, **par).forward_batch(freqs))
