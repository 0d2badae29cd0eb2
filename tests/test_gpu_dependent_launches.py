"""Dependent launches against plain ones: a value read before the kernel that
writes it has ended would change the iteration, so all bits agree."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("opts", [dict(precision=0), dict(precision=0, forward_interleaved=1), dict(precision=1),
                                  dict(precision=1, forward_interleaved=1), dict(precision=1, gradcorr_overlap=0),
                                  dict(precision=1, gradcorr=0, ssor_form=0), dict(precision=1, ssor_relax=1.0001)])
@pytest.mark.parametrize("lo,hi,nf", [(3, 5, 1), (4, 5, 8), (5, 6, 2)])
def test_plain_and_dependent(lib, lo, hi, nf, opts):
    """Fields, impedances and gradients, with the divergence correction's own chain
    of launches: one plain run, then three dependent ones."""
    from maple3dmt_gb300 import mesh, workloads
    from maple3dmt_gb300.solver import solver_for_survey
    freqs = np.logspace(-1, 2, 8)[:nf]
    sv = mesh.small_survey(min_level=lo, max_level=hi, freqs=freqs)
    s = solver_for_survey(sv, bicgstab_tol=1e-8, bicgstab_maxiter=3000, **opts)
    obs, err = workloads.halfspace_data(sv.stations, freqs, seed=1)
    ref = None
    for plain in (True, False, False, False):
        s.test_set_plain_launches(plain)
        got = s.forward_batch(freqs, with_fields=True) + s.gradient_batch(freqs, obs, err)
        if ref is None:
            ref = got
        for a, b in zip(got, ref):
            assert np.array_equal(a, b)
    assert s.stats()["divcorr_calls"] > 0
