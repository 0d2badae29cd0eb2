"""Hermitian inner products of interleaved batches at the edges of the launch
rule (one pair a thread, 64 blocks, two pairs a thread, 304 blocks), with odd
remainders of the four running sums, against NumPy's extended precision."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# A result is a sum over chains of at most n K / (304 * 256 * 4) + 3 pairs, 8
# sums within a warp and block and at most 10 + 5 over the blocks: fewer than
# 128 roundings for the sizes here, each of half an ulp of a partial sum.
BOUND = 128 * 2.0 ** -53


@pytest.mark.parametrize("K", [1, 2, 4, 8, 16])
@pytest.mark.parametrize("pairs", [1, 255, 257, 63 * 256, 64 * 256 + 1, 128 * 256 + 1, 304 * 512, 304 * 512 + 1,
                                   304 * 256 * 4 + 1, 304 * 256 * 7 + 3])
def test_dot_at_launch_rule_edges(lib, pairs, K):
    import torch
    from maple3dmt_gb300 import mesh
    from maple3dmt_gb300.solver import solver_for_survey
    n = max(1, -(-pairs // K))
    s = solver_for_survey(mesh.small_survey(min_level=2, max_level=2, freqs=(1.0,)))
    rng = np.random.default_rng(n + K)
    x, y = (rng.normal(size=(n, K, 2)) for _ in range(2))
    dx, dy = (torch.from_numpy(a).cuda() for a in (x, y))
    out = torch.full((K, 2), float("nan"), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    s.dot_batched(dx.data_ptr(), dy.data_ptr(), n, K, out.data_ptr())
    torch.cuda.synchronize()
    a, b = x.astype(np.longdouble), y.astype(np.longdouble)
    want = np.stack([(a * b).sum((0, 2)), (a[:, :, 0] * b[:, :, 1] - a[:, :, 1] * b[:, :, 0]).sum(0)], 1)
    scale = (np.abs(a).sum(2) * np.abs(b).sum(2)).sum(0)
    assert (np.abs(out.cpu().numpy() - want) <= BOUND * scale[:, None]).all()
