"""The grid reductions of the FP32 kernels against exact sums: no less precise
than FP64 accumulation, over the whole FP32 range of the terms, and with its
results beyond it."""
import ctypes as C
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _sum(lib, v, many):
    n, K = v.shape[:2]
    v = np.ascontiguousarray(v, np.float32)
    out = np.full((K, 2), np.nan)
    rc = lib.m3d_test_sum_f32(v.ctypes.data_as(C.POINTER(C.c_float)), n, K, many,
                              out.ctypes.data_as(C.POINTER(C.c_double)))
    assert rc == 0
    return out


def _cases(rng, n, K):
    shape = (n, K, 2)
    yield "ordinary", rng.normal(size=shape)
    yield "squares", rng.normal(size=shape) ** 2
    yield "wide", rng.normal(size=shape) * 2.0 ** rng.integers(-140, 100, shape)
    c = (rng.normal(size=shape) * 2.0 ** rng.integers(-40, 40, shape)).astype(np.float32)
    c[n // 2:2 * (n // 2)] = -c[:n // 2] * np.float32(1 + 2.0 ** -22)
    yield "cancelling", rng.permutation(c)
    yield "tiny", rng.integers(-9, 9, shape) * 2.0 ** -149


@pytest.mark.parametrize("K", [2, 4, 8, 16])
@pytest.mark.parametrize("n", [1, 7, 513, 19001])
@pytest.mark.parametrize("many", [0, 1])
def test_against_exact_sums(lib, n, K, many):
    """Three floats: the last conversion's half ulp, and less than 2^-58 of the sum
    of the moduli (each step's error is below 2^-71 of a partial sum, and no
    chain is longer than 8192); FP64 alone would allow 2^-53 a step."""
    for name, v in _cases(np.random.default_rng(100 * n + K), n, K):
        v = v.astype(np.float32)
        got = _sum(lib, v, many)
        for k in range(K):
            for part in range(2):
                x = v[:, k, part].astype(np.float64).tolist()
                want = math.fsum(x)
                bound = 2.0 ** -53 * abs(want) + 2.0 ** -58 * math.fsum(map(abs, x))
                assert abs(got[k, part] - want) <= bound, (name, k, part)


@pytest.mark.parametrize("K", [2, 16])
@pytest.mark.parametrize("many", [0, 1])
def test_beyond_the_fp32_range(lib, K, many):
    """Sums beyond 3.4e38 as FP64 gives them (128 steps of 2^-53 at most), infinities
    and NaN where FP64 has them, and only there."""
    rng = np.random.default_rng(K)
    n = 5000
    v = (rng.uniform(1.0, 3.0, (n, K, 2)) * 1e38).astype(np.float32)
    v[:, 0, 1] = rng.normal(size=n)
    got = _sum(lib, v, many)
    want = v.astype(np.float64).sum(0)
    scale = np.abs(v.astype(np.float64)).sum(0)
    assert (np.abs(got - want) <= 128 * 2.0 ** -53 * scale).all()
    v = rng.normal(size=(n, K, 2)).astype(np.float32)
    v[17, 0, 0] = np.inf
    v[99, 0, 1] = -np.inf
    v[3, 1, 0], v[4000, 1, 0] = np.inf, -np.inf
    v[2500, 1, 1] = np.nan
    got = _sum(lib, v, many)
    assert got[0, 0] == np.inf and got[0, 1] == -np.inf and np.isnan(got[1]).all()
    if K > 2:
        want = v[:, 2:].astype(np.float64).sum(0)
        assert (np.abs(got[2:] - want) <= 128 * 2.0 ** -53 * np.abs(v[:, 2:].astype(np.float64)).sum(0)).all()
