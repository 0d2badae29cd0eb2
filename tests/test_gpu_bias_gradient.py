"""The bias gradient of the output layer is the sum of the BF16 output gradients:
as precise as FP64 accumulation, rounded to FP32 once."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grid", [(1, 1, 8, 16), (2, 5, 8, 32), (4, 32, 32, 32)])
@pytest.mark.parametrize("kind", ["ordinary", "cancelling", "beyond"])
def test_output_bias_gradient(lib, grid, kind):
    """Half an ulp of FP32, and 2^-45 of the moduli for the FP64 sums over threads and
    splits (fewer than 256 steps).  `beyond`: partial sums leave the FP32 range."""
    import torch
    from maple3dmt_gb300.learned import Cnn
    rng = np.random.default_rng(len(kind))
    dy = rng.normal(size=grid + (6,))
    if kind == "cancelling":
        half = dy.reshape(2, -1)
        half[1] = -half[0] * (1 + 2.0 ** -7 * rng.integers(0, 2, half[0].shape))
        dy = dy * 2.0 ** rng.integers(-30, 30, 6)
    if kind == "beyond":
        dy = np.where(np.arange(dy.size).reshape(dy.shape) // 6 % 2 == 0, 2e38, -2e38) * (1 + 0.25 * np.abs(np.sin(dy)))
        dy.reshape(-1, 6)[:4] = np.abs(dy.reshape(-1, 6)[:4])
    dy = dy.astype(np.float32)
    net = Cnn(layers=2, c_in=8, hidden=32, c_out=6)
    _, db, _ = net.backward(rng.normal(size=grid + (8,)).astype(np.float32), dy)
    x = torch.from_numpy(dy).bfloat16().double().numpy().reshape(-1, 6)
    for c in range(6):
        want, mod = math.fsum(x[:, c].tolist()), math.fsum(np.abs(x[:, c]).tolist())
        if abs(want) > 3.4028235e38:
            assert db[1, c] == math.copysign(math.inf, want)
        else:
            assert abs(float(db[1, c]) - want) <= 2.0 ** -24 * abs(want) + 2.0 ** -45 * mod, (c, db[1, c], want)
