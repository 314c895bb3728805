"""Silverman bandwidth over column counts, row counts around the blocks' shares,
ties and extreme values, against the FP64 statistics (1e-12, the bar of the
existing test)."""
import numpy as np
import pytest
import torch

from oracle import fp64

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [1, 2, 3, 16, 17, 48, 64])
@pytest.mark.parametrize("n", [1, 2, 3, 5, 63, 65, 4099, 70001])
def test_silverman_matches_fp64(cuda_dev, n, d):
    from fsk import ops

    rng = np.random.default_rng(100 * d + n)
    x = rng.standard_normal((n, d)) * 10.0 ** rng.uniform(-3, 3, d) + 10.0 ** rng.uniform(-2, 2, d)
    x[:, 0] = np.round(x[:, 0])                     # ties
    if d > 2:
        x[:, 1] = rng.choice([-1e30, 0.0, 1e-30, 1e30], n)
    x = x.astype(np.float32)
    got = float(ops.silverman(torch.from_numpy(x).to(cuda_dev)))
    ops.device_status(cuda_dev)
    assert got == pytest.approx(fp64.silverman_nd(x), rel=1e-12)
    if d == 1:
        got = float(ops.silverman(torch.from_numpy(x).to(cuda_dev), rule="sdkde_1d"))
        assert got == pytest.approx(fp64.sdkde_1d(x[:, 0]), rel=1e-12)
