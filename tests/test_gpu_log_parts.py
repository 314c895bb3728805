"""Exact log-densities over lists of every length: the data is split into more
parts the shorter the list, in partial rows as long as the list.

Tolerance: the bar of the exact log-density tests, 1e-5 + 2e-6 |log p|."""
import math

import pytest
import torch

from test_gpu_work_split import _rows

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 33, 5000, 70001])
@pytest.mark.parametrize("m,far", [(1, 1), (64, 64), (65, 65), (1000, 1), (1000, 63), (3000, 200), (200, 200)])
def test_list_lengths(cuda_dev, n, m, far):
    from fsk import ops

    x, q, h = _rows(n, 1), _rows(m, 2), 0.9
    q[torch.arange(far, device=q.device) * (m // far)] += 60.0
    got = ops.kde16_sum(q, x, h, log_exact=True, out_scale=0.5)
    again = ops.kde16_sum(q, x, h, log_exact=True, out_scale=0.5)
    ops.device_status(cuda_dev)
    assert torch.equal(got, again)
    xd = x.double()
    for i in range(0, m, 200):
        d2 = ((q[i:i + 200].double()[:, None] - xd[None]) ** 2).sum(-1)
        ref = torch.logsumexp(d2 * (-0.5 / (h * h)), 1) + math.log(0.5)
        assert ((got[i:i + 200] - ref).abs() <= 1e-5 + 2e-6 * ref.abs()).all()
