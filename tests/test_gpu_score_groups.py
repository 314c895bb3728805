"""Accumulation error of the score's weighted sums by the length of the tensor
core's accumulation groups, against FP64.

Rows sorted by a feature keep the terms of a group alike, so the truncation of
the FP32 accumulation adds up: ~4e-8 of the debiased points per data tile of the
group (four K steps of up to one ulp, half of it on average, on a partial sum
that is half the whole on average, halved again by the shift).  Three tiles,
1.2e-7, are the bound at sizes where a CTA has fewer than 60 tiles."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _sorted_rows(n):
    g = torch.Generator(device="cuda")
    g.manual_seed(1)
    x = torch.randn((n, 16), generator=g, device="cuda")
    return x[torch.argsort(x[:, 0])].contiguous()


@pytest.mark.parametrize("n", [6340, 8454, 9511, 10007, 11021])
def test_debiased_error_of_small_problems(cuda_dev, n):
    from fsk import ops

    x, h, eps = _sorted_rows(n), 1.7, 1e-12
    deb = ops.sdshift16(x, h, eps)
    ops.device_status(cuda_dev)
    q, d = x[:700].double(), x.double()
    dist = torch.zeros((700, n), dtype=torch.float64, device=cuda_dev)
    for k in range(16):
        dist += (q[:, k:k + 1] - d[None, :, k]) ** 2
    phi = torch.exp(-dist / (2.0 * h * h))
    ref = 0.5 * (q + (phi @ d) / (phi.sum(1) + eps)[:, None])
    assert float((deb[:700] - ref).norm() / ref.norm()) <= 1.2e-7
