"""Score sums of rows with one close neighbour, which the kernel recomputes.

pdf = 1 + phi.  phi from FP32 differences: ex2 to 2^-22.5, the squared distance to
4 x 2^-24 times |ln phi| <= 2, both times phi / (1 + phi) <= 1/2, and the final
rounding 2^-24: below 2^-22 together."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 64, 4096, 20000])
def test_isolated_pairs(cuda_dev, n):
    from fsk import ops

    g = torch.Generator(device=cuda_dev)
    g.manual_seed(n)
    h = 0.7
    a = torch.randn((n // 2, 16), generator=g, device=cuda_dev) * 40.0
    u = torch.randn((n // 2, 16), generator=g, device=cuda_dev)
    length = 0.3 + 1.6 * torch.rand((n // 2, 1), generator=g, device=cuda_dev)
    x = torch.stack([a, a + u * (length * h / u.norm(dim=1, keepdim=True))], 1).view(n, 16)
    x = x[torch.randperm(n, generator=g, device=cuda_dev)].contiguous()
    pdf, w = ops.empscore16(x, h)
    ops.device_status(cuda_dev)
    worst = 0.0
    for i in range(0, n, 256):
        d = torch.zeros((min(256, n - i), n), dtype=torch.float64, device=cuda_dev)
        for k in range(16):
            d += (x[i:i + 256, k:k + 1].double() - x[None, :, k].double()) ** 2
        ref = torch.exp(-d / (2 * h * h)).sum(1)
        worst = max(worst, float(((pdf[i:i + 256] - ref).abs() / ref).max()))
    assert worst <= 2.0 ** -22, worst
