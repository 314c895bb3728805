"""Values at the ends of the FP32 range in the tensor-core paths."""
import pytest
import torch

pytestmark = pytest.mark.gpu
FLT_MAX = 3.4028234663852886e38


def _rows(n, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return torch.randn((n, 16), generator=g, device="cuda")


@pytest.mark.parametrize("value", [-FLT_MAX, FLT_MAX, 1e36, -3.3e33])
@pytest.mark.parametrize("n,m", [(3, 5), (300, 257), (5000, 700), (70001, 300)])
def test_constant_column_of_large_values(cuda_dev, value, n, m):
    """A column with the same value in every row (a mask of the type's lowest
    value, say) adds nothing to any distance: the sums are those with the column
    at 0, whose centred operands are the same bits."""
    from fsk import ops

    x, q, h = _rows(n, 1), _rows(m, 2), 0.9
    x[:, 5] = q[:, 5] = 0.0
    want = ops.kde16_sum(q, x, h)
    pdf, w = ops.empscore16(x, h)
    deb = ops.sdshift16(x, h, 1e-12)
    x[:, 5] = q[:, 5] = value
    assert torch.equal(ops.kde16_sum(q, x, h), want)
    pdf2, w2 = ops.empscore16(x, h)
    deb2 = ops.sdshift16(x, h, 1e-12)
    ops.device_status(cuda_dev)
    rest = [k for k in range(16) if k != 5]
    assert torch.equal(pdf2, pdf)
    assert torch.equal(w2[:, rest], w[:, rest]) and torch.equal(deb2[:, rest], deb[:, rest])
