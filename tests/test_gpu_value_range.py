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


@pytest.mark.parametrize("eps", [1e29, 1e31, 1e38, 1e39, 1e300, float("inf")])
def test_shift_with_a_large_eps(cuda_dev, eps):
    """W / (pdf + eps) vanishes: half of each point, and the score -x / h^2."""
    from fsk import ops

    x, h = _rows(700, 3), 0.8
    deb, pdf, w, score = ops.sdshift16(x, h, eps, return_debug=True)
    one_call = ops.sdkde16(x, x[:100], h, eps=eps, return_debiased=True)[1]
    ops.device_status(cuda_dev)
    assert torch.equal(deb, 0.5 * x) and torch.equal(one_call, 0.5 * x)
    want = -x.double() / (h * h)
    assert ((score - want).abs() <= 2.0 ** -24 * want.abs()).all()
    plain = ops.empscore16(x, h)
    assert torch.equal(pdf, plain[0]) and torch.equal(w, plain[1])


def test_weighted_sums_past_the_largest_float(cuda_dev):
    """300 points at 1e37: their weighted sum 3e39 is infinite in FP32 and their
    mean is not.  Sums within the 2e-6 of the score tests."""
    from fsk import ops

    x = torch.full((300, 16), 1e37, device=cuda_dev)
    x[:, 3] = 2.0
    deb, pdf, w, score = ops.sdshift16(x, 0.5, 0.0, return_debug=True)
    ops.device_status(cuda_dev)
    assert torch.equal(deb, x) and (score == 0).all()
    assert ((pdf - 300).abs() <= 2e-6 * 300).all() and ((w[:, 3] - 600).abs() <= 2e-6 * 600).all()
    assert torch.isposinf(w[:, 0]).all()


@pytest.mark.parametrize("value", [-FLT_MAX, 3e38, 1e38, -1e36])
@pytest.mark.parametrize("h", [1e-3, 0.9, 500.0])
def test_shift_of_points_near_the_largest_float(cuda_dev, value, h):
    """A constant column stays where it is, with few neighbours (the weighted sum is
    the point itself) and with many."""
    from fsk import ops

    x = _rows(300, 4)
    x[:, 9] = value
    deb = ops.sdshift16(x, h, 0.0)
    deb2, _, _, score = ops.sdshift16(x, h, 1e-12, return_debug=True)
    ops.device_status(cuda_dev)
    assert torch.equal(deb[:, 9], x[:, 9]) and torch.equal(deb2[:, 9], x[:, 9])
    assert torch.isfinite(deb).all() and torch.isfinite(score).all()
