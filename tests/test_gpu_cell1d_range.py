"""The range of the 1-D cell expansions: queries far outside the data, bandwidths,
scales and sizes at the ends of what the FP32 tables hold, against the pair
kernel (the same queries in chunks below the dispatch size) or the exact value.

Where both sums are formed they are compared at 1e-5, the pair kernel's own
exponent rounding in the far tail."""
import pytest
import torch

pytestmark = pytest.mark.gpu
PAIRS = 1 << 30
FLT_MAX = 3.4028234663852886e38


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _mixture(n, seed):
    g = _gen(seed)
    x = torch.randn(n, generator=g, device="cuda")
    u = torch.rand(n, generator=g, device="cuda")
    return torch.where(u < 0.3, x * 0.3 - 2.0, torch.where(u < 0.7, x * 0.5 + 0.5, x * 0.8 + 3.0))


def _pairs(q, x, h, **kw):
    from fsk import ops

    step = max(1, (PAIRS - 1) // x.numel())
    return torch.cat([ops.kde1d_sum(q[i:i + step], x, h, **kw) for i in range(0, q.numel(), step)])


@pytest.mark.parametrize("seed", range(6))
def test_queries_far_from_the_data(cuda_dev, seed):
    from fsk import ops

    x = _mixture(1 << 20, seed)
    lo, hi = float(x.min()), float(x.max())
    h = 0.9 * float(x.std()) * x.numel() ** -0.2 * (1.0, 0.3, 4.0)[seed % 3]
    steps = torch.tensor([0.0, 15.0, 20.0, 100.0, 1e3, 1e4, 1e5, 1e6, 1e9], dtype=torch.float64)
    ends = torch.tensor([1e4, 1e5, 1e6, 1e9, 1e19, 3e19, 1e20, FLT_MAX, float("inf")], dtype=torch.float64)
    q = torch.cat([hi + steps * h, lo - steps * h, ends, -ends, torch.linspace(lo, hi, 1100).double()])
    q = q.float().to(cuda_dev)
    assert x.numel() * q.numel() >= PAIRS
    forms = [{}, {"atomic": True}, {"log_eps": 1e-12}, {"log_eps": 0.0}, {"out_scale": -2.0}]
    for kw in forms:
        got, want = ops.kde1d_sum(q, x, h, **kw), _pairs(q, x, h, **kw)
        same = got == want   # zeros and infinities of the logarithm
        near = (got - want).abs() <= 1e-5 * (want.abs() + ("log_eps" in kw))
        assert (same | near).all(), (kw, q[~same], got[~same], want[~same])
    ops.device_status(cuda_dev)
    got = ops.kde1d_sum(q, x, h)
    assert (got[1:9] == 0).all() and (got[10:18] == 0).all() and (got[18:36] == 0).all()


@pytest.mark.parametrize("h", [1e-300, 1e-160, 1e-40, 1e-30, 1e-22, 1e-16, 2e-15, 1e-10, 1e10, 9e17, 2e18, 1e20, 1e28, 1e29,
                               1e30, 1e37, 3e38, 1e39, 1e160, 1e300])
@pytest.mark.parametrize("unit", ["one", "h"])
def test_bandwidths_of_any_size(cuda_dev, h, unit):
    """Data of spread 1 and of spread h: finite where the pair kernel is, and equal."""
    from fsk import ops

    s = 1.0 if unit == "one" else min(max(h, 1e-37), 1e37)
    x = (_mixture(1 << 18, 3).double() * s).float()
    q = (torch.linspace(-12, 12, 4200, dtype=torch.float64, device="cuda") * s).float()
    for kw in ({}, {"log_eps": 1e-12}):
        got, want = ops.kde1d_sum(q, x, h, **kw), _pairs(q, x, h, **kw)
        assert torch.equal(got.isnan(), want.isnan())
        ok = (got == want) | ((got - want).abs() <= 1e-5 * (want.abs() + ("log_eps" in kw))) | want.isnan()
        assert ok.all(), (kw, q[~ok], got[~ok], want[~ok])
    ops.device_status(cuda_dev)


def test_densities_past_the_largest_float(cuda_dev):
    """4e8 points at one place times 9e29 is infinite, not NaN; times 8e29 it is 3.2e38."""
    from fsk import ops

    n = 400_000_000
    x = torch.full((n,), 1.5, device=cuda_dev)
    q = torch.tensor([1.5, 1.5, 40.0], device=cuda_dev)
    got = ops.kde1d_sum(q, x, 1.0, out_scale=9e29)
    assert torch.isposinf(got[:2]).all() and float(got[2]) == 0.0
    assert torch.isneginf(ops.kde1d_sum(q, x, 1.0, out_scale=-9e29)[:2]).all()
    fits = ops.kde1d_sum(q, x, 1.0, out_scale=8e29)
    ops.device_status(cuda_dev)
    assert (fits[:2].double() / 3.2e38 - 1).abs().max() <= 5e-7


def test_more_than_2p32_points(cuda_dev):
    """The sum of 2^32 + 2^26 equal points at their place (the 64-bit fixed-point
    moments hold 2^31)."""
    from fsk import ops

    n = (1 << 32) + (1 << 26)
    x = torch.full((n,), 0.5, device=cuda_dev)
    q = torch.tensor([0.5, 1.5], device=cuda_dev)
    got = ops.kde1d_sum(q, x, 1.0).double()
    ops.device_status(cuda_dev)
    want = n * torch.exp(torch.tensor([0.0, -0.5], dtype=torch.float64, device=cuda_dev))
    assert ((got - want).abs() <= 5e-7 * want).all()
