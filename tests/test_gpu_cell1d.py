"""1-D KDE by cell expansions (many points at many queries) against FP64 and
against the pair kernel, which the same queries reach in chunks below the
dispatch size.

Tolerance: 5e-7 relative down to 1e-30 of the peak density (exp2f 2 ulp,
moments and Horner a few roundings); the pair kernel's own exponent rounding
reaches 5e-6 there, so the two are compared at 1e-5."""
import pytest
import torch

pytestmark = pytest.mark.gpu
PAIRS = 1 << 30   # the expansions apply from here (and from 4096 points)


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _points(kind, n):
    g = _gen(11)
    x = torch.randn(n, generator=g, device="cuda")
    if kind == "mixture":
        x = torch.where(torch.rand(n, generator=g, device="cuda") < 0.4, x * 0.3 + 3.0, x - 1.0)
    elif kind == "offset":
        x = x * 0.7 + 100.0
    elif kind == "constant":
        x = torch.full_like(x, -2.75)
    elif kind == "outlier":
        x[n // 2] = 1e6
    elif kind == "uniform":
        x = torch.rand(n, generator=g, device="cuda") * 40.0
    return x


def _direct(q, x, h, **kw):
    from fsk import ops

    step = max(1, (PAIRS - 1) // x.numel())
    return torch.cat([ops.kde1d_sum(q[i:i + step], x, h, **kw) for i in range(0, q.numel(), step)])


@pytest.mark.parametrize("kind", ["normal", "mixture", "offset", "constant", "outlier", "uniform"])
@pytest.mark.parametrize("n,m", [(4096, 262144), (65537, 16411), (1 << 20, 1025)])
def test_cells_match_fp64_and_pairs(cuda_dev, kind, n, m):
    from fsk import ops

    assert n * m >= PAIRS
    x = _points(kind, n)
    h = {"constant": 0.5}.get(kind, 0.9 * float(torch.quantile((x[:4096] - x[:4096].median()).abs(), 0.6)) * n ** -0.2)
    centre = float(x.median())
    g = _gen(5)
    q = centre + torch.randn(m, generator=g, device="cuda") * 2.0
    q[: m // 8] = torch.linspace(float(x.min().clamp_min(-60.0)) - 10 * h, float(x.max().clamp_max(160.0)) + 10 * h,
                                 m // 8, device="cuda")
    got = ops.kde1d_sum(q, x, h)
    atomic = ops.kde1d_sum(q, x, h, atomic=True)
    again = ops.kde1d_sum(q, x, h)
    ops.device_status(cuda_dev)
    assert torch.equal(got, again)
    sel = torch.cat([torch.arange(0, m, max(1, m // 300)), torch.arange(0, 40), torch.arange(m // 8 - 40, m // 8)])
    sel = sel.to(q.device)
    ref = torch.stack([torch.exp(-0.5 * ((x.double() - v) / h) ** 2).sum() for v in q[sel].double()])
    ok = ref > 1e-30 * ref.max()
    tol = 1e-5 if kind == "outlier" else 5e-7    # the outlier's extent leaves the pair kernel in charge
    for out in (got, atomic):
        assert ((out[sel] - ref).abs() <= tol * ref)[ok].all(), float(((out[sel] - ref).abs() / ref)[ok].max())
    pairs = _direct(q, x, h)
    big = pairs > 1e-20
    assert ((got - pairs).abs() <= 1e-5 * pairs)[big].all()
    logs = ops.kde1d_sum(q, x, h, out_scale=0.25 / n, log_eps=1e-12)
    want = torch.log(got.double() * (0.25 / n) + 1e-12)
    assert ((logs - want).abs() <= 1e-6 * (1.0 + want.abs())).all()


def test_non_finite_inputs_as_the_pair_kernel(cuda_dev):
    from fsk import ops

    x = _points("normal", 1 << 18)
    q = torch.linspace(-3, 3, 5000, device="cuda")
    q[7], q[8], q[9] = float("inf"), float("-inf"), float("nan")
    got, pairs = ops.kde1d_sum(q, x, 0.1), _direct(q, x, 0.1)
    assert torch.equal(torch.isnan(got), torch.isnan(pairs)) and float(got[7]) == float(got[8]) == 0.0
    for bad in (float("inf"), float("nan")):
        x[3] = bad
        got, pairs = ops.kde1d_sum(q, x, 0.1), _direct(q, x, 0.1)
        assert torch.equal(torch.isnan(got), torch.isnan(pairs))
        fine = ~torch.isnan(pairs)
        assert torch.allclose(got[fine], pairs[fine], rtol=1e-6, atol=0.0)
    ops.device_status(cuda_dev)
