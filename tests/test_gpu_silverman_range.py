"""Silverman bandwidth on data with NaNs and on more than 2^32 rows."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _expected(x):
    """0.9 mean(min(std, IQR / 1.34)) n^(-1/(d+4)) in FP64; a NaN sorts last, a
    column's smaller value is the one that is not NaN, and 0 is replaced by 1."""
    n, d = x.shape
    s = torch.sort(x, 0).values.double()

    def quantile(p):
        v = p * (n - 1)
        i = int(math.floor(v))
        a, b = s[i], s[min(i + 1, n - 1)]
        return torch.lerp(a, b, v - i)

    iqr = (quantile(0.75) - quantile(0.25)) / 1.34
    sigma = float(torch.fmin(x.double().std(0, correction=0), iqr).mean())
    return 0.9 * (1.0 if sigma <= 0 else sigma) * n ** (-1.0 / (d + 4))


@pytest.mark.parametrize("n,d", [(1, 1), (2, 1), (5, 1), (255, 1), (4099, 3), (300, 16), (1000, 49)])
@pytest.mark.parametrize("share", [0.0, 0.1, 0.3, 1.0])
def test_nan_values(cuda_dev, n, d, share):
    from fsk import ops

    g = torch.Generator(device=cuda_dev)
    g.manual_seed(n + d)
    x = torch.randn((n, d), generator=g, device=cuda_dev)
    x[: max(1, int(share * n)), 0] = float("nan")
    got, want = float(ops.silverman(x)), _expected(x)
    ops.device_status(cuda_dev)
    assert math.isnan(got) == math.isnan(want), (got, want)
    assert math.isnan(want) or abs(got - want) <= 1e-12 * abs(want), (got, want)


def test_more_than_2p32_rows(cuda_dev):
    """Ranks beyond 32 bits: 6e9 rows, 5860000 copies of the values v |v|, v = -512
    .. 511.  std 512^2 / sqrt 5 is above IQR / 1.34, so the quartiles decide."""
    from fsk import ops

    copies = 5_860_000
    v = torch.arange(-512, 512, device=cuda_dev, dtype=torch.float32)
    v = v * v.abs()
    x = v.repeat(copies).view(-1, 1)
    n = x.shape[0]
    assert 0.75 * (n - 1) > 1 << 32
    got = float(ops.silverman(x))
    ops.device_status(cuda_dev)
    del x
    w = v.double()
    q25 = float(torch.lerp(w[255], w[256], 0.75))   # 0.25 (n - 1) = 256 copies - 0.25
    q75 = float(torch.lerp(w[767], w[768], 0.25))
    want = 0.9 * (q75 - q25) / 1.34 * n ** -0.2
    assert abs(got - want) <= 1e-12 * want
