"""Work split and operand preparation of the tensor-core kernels at the sizes
and scales where they can go wrong, against FP64 sums formed on the GPU.

Tolerances are the bars of the KDE and score tests: densities 1e-5 relative,
pdf and weighted sums 2e-6 (weighted sums relative to their own scale)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _phi64(q, x, h):
    q, x = q.double(), x.double()
    mu = x.mean(0)
    q, x = q - mu, x - mu
    d2 = ((q * q).sum(1)[:, None] + (x * x).sum(1)[None, :] - 2.0 * (q @ x.T)).clamp_min(0.0)
    return (d2 * (-0.5 / (h * h))).exp()


def _rows(n, seed, scale=1.0, dev="cuda"):
    g = torch.Generator(device=dev)
    g.manual_seed(seed)
    return torch.randn((n, 16), generator=g, device=dev) * scale


# (m, n): one tile in all; fewer tiles than SMs; a line of fewer tiles than
# CTAs; whole blocks with and without a rest; long lines with ragged ends
@pytest.mark.parametrize("m,n", [(1, 1), (1, 40000), (257, 129), (38912, 100), (38913, 100), (39169, 300),
                                 (77825, 129), (5000, 20001), (40000, 1000)])
def test_kde_work_line(cuda_dev, m, n):
    from fsk import ops

    x, q, h = _rows(n, 1), _rows(m, 2), 0.9
    got = ops.kde16_sum(q, x, h)
    log = ops.kde16_sum(q, x, h, log_exact=True)
    atomic = ops.kde16_sum(q, x, h, atomic=True)
    ops.device_status(cuda_dev)
    for i in range(0, m, 8192):
        ref = _phi64(q[i:i + 8192], x, h).sum(1)
        assert ((got[i:i + 8192] - ref).abs() <= 1e-5 * ref).all()
        assert ((atomic[i:i + 8192] - ref).abs() <= 1e-5 * ref).all()
        assert ((log[i:i + 8192] - ref.log()).abs() <= 1e-5 + 1e-6 * ref.log().abs()).all()


@pytest.mark.parametrize("n", [1, 65, 256, 257, 2047, 10007, 38912, 38913, 40001])
def test_score_work_line_and_shift(cuda_dev, n):
    from fsk import ops

    x, h, eps = _rows(n, 3), 0.9, 1e-12
    pdf, w = ops.empscore16(x, h)
    deb, pdf2, w2, score = ops.sdshift16(x, h, eps, feature_major=True, return_debug=True)
    only = ops.sdshift16(x, h, eps)
    ops.device_status(cuda_dev)
    assert torch.equal(pdf, pdf2) and torch.equal(w, w2) and torch.equal(deb, only)
    for i in range(0, n, 4096):
        phi = _phi64(x[i:i + 4096], x, h)
        p64 = phi.sum(1)
        w64 = phi @ x.double()
        m64 = w64 / (p64 + eps)[:, None]
        d64 = 0.5 * (x[i:i + 4096].double() + m64)
        assert ((pdf[i:i + 4096] - p64).abs() <= 2e-6 * p64).all()
        assert ((w[i:i + 4096] - w64).abs() <= 2e-6 * (w64.abs() + p64[:, None])).all()
        assert ((deb[i:i + 4096] - d64).abs() <= 2e-6 * (d64.abs() + 1.0)).all()
        s64 = (m64 - x[i:i + 4096].double()) / (h * h)
        assert ((score[i:i + 4096] - s64).abs() <= 4e-6 * (s64.abs() + 1.0) / (h * h)).all()


@pytest.mark.parametrize("scale", [1e-15, 1e-4, 3.0, 4097.0, 1e9])
@pytest.mark.parametrize("spread", [1.0, 30.0])
def test_operand_scales(cuda_dev, scale, spread):
    """The power-of-two operand scales over units of measure and query spreads."""
    from fsk import ops

    h = 0.8 * scale * spread
    x, q = _rows(700, 5, scale), _rows(300, 6, scale * spread)
    ref = _phi64(q, x, h).sum(1)
    got = ops.kde16_sum(q, x, h)
    ops.device_status(cuda_dev)
    assert ((got - ref).abs() <= 1e-5 * ref).all()


def test_constant_points_and_unaligned_rows(cuda_dev):
    from fsk import ops

    one = torch.full((300, 16), 2.5, device=cuda_dev)
    assert torch.equal(ops.kde16_sum(one, one, 0.5), torch.full((300,), 300.0, device=cuda_dev))
    assert torch.equal(ops.sdshift16(one, 0.5, 0.0), one)
    # rows that start 4 bytes past a 16-byte boundary
    flat = torch.empty(1000 * 16 + 1, device=cuda_dev)
    x = flat[1:].view(1000, 16)
    x.copy_(_rows(1000, 7))
    assert x.data_ptr() % 16 == 4
    y = x.clone()
    assert torch.equal(ops.kde16_sum(x, x, 0.7), ops.kde16_sum(y, y, 0.7))
    for a, b in zip(ops.empscore16(x, 0.7), ops.empscore16(y, 0.7)):
        assert torch.equal(a, b)
