"""Any-d KDE and its row reduction at the sizes where the split of the data and
the reduction's threads per row change, against FP64 (tolerance of the any-d
tests: FP32 differences and exp2, 1e-5 relative)."""
import time

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [16, 17, 31, 32, 33, 64])
@pytest.mark.parametrize("n,m", [(127, 1), (3000, 129), (20000, 5000), (700, 65536), (700, 65535), (5000, 20000)])
def test_splits_and_rows(cuda_dev, d, n, m):
    from fsk import ops

    g = torch.Generator(device=cuda_dev)
    g.manual_seed(d)
    x = torch.randn((n, d), generator=g, device=cuda_dev)
    q = torch.randn((m, d), generator=g, device=cuda_dev)
    h = 0.5 * d ** 0.5
    got = ops.kde_nd_sum(q, x, h)
    ops.device_status(cuda_dev)
    sel = torch.cat([torch.arange(0, min(m, 40)), torch.arange(max(0, m - 40), m)]).to(cuda_dev)
    dist = ((q[sel, None, :].double() - x[None, :, :].double()) ** 2).sum(2) if n <= 5000 else torch.stack(
        [((v - x.double()) ** 2).sum(1) for v in q[sel].double()])
    ref = torch.exp(-dist / (2 * h * h)).sum(1)
    assert ((got[sel] - ref).abs() <= 1e-5 * ref).all()


def test_host_time_of_the_split():
    """The split of one block of rows over many points is chosen among a few
    candidates, not every count (1824 of them took 21 us, three times a call)."""
    from fsk import _build, _lib

    _build.build()
    lib = _lib.load()
    best = 1.0
    for _ in range(20):
        t = time.perf_counter()
        for _ in range(200):
            lib.fsk_kde_nd_workspace_bytes(200, 400000, 32, 0)
        best = min(best, (time.perf_counter() - t) / 200)
    assert best < 8e-6
