"""The captured SD-KDE call's workspace is that of its own output form, at shapes
where the KDE's share of it is the larger one."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,m", [(300, 200), (1984, 23808), (2000, 60000)])
@pytest.mark.parametrize("kw", [{}, {"log_exact": True}, {"log_eps": 1e-9}, {"log_exact": True, "precision": "ieee"}])
def test_every_output_form_is_captured(cuda_dev, n, m, kw):
    from fsk import ops

    g = torch.Generator(device=cuda_dev)
    g.manual_seed(n)
    x = torch.randn((n, 16), generator=g, device=cuda_dev)
    q = torch.randn((m, 16), generator=g, device=cuda_dev) * 1.5
    want = ops.sdkde16(x, q, 0.9, **kw)
    got = ops.SDKDEGraph(x, q, 0.9, **kw).replay()
    ops.device_status(cuda_dev)
    assert torch.equal(got, want)
