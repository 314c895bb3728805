"""Local polynomials of the 1-D cell expansions where they meet the cells that
are visited one by one: gaps, tails, cell edges and single cells, against FP64.

Tolerance 3e-7 relative where the density is above 1e-30 of its peak: a visited
cell carries exp2f (2 ulp) and a few roundings, a polynomial 12 node values to
1e-8 times at most 2 (the change over a cell) and the final rounding (6e-8)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("gap", [0.0, 3.0, 8.0, 25.0])
@pytest.mark.parametrize("n,h", [(4096, 0.5), (4099, 0.11), (70001, 0.05)])
def test_gaps_and_cell_edges(cuda_dev, gap, n, h):
    from fsk import ops

    g = torch.Generator(device="cuda")
    g.manual_seed(3)
    x = torch.rand(n, generator=g, device="cuda") * (4.0 * h)
    x[n // 3:] += (4.0 + gap) * h
    lo, hi = float(x.min()), float(x.max())
    m = (1 << 30) // n + 1
    edges = lo + torch.arange(0, int((hi - lo) / h * 4) + 2, device="cuda") * (0.25 * h)
    q = torch.cat([edges, torch.nextafter(edges, edges + 1), torch.nextafter(edges, edges - 1),
                   torch.linspace(lo - 9 * h, hi + 9 * h, 500, device="cuda")])
    sel = q.numel()
    q = torch.cat([q, lo + (hi - lo) * torch.rand(m - sel, generator=g, device="cuda")])
    got = ops.kde1d_sum(q, x, h)[:sel].double()
    ops.device_status(cuda_dev)
    ref = torch.stack([torch.exp(-0.5 * ((x.double() - v) / h) ** 2).sum() for v in q[:sel].double()])
    ok = ref > 1e-30 * ref.max()
    assert ((got - ref).abs() <= 3e-7 * ref)[ok].all(), float(((got - ref).abs() / ref)[ok].max())
