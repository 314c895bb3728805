"""The two paths of the 1-D KDE above the size where the cell expansions are
tried: against each other at full size, on a second stream, in a captured graph
and in the bounds-check build.  One point far outside makes the data too spread
for the expansions and adds nothing to any other query: the pair kernel runs.

The paths are compared at 1e-5, the pair kernel's exponent rounding in the tail."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
FAR = 1e7


def _set(n, seed, dev):
    g = torch.Generator(device=dev)
    g.manual_seed(seed)
    x = torch.randn(n, generator=g, device=dev)
    return torch.where(torch.rand(n, generator=g, device=dev) < 0.4, x * 0.3 + 3.0, x - 1.0)


def _with_far(x):
    return torch.cat([x, torch.full((1,), FAR, device=x.device)])


def test_pair_kernel_at_full_size(cuda_dev):
    """2^22 points at 2^20 queries: split-K and atomic pair sums (their own kernels,
    0.5 s each) and the expansions."""
    from fsk import ops, workloads

    x = torch.from_numpy(workloads.gmm3_1d(1 << 22, seed=0)).to(cuda_dev)
    q = torch.from_numpy(workloads.grid_1d(1 << 20)).to(cuda_dev)
    h = 0.05   # the tables hold a spread of 447 h
    cells = ops.kde1d_sum(q, x, h)
    split_k = ops.kde1d_sum(q, _with_far(x), h)
    atomic = ops.kde1d_sum(q, _with_far(x), h, atomic=True)
    ops.device_status(cuda_dev)
    assert not torch.equal(split_k, cells)
    keep = cells > 1e-20 * cells.max()
    for a, b in ((split_k, cells), (atomic, cells), (atomic, split_k)):
        assert ((a - b).abs() <= 1e-5 * b)[keep].all()


def test_second_stream(cuda_dev):
    from fsk import ops

    n, m = 1 << 18, 8192
    xs = [_set(n, 1, cuda_dev), _with_far(_set(n, 2, cuda_dev)), _set(n, 3, cuda_dev)]
    q = torch.linspace(-5, 5, m, device=cuda_dev)
    want = [ops.kde1d_sum(q, x, 0.05) for x in xs]
    streams = [torch.cuda.Stream(cuda_dev) for _ in xs]
    torch.cuda.synchronize(cuda_dev)
    got = []
    for _ in range(20):
        for x, s in zip(xs, streams):
            with torch.cuda.stream(s):
                got.append(ops.kde1d_sum(q, x, 0.05))
    torch.cuda.synchronize(cuda_dev)
    ops.device_status(cuda_dev)
    for i, y in enumerate(got):
        assert torch.equal(y, want[i % 3])


def test_captured_graph_takes_the_path_of_each_replay(cuda_dev):
    from fsk import ops

    n, m = 1 << 18, 8192
    q = torch.linspace(-5, 5, m, device=cuda_dev)
    x = _set(n, 1, cuda_dev)
    side = torch.cuda.Stream(cuda_dev)
    side.wait_stream(torch.cuda.current_stream(cuda_dev))
    with torch.cuda.stream(side):
        ops.kde1d_sum(q, x, 0.05)
    torch.cuda.current_stream(cuda_dev).wait_stream(side)
    torch.cuda.synchronize(cuda_dev)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = ops.kde1d_sum(q, x, 0.05)
    for seed, far in ((1, False), (2, True), (3, False), (4, True)):
        fresh = _set(n, seed, cuda_dev)
        if far:
            fresh[7] = FAR
        x.copy_(fresh)
        graph.replay()
        got = out.clone()
        assert torch.equal(got, ops.kde1d_sum(q, fresh, 0.05))
    ops.device_status(cuda_dev)


def test_bounds_check_build(cuda_dev, monkeypatch):
    from fsk import _build, ops
    from fsk import _lib as L

    def run():
        outs = []
        for n, m in ((4096, 262145), (65537, 16411), (1 << 20, 1025)):
            q = torch.linspace(-30, 40, m, device=cuda_dev)
            for x in (_set(n, 5, cuda_dev), _with_far(_set(n, 5, cuda_dev))):
                for kw in ({}, {"atomic": True}, {"log_eps": 1e-9}):
                    outs.append(ops.kde1d_sum(q, x, 0.05, **kw))
        ops.device_status(cuda_dev)   # raises on a reported index
        return outs

    want = run()
    checked, normal = L.load(_build.build(checked=True)), L.load()
    monkeypatch.setattr(L, "_lib", checked)
    assert L.load() is checked
    got = run()
    monkeypatch.setattr(L, "_lib", normal)
    for a, b in zip(got, want):
        np.testing.assert_allclose(a.cpu().numpy(), b.cpu().numpy(), rtol=1e-6, atol=1e-37)
