"""Surrogate inference with two query tiles in turn against one tile per block.

A query's output is the same sequence of operations whichever tile, turn or
block it falls in, so a large batch (two tiles in turn, an odd last tile, a
partial last tile, several turns per block) equals the small batches that it
is made of (at most one tile per block) bit for bit: tolerance 0.
"""
import pytest
import torch

from test_gpu_mlp import _case, _dev

pytestmark = pytest.mark.gpu

TILE = 128


@pytest.mark.parametrize("members,tiles,last", [(1, 1, 1), (1, 305, 127), (3, 51, 128), (4, 39, 1), (4, 76, 128),
                                                (4, 117, 77), (8, 60, 5), (8, 19, 128), (8, 21, 9)])
def test_two_tiles_in_turn_equal_one(cuda_dev, members, tiles, last):
    from fsk import ops

    batch = TILE * (tiles - 1) + last
    _, params, x, mean, istd = _case(5, batch, members)
    P, X, M, S = (_dev(a, cuda_dev) for a in (params, x, mean, istd))
    packed = ops.mlp_pack(P, members, M, S, 1.5, -0.25)
    got = ops.mlp_infer(packed, members, X)
    piece = TILE * min(16, torch.cuda.get_device_properties(cuda_dev).multi_processor_count // members)
    want = torch.cat([ops.mlp_infer(packed, members, X[i:i + piece].contiguous()) for i in range(0, batch, piece)], 1)
    assert bool(torch.isfinite(got).all())
    assert torch.equal(got, want)
