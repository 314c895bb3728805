"""Device times of the 1-D KDE where the cell expansions are tried: one entry per
call that covers the path taken, and no pairs booked for a pair kernel that
returned at once."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
KDE1D, KDE1D_CELL = 5, 13


def _timed(fn):
    from fsk import _lib as L

    lib = L.load()
    ids, nl = np.zeros(16, np.int32), np.zeros(16, np.int64)
    ms, work = np.zeros(16), np.zeros(16)
    args = (ids.ctypes.data, nl.ctypes.data, ms.ctypes.data, work.ctypes.data, 16)
    fn()
    lib.fsk_timer_collect(*args)
    lib.fsk_timer_enable(1)
    try:
        fn()
    finally:
        lib.fsk_timer_enable(0)
    rows = lib.fsk_timer_collect(*args)
    return {int(ids[r]): (int(nl[r]), float(ms[r]), float(work[r])) for r in range(rows)}


def test_one_entry_for_the_path_taken(cuda_dev):
    from fsk import ops

    n, m = 1 << 20, 4096
    g = torch.Generator(device=cuda_dev)
    g.manual_seed(1)
    x = torch.randn(n, generator=g, device=cuda_dev)
    q = torch.randn(m, generator=g, device=cuda_dev)
    below = _timed(lambda: ops.kde1d_sum(q[:512], x, 0.1))
    assert set(below) == {KDE1D} and below[KDE1D][2] == n * 512
    cells = _timed(lambda: ops.kde1d_sum(q, x, 0.1))
    assert set(cells) == {KDE1D_CELL} and cells[KDE1D_CELL][0] == 1 and cells[KDE1D_CELL][2] == n * m
    x[5] = 1e6   # too spread: the pair kernel does the work, in the same entry
    pairs = _timed(lambda: ops.kde1d_sum(q, x, 0.1))
    assert set(pairs) == {KDE1D_CELL} and pairs[KDE1D_CELL][2] == n * m
    # the pair rate is that of the exp unit, at most ~1e13 per second
    assert pairs[KDE1D_CELL][1] >= n * m / 1.2e13 * 1e3 > cells[KDE1D_CELL][1]
