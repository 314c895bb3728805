"""Training products at tile edges: forward values and every
gradient block against FP64 with the model's bf16 roundings.

Tolerance (2-norm): tanh.approx is good to 2^-11 and enters every layer once
forward and once backward, roughly 6 x 5e-4 when nothing averages out: 5e-3."""
import pytest
import torch

pytestmark = pytest.mark.gpu
H, D = 256, 16
BLOCKS = (("W1", H * D), ("b1", H), ("W2", H * H), ("b2", H), ("W3", H * H), ("b3", H), ("w4", H), ("b4", 1))


def _bf(t):
    return t.float().bfloat16().double()


def _reference(params, x, mean, istd, dy):
    w1, b1, w2, b2, w3, b3, w4, b4 = torch.split(params.double(), [s for _, s in BLOCKS])
    ws = [_bf(w1).view(H, D), _bf(w2).view(H, H), _bf(w3).view(H, H)]
    a, z = [_bf((x - mean) * istd)], []
    for w, b in zip(ws, (b1, b2, b3)):
        z.append(a[-1] @ w.T + b)
        a.append(_bf(torch.nn.functional.silu(z[-1])))
    y = a[-1] @ _bf(w4) + b4
    out = [None] * 8
    out[6], out[7] = dy @ a[-1], dy.sum()[None]
    da = dy[:, None] * _bf(w4)[None, :]
    for l in (2, 1, 0):
        sg = torch.sigmoid(z[l])
        dz = da * sg * (1.0 + z[l] * (1.0 - sg))
        out[2 * l], out[2 * l + 1] = (dz.T @ a[l]).reshape(-1), dz.sum(0)
        da = dz @ ws[l]
    return y, out


@pytest.mark.parametrize("batch,members", [(1, 1), (31, 3), (33, 1), (127, 2), (129, 8), (1000, 5), (8192, 1)])
def test_training_pass_matches_fp64(cuda_dev, batch, members):
    from fsk import ops

    g = torch.Generator(device="cuda")
    g.manual_seed(batch + members)
    rand = lambda *s: torch.rand(*s, generator=g, device="cuda") * 2.0 - 1.0
    parts = []
    for _ in range(members):
        parts += [rand(H * D) * 0.6, rand(H) * 0.1, rand(H * H) * 0.15, rand(H) * 0.1, rand(H * H) * 0.15,
                  rand(H) * 0.1, rand(H) * 0.06, rand(1)]
    params = torch.cat(parts).contiguous()
    x, mean, istd = rand(batch, D) * 3.0, rand(D), rand(D).abs() + 0.5
    dy = (rand(members, batch) + 0.3) / batch
    ws = ops.mlp_train_workspace(members, batch, cuda_dev)
    y = ops.mlp_fwd(params, members, x, mean, istd, ws)
    grads = ops.mlp_bwd(params, members, batch, dy, ws)
    again = ops.mlp_bwd(params, members, batch, dy, ws)     # the forward's buffers stay as they were
    ops.device_status(cuda_dev)
    assert ((grads - again).norm() <= 1e-5 * grads.norm())
    size = params.numel() // members
    for k in range(members):
        ref_y, ref_g = _reference(params[k * size:(k + 1) * size], x, mean, istd, dy[k].double())
        assert (y[k] - ref_y).norm() <= 5e-3 * ref_y.norm()
        at = k * size
        for (name, count), ref in zip(BLOCKS, ref_g):
            got = grads[at:at + count]
            at += count
            assert (got - ref).norm() <= 5e-3 * ref.norm(), name
