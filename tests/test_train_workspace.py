"""Size of the surrogate's training workspace (host side of the library)."""
import pytest


@pytest.mark.parametrize("members", [1, 4, 8])
@pytest.mark.parametrize("batch", [1024, 8192, 100000, 4000000])
def test_no_more_than_28_bytes_per_activation(members, batch):
    """Three layers of 256 features keep z (FP32) and a (bf16), and two buffers take
    the gradients in turn: 26 bytes per feature, beside the inputs and the bf16
    weights.  With FP32 activations and the gradients written over z it was 28."""
    from fsk import _build, _lib

    _build.build()
    size = _lib.load().fsk_mlp_train_workspace_bytes(members, batch)
    assert size <= 28 * members * batch * 256 + 64 * batch
