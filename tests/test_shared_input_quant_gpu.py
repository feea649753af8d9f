"""wuda_layer_decode lets the mHC pre of the feed-forward half quantise the shared expert's input.  Its bytes must be those of the
quantisation by itself, also in groups whose values are tiny (their scales lie below the fused kernel's own clamp) or zero: the
layer called as one against the same entry points called one by one, with such groups made by the norm's weights."""
import pytest
import torch

from wuda_b200.layer_setup import build_random_layer

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch", [1, 6])
def test_tiny_and_zero_groups(batch):
    outs = []
    for native in (False, True):
        layer, slots, x = build_random_layer(batch, 1500, seed=5, native=native, topk=512, experts=32, inter=512, moe_topk=4)
        norm = layer.ffn.ffn_norm
        norm[:128] = 0
        norm[128:256] *= 1e-3       # amax about 4e-3: below 448e-4
        norm[256:384] *= 1e-7
        norm[384:512] *= 1e3
        layer.prepare(slots)
        outs.append(layer.launch(x, batch).clone())
        torch.cuda.synchronize()
        layer.check_status()
    assert bool(torch.isfinite(outs[0].float()).all()) and torch.equal(*outs)
