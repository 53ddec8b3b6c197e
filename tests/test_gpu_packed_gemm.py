"""GEMM-family layers and MLPs in the forms that a pass gives them, against the CPU oracle and the layers called one
by one.  Integers and bits are exact; logits are one fp32 multiply-add on an exact integer (rounded once here, twice
in the oracle: 2^-23 of the larger term)."""
import numpy as np
import pytest
import torch

import util
from tcbnn_b200 import models, ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch", [8, 100])
def test_small_mlp_follows_weights_and_parameters_written_between_passes(cuda, batch):
    """Layers of a pass read weights, thresholds, scale and bias ahead of the wait for the layer in front: what the
    library or torch writes into them right before a pass counts in it."""
    spec = models.mlp_spec(batch)
    w, other = models.synthetic_weights(spec, 31), models.synthetic_weights(spec, 33)
    x = models.synthetic_input(spec, 32)
    net, plain = models.Network(spec, w, x), models.Network(spec, other, x)
    for _ in range(4):
        net.forward()
    want = plain.forward().clone()
    assert not torch.equal(net.forward(), want)
    for n, p in zip(net.layers[1:], plain.layers[1:]):
        for name in ("weight_gpu", "bn_gpu", "bn_scale_gpu", "bn_bias_gpu"):
            if hasattr(n, name):
                getattr(n, name).copy_(getattr(p, name))
    assert torch.equal(net.forward(), want)
    g = util.rng(batch)
    src = torch.from_numpy(util.rand_words(g, (1024, 4)).view(np.int32)).to(cuda)
    big, zero = torch.zeros((1024, 4), dtype=torch.int32, device=cuda), torch.zeros(1024, device=cuda)
    for _ in range(3):                                   # the library's own launch in front of the pass
        ops.fc_layer(src, big, zero, 128, out=net.layers[2].weight_gpu)
        got = net.forward().clone()
        plain.layers[2].weight_gpu.copy_(net.layers[2].weight_gpu)
        assert torch.equal(got, plain.forward())
        src.bitwise_not_()
