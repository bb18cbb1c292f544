"""Numbers as the entry points take them: whatever ``float`` converts, and the documented errors for the rest."""

import pytest
import torch

import oops_b200 as oops

pytestmark = pytest.mark.gpu


def test_scale(cuda):
    q = torch.randn(1, 4, 16, 2, 32, device=cuda, dtype=torch.bfloat16)
    tokens = torch.randn(2, 3, 16, 24, device=cuda, dtype=torch.bfloat16)
    calls = [lambda s: oops.triangle_attention(q, q, q, scale=s), lambda s: oops.triangle_attention_gated(q, q, q, q, scale=s),
             lambda s: oops.pair_bias_attention(tokens, tokens, tokens, scale=s)]
    for call in calls:
        want = call(0.5)
        for scale in ("0.5", torch.tensor(0.5), torch.tensor(0.5, device=cuda).cpu().numpy()):
            assert torch.equal(call(scale), want)
        for scale, error in (("half", ValueError), ([0.5], TypeError), (0.5j, TypeError), (10**400, OverflowError)):
            with pytest.raises(error):
                call(scale)


def test_layer_norm(cuda):
    x = torch.randn(6, 16, device=cuda)
    want = oops.layer_norm(x, 16, eps=1e-3)
    for eps in ("1e-3", torch.tensor(1e-3, dtype=torch.float64)):
        assert torch.equal(oops.layer_norm(x, 16, eps=eps), want)
    for eps in (None, [1e-3]):
        with pytest.raises(TypeError):
            oops.layer_norm(x, 16, eps=eps)
    for width in (2**70, -(2**70), -1, 0):
        with pytest.raises(oops.OOpsUnsupportedError):
            oops.layer_norm(x, width)
