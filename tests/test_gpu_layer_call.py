"""The layer's one-call path (flymoe_moe_layer) against the same pieces enqueued one by one, bit for bit.

forward() takes the pieces when GEMM timing is on, so both paths are reachable from the same object.  "reduce" mode
is deterministic; "atomic" adds two terms per token here, whose sum does not depend on their order."""
import pytest
import torch

from flydsl_b200 import _lib, workloads as wl
from flydsl_b200.layer import FusedMoEBlockscale, quant_act_1x128

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["atomic", "reduce"])
@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("tokens,tile_m,logits_dtype", [(1, 16, torch.float32), (77, 32, torch.bfloat16),
                                                        (300, 64, torch.float16), (300, 128, torch.float32)])
def test_one_call_equals_the_pieces(tokens, tile_m, logits_dtype, out_dtype, mode):
    cfg = wl.MoEConfig("call", tokens, 384, 256, 6, 2, 11)
    layer = FusedMoEBlockscale(*wl.make_weights(cfg, device="cuda"), cfg.topk, max_tokens=tokens + 3, tile_m=tile_m,
                               out_dtype=out_dtype, stage2_mode=mode)
    logits = wl.make_logits(cfg, device="cuda").to(logits_dtype)
    xq, xs_t = quant_act_1x128(wl.make_activations(cfg, device="cuda")[0])
    one = layer(logits, xq, xs_t).clone()
    layer.timing_events = []
    pieces = layer(logits, xq, xs_t).clone()
    torch.cuda.synchronize()
    assert _lib.device_status() == 0 and len(layer.timing_events) == 2
    assert one.shape == pieces.shape == (tokens, cfg.model_dim)
    assert torch.equal(one, pieces)


def test_one_call_refuses_what_the_pieces_refuse():
    cfg = wl.MoEConfig("call", 8, 256, 128, 4, 2, 11)
    layer = FusedMoEBlockscale(*wl.make_weights(cfg, device="cuda"), cfg.topk, max_tokens=8, tile_m=16)
    logits = wl.make_logits(cfg, device="cuda")
    xq, xs_t = quant_act_1x128(wl.make_activations(cfg, device="cuda")[0])
    with pytest.raises(ValueError, match="exceeds max_tokens"):
        layer(logits.repeat(2, 1), xq.view(torch.uint8).repeat(2, 1), xs_t.repeat(1, 2))
    with pytest.raises(ValueError, match="logits"):
        layer(logits.double(), xq, xs_t)
    with pytest.raises(ValueError, match="xq"):
        layer(logits, xq[:4], xs_t)
    with pytest.raises(ValueError, match="contiguous"):
        layer(logits, xq, xs_t.t())
