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


def _layer_and_inputs(cls):
    cfg = wl.MoEConfig("call", 40, 256, 128, 6, 2, 11)
    layer = cls(*wl.make_weights(cfg, device="cuda"), cfg.topk, max_tokens=cfg.tokens, tile_m=16, stage2_mode="reduce")
    xq, xs_t = quant_act_1x128(wl.make_activations(cfg, device="cuda")[0])
    return layer, wl.make_logits(cfg, device="cuda"), xq, xs_t


class _FirstExperts(FusedMoEBlockscale):
    """A router of its own: experts 0 and 1, equal weights."""

    def gate(self, logits, tokens, stream):
        self.topk_ids[:tokens] = torch.arange(self.topk, dtype=torch.int32, device=self.device)
        self.topk_weights[:tokens] = 1.0 / self.topk


def test_an_overridden_piece_is_used():
    layer, logits, xq, xs_t = _layer_and_inputs(_FirstExperts)
    got = layer(logits, xq, xs_t).clone()
    T = logits.shape[0]
    ids = torch.arange(2, dtype=torch.int32, device="cuda").repeat(T, 1)
    tw = torch.full((T, 2), 0.5, device="cuda")
    want = layer.experts_forward(ids, tw, xq, xs_t, T, torch.cuda.current_stream().cuda_stream)[:T]
    assert torch.equal(got, want)
    # a piece replaced on the object
    plain, *_ = _layer_and_inputs(FusedMoEBlockscale)
    calls = []
    plain.experts_forward = lambda *a, **k: (calls.append(1), FusedMoEBlockscale.experts_forward(plain, *a, **k))[1]
    plain(logits, xq, xs_t)
    torch.cuda.synchronize()
    assert calls == [1] and _lib.device_status() == 0
