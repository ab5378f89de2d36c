"""Launches whose tiles' K range is shared by a cluster of CTAs, routed, both stages: every operand type, output type
and way of storing, against float64 on the same codes.  The route is asserted, not assumed.

Tolerances: products of the codes are exact in fp32, and fp32 sums in another order differ by well under 1e-5 of the
largest; a 16-bit result adds one rounding (half of EPS, relative), accumulation in 16 bits one for each of a token's
two terms and one for their sum."""
import pytest
import torch

from flydsl_b200 import _lib
from flydsl_b200.kernels import moe_blockscale_2stage as bs
from flydsl_b200.kernels import moe_gemm_2stage as pt
from tests.test_gpu_gemm_routes import EPS, FP8, _sort

pytestmark = pytest.mark.gpu
E, TOPK = 4, 2
TORCH = {"f16": torch.float16, "bf16": torch.bfloat16, "f32": torch.float32}


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _codes(shape, kind, g):
    if kind == "int8":
        return torch.randint(-127, 128, shape, generator=g, device="cuda", dtype=torch.int8)
    x = torch.randn(shape, generator=g, device="cuda")
    return x.to({"fp8": FP8, "bf16": torch.bfloat16, "fp16": torch.float16}[kind])


def _routed(T, seed=7):
    g = _gen(seed)
    ids = torch.rand((T, E), generator=g, device="cuda").argsort(1)[:, :TOPK].to(torch.int32).contiguous()
    return ids, torch.rand((T, TOPK), generator=g, device="cuda") + 0.1


def _assert_shared(stage, scaling, T, n, k_bytes, blocks, tile_m):
    assert _lib.load().flymoe_gemm_ksplit(stage, scaling, T, TOPK, n, k_bytes, blocks, tile_m, None) > 1


def _rows(ids, a, w, rows_of):
    """float64 [T*k, n]: row p is a[rows_of(p)] . w[expert of pair p]^T (factors applied to float64 operands)."""
    y = torch.empty((ids.numel(), w[0].shape[0]), dtype=torch.float64, device="cuda")
    for e in range(E):
        sel = torch.nonzero(ids.view(-1) == e).view(-1)
        y[sel] = a(rows_of(sel)) @ w[e].t()
    return y


def _check(got, ref, out):
    """fp32 sums, or one rounding to 16 bits."""
    tol = 1e-5 * float(ref.abs().max()) + (EPS[TORCH[out]] if out != "f32" else 1e-5) * ref.abs()
    err = (got.double() - ref).abs()
    assert bool((err <= tol).all()), (out, float((err - tol).max()), float(ref.abs().max()))


def _check_sum(got, terms, out):
    """Weighted terms of a token added up in memory of type `out`."""
    ref = terms.sum(1)
    eps = EPS[TORCH[out]] if out != "f32" else 0.0
    tol = 1e-5 * float(terms.abs().max()) + eps * (terms.abs().sum(1) + ref.abs())
    err = (got.double() - ref).abs()
    assert bool((err <= tol).all()), (out, float((err - tol).max()), float(ref.abs().max()))


# (tokens, row block, stage-1 columns, stage-2 columns): about 10-20, 20-30 and 35-60 tiles, so clusters of 8, 4 and 2;
# stage-2 columns 128 mod 256 leave the last tile half empty
SIZES = [(5, 16, 256, 640), (20, 32, 512, 1280), (20, 64, 1024, 1664), (20, 16, 1024, 1664)]


@pytest.mark.parametrize("T,tile_m,n1,n2", SIZES)
@pytest.mark.parametrize("kind", ["fp8", "int8", "bf16", "fp16"])
def test_pertoken(kind, T, tile_m, n1, n2):
    K, g = 1152, _gen(11)                      # 9 K blocks of 8-bit operands: uneven shares
    half = kind in ("bf16", "fp16")
    kb = K * (2 if half else 1)
    ids, tw = _routed(T)
    (s_ids, s_w, s_e, nv), blocks = _sort(ids, tw, E, tile_m)
    _assert_shared(1, _lib.SCALE_PER_TOKEN, T, n1, kb, blocks, tile_m)
    _assert_shared(2, _lib.SCALE_PER_TOKEN, T, n2, kb, blocks, tile_m)
    x, a2 = _codes((T, K), kind, g), _codes((T * TOPK, K), kind, g)
    w1, w2 = _codes((E, 2 * n1, K), kind, g), _codes((E, n2, K), kind, g)
    none = torch.empty(0, device="cuda")
    # scales that bring a sum of K products to the order of one, so that the activation is neither linear nor saturated
    mag = {"int8": 5e-6}.get(kind, 0.03)
    sx, sa = (torch.rand(n, generator=g, device="cuda") + 0.5 for n in (T, T * TOPK))
    sw1, sw2 = ((torch.rand(n, generator=g, device="cuda") + 0.5) * mag for n in (E * 2 * n1, E * n2))
    if half:
        w1, w2 = (w * mag for w in (w1, w2))

    def a64(t, s):
        return (lambda p: t[p].double()) if half else (lambda p: t[p].double() * s[p].double()[:, None])

    def w64(w, s):
        return [w[e].double() if half else w[e].double() * s.view(E, -1)[e].double()[:, None] for e in range(E)]

    common = dict(experts=E, topk=TOPK, tile_m=tile_m, tile_k=128, in_dtype=kind, w_layout="plain")
    both = _rows(ids, a64(x, sx), w64(w1, sw1), lambda p: p // TOPK)
    h = torch.nn.functional.silu(both[:, :n1]) * both[:, n1:] * tw.view(-1, 1).double()
    for out in ("f16", "bf16"):
        o1 = torch.full((T * TOPK, n1), 7.0, dtype=TORCH[out], device="cuda")
        pt.compile_moe_gemm1(model_dim=K, inter_dim=n1, tile_n=128, doweight_stage1=True, out_dtype=out, **common)(
            o1, x, w1, none if half else sx, none if half else sw1, s_ids, s_e, s_w, nv, T, n1, K, blocks)
        _check(o1, h, out)
    pairs = _rows(ids, a64(a2, sa), w64(w2, sw2), lambda p: p)
    weighted = pairs * tw.view(-1, 1).double()
    for out, acc in (("f16", True), ("bf16", True), ("f32", True), ("f16", False), ("bf16", False)):
        o2 = torch.zeros((T if acc else T * TOPK, n2), dtype=TORCH[out], device="cuda")
        pt.compile_moe_gemm2(model_dim=n2, inter_dim=K, tile_n=256, doweight_stage2=True, out_dtype=out, accumulate=acc,
                             **common)(o2, a2, w2, none if half else sa, none if half else sw2, s_ids, s_e, s_w, nv, T, n2, K,
                                       blocks)
        if acc:
            _check_sum(o2, weighted.view(T, TOPK, n2), out)
        else:
            _check(o2, weighted, out)
    torch.cuda.synchronize()
    assert _lib.device_status() == 0


# the last one runs three rounds of tiles per cluster
@pytest.mark.parametrize("T,tile_m,n1,n2,K", [s + (1152,) for s in SIZES] + [(5, 16, 256, 7680, 7168)])
def test_blockscale(T, tile_m, n1, n2, K):
    g = _gen(13)
    ids, tw = _routed(T)
    (s_ids, s_w, s_e, nv), blocks = _sort(ids, tw, E, tile_m)
    _assert_shared(1, _lib.SCALE_BLOCK128, T, n1, K, blocks, tile_m)
    _assert_shared(2, _lib.SCALE_BLOCK128, T, n2, K, blocks, tile_m)
    x, a2 = _codes((T, K), "fp8", g), _codes((T * TOPK, K), "fp8", g)
    w1, w2 = _codes((E, 2 * n1, K), "fp8", g), _codes((E, n2, K), "fp8", g)
    sx, sa = (torch.rand((K // 128, n), generator=g, device="cuda") + 0.5 for n in (T, T * TOPK))
    sw1, sw2 = ((torch.rand((E, n // 128, K // 128), generator=g, device="cuda") + 0.5) * 0.03 for n in (2 * n1, n2))

    def a64(t, s):
        return lambda p: t[p].double() * s.t()[p].double().repeat_interleave(128, 1)

    def w64(w, s):
        return [w[e].double() * s[e].double().repeat_interleave(128, 0).repeat_interleave(128, 1) for e in range(E)]

    common = dict(experts=E, topk=TOPK, tile_m=tile_m, tile_k=128, w_layout="plain")
    both = _rows(ids, a64(x, sx), w64(w1, sw1), lambda p: p // TOPK)
    h = torch.nn.functional.silu(both[:, :n1]) * both[:, n1:]
    for out in ("f16", "bf16"):
        o1 = torch.full((T * TOPK, n1), 7.0, dtype=TORCH[out], device="cuda")
        bs.compile_moe_blockscale_gemm1(model_dim=K, inter_dim=n1, tile_n=128, doweight_stage1=False, out_dtype=out, **common)(
            o1, x, w1, sx, sw1.view(-1), s_ids, s_e, s_w, nv, T, n1, K, blocks, None)
        _check(o1, h, out)
    pairs = _rows(ids, a64(a2, sa), w64(w2, sw2), lambda p: p)
    weighted = pairs * tw.view(-1, 1).double()
    for out, acc in (("f16", True), ("bf16", True), ("f32", True), ("f16", False), ("bf16", False)):
        o2 = torch.zeros((T if acc else T * TOPK, n2), dtype=TORCH[out], device="cuda")
        bs.compile_moe_blockscale_gemm2(model_dim=n2, inter_dim=K, tile_n=256, doweight_stage2=True, out_dtype=out,
                                        accumulate=acc, **common)(o2, a2, w2, sa, sw2.view(-1), s_ids, s_e, s_w, nv, T, n2, K,
                                                                  blocks)
        if acc:
            _check_sum(o2, weighted.view(T, TOPK, n2), out)
        else:
            _check(o2, weighted, out)
    torch.cuda.synchronize()
    assert _lib.device_status() == 0
