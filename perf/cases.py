"""Performance cases of the framework: what a serving process has it do, through its public entry points.

Three families, each over the range of sizes it is used at:

* ``layer``     bf16 hidden states and router logits -> 1x128 quantiser -> fused FP8 block-scaled MoE layer
                (gating, sort, stage 1, stage 2); decode to prefill, uniform and skewed routing, both
                stage-2 modes, both output types.
* ``pertoken``  already-routed tokens through the reference-shaped launchers of the per-token-scale
                family: sort, ``compile_moe_gemm1``, ``compile_moe_gemm2`` (fp8, int8 and 16-bit operands).
* ``dense``     the dense FP8 block-scaled GEMM launcher (projections around the experts).

Sizes are those of ``flydsl_b200.workloads``, the tests and ``bench.py``, and neighbours of them.
"""

from __future__ import annotations

import math

import torch

from flydsl_b200 import workloads as wl
from flydsl_b200.kernels.blockscale_preshuffle_gemm import compile_blockscale_preshuffle_gemm
from flydsl_b200.kernels.moe_blockscale_2stage import prepare_weight, shuffle_weight
from flydsl_b200.kernels.moe_gemm_2stage import compile_moe_gemm1, compile_moe_gemm2
from flydsl_b200.kernels.moe_sorting_kernel import moe_sorting_flydsl
from flydsl_b200.layer import FusedMoEBlockscale, quant_act_1x128

FP8 = torch.float8_e4m3fn
_DT = {"f32": torch.float32, "bf16": torch.bfloat16, "f16": torch.float16}
# (model_dim, inter_dim, experts, topk) of the repository's configurations
_TINY, _MIXTRAL, _DSV3 = (1024, 512, 8, 2), (4096, 14336, 8, 2), (7168, 2048, 256, 8)
# ceilings for a drawn case: the operations and the weight bytes of the largest listed ones
_MAX_FLOPS = 6.0 * 8192 * 2 * 4096 * 14336
_MAX_WEIGHT_BYTES = 3.0 * 256 * 7168 * 2048


def _layer(name, tokens, dims, *, routing="uniform", logits="f32", out="bf16", mode="atomic"):
    H, I, E, k = dims
    return {"name": name, "family": "layer", "tokens": tokens, "model_dim": H, "inter_dim": I, "experts": E, "topk": k,
            "routing": routing, "logits": logits, "out": out, "mode": mode}


def _pertoken(name, tokens, dims, in_dtype, out, tile_m):
    H, I, E, k = dims
    return {"name": name, "family": "pertoken", "tokens": tokens, "model_dim": H, "inter_dim": I, "experts": E, "topk": k,
            "in_dtype": in_dtype, "out": out, "tile_m": tile_m}


def _dense(name, m, n, k, out):
    return {"name": name, "family": "dense", "m": m, "n": n, "k": k, "out": out}


def listed():
    return [
        # a small model's decode step: five short launches, time is launches and latency
        _layer("layer-tiny-t32", 32, _TINY),
        # one sequence decoding on a few wide experts: two experts' weights per step
        _layer("layer-mixtral-t1", 1, _MIXTRAL),
        # a decode batch on the same layer: every expert's weights, about 32 rows each
        _layer("layer-mixtral-t128", 128, _MIXTRAL),
        # long prefill on the same layer: tensor cores
        _layer("layer-mixtral-t8192", 8192, _MIXTRAL),
        # decode batch on many narrow experts (the benchmark's decode leg): weight streaming
        _layer("layer-dsv3-t64", 64, _DSV3),
        # a mixed or chunked-prefill batch of no round size, 16-bit router and f16 output
        _layer("layer-dsv3-t777", 777, _DSV3, logits="bf16", out="f16"),
        # prefill (the benchmark's headline configuration)
        _layer("layer-dsv3-t4096", 4096, _DSV3),
        # prefill with the skewed routing real routers show, deterministic combine
        _layer("layer-dsv3-t4096-zipf", 4096, _DSV3, routing="zipf", mode="reduce"),
        # per-token-scale FP8 at the odd shape of the reference's own large test
        _pertoken("pertoken-fp8-t333", 333, (4096, 2048, 17, 9), "fp8", "f16", 64),
        # unquantised 16-bit experts, medium prefill
        _pertoken("pertoken-bf16-t1024", 1024, _MIXTRAL, "bf16", "bf16", 128),
        # a projection during decode (the 2112-column weight: a ragged last tile)
        _dense("dense-m64-n2112-k7168", 64, 2112, 7168, "bf16"),
        # a projection during prefill
        _dense("dense-m4096-n7168-k2304", 4096, 7168, 2304, "bf16"),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    """One more case of the same ranges (token counts spread over their logarithm, odd ones included)."""
    while True:
        family = rng.choice(("layer", "layer", "layer", "pertoken", "dense"))
        if family == "dense":
            n, k = rng.choice(((7168, 2304), (2112, 7168), (3072, 1536), (7168, 2048), (1536, 7168), (4608, 7168),
                               (1280, 7168)))
            c = _dense("", _log_int(rng, 1, 8192), n, k, rng.choice(("bf16", "fp16")))
        elif family == "pertoken":
            dims = rng.choice(((4096, 2048, 17, 9), (1024, 256, 8, 2), _MIXTRAL, (7168, 2048, 32, 8)))
            tokens = _log_int(rng, 1, 4096)
            c = _pertoken("", tokens, dims, rng.choice(("fp8", "fp8", "int8", "bf16", "fp16")),
                          rng.choice(("bf16", "f16")), _tile_m(tokens, dims[2], dims[3]))
            if c["in_dtype"] == "fp16":
                c["out"] = "f16"               # stage 1's output is stage 2's input
            elif c["in_dtype"] == "bf16":
                c["out"] = "bf16"
        else:
            dims = rng.choice((_TINY, _MIXTRAL, _MIXTRAL, _DSV3, _DSV3, (2048, 1024, 64, 6)))
            c = _layer("", _log_int(rng, 1, 8192), dims, routing=rng.choice(("uniform", "uniform", "zipf")),
                       logits=rng.choice(("f32", "bf16", "f16")), out=rng.choice(("bf16", "bf16", "f16")),
                       mode=rng.choice(("atomic", "atomic", "reduce")))
        del c["name"]
        ebytes = 2 if c.get("in_dtype") in ("bf16", "fp16") else 1
        if family != "dense":
            weights = 3.0 * c["experts"] * c["model_dim"] * c["inter_dim"] * ebytes
            if weights > _MAX_WEIGHT_BYTES:
                continue
        # 16-bit operands run at half the 8-bit rate
        if work(c)["flops"] * ebytes <= _MAX_FLOPS:
            return c


# ----------------------------------------------------------------------------------------- inputs
def _tile_m(tokens, experts, topk):
    """Row block a caller picks: the smallest that covers the mean rows per expert (as bench.py does)."""
    rows = tokens * topk / experts
    return next((m for m in (16, 32, 64) if rows <= m), 128)


def _config(case, seed):
    return wl.MoEConfig("case", case["tokens"], case["model_dim"], case["inter_dim"], case["experts"], case["topk"], seed,
                        case.get("routing", "uniform"))


def _randn(shape, seed, std=1.0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(shape, generator=g, device="cuda", dtype=torch.float32) * std


def prepare(case, seed):
    seed = int(seed) % (1 << 30)
    return {"layer": _prepare_layer, "pertoken": _prepare_pertoken, "dense": _prepare_dense}[case["family"]](case, seed)


def _prepare_layer(case, seed):
    """The model's layer with its weights, and one batch's hidden states and router logits."""
    cfg = _config(case, seed)
    weights = wl.make_weights(cfg, device="cuda")
    layer = FusedMoEBlockscale(*weights, cfg.topk, max_tokens=cfg.tokens,
                               tile_m=_tile_m(cfg.tokens, cfg.experts, cfg.topk), out_dtype=_DT[case["out"]],
                               stage2_mode=case["mode"])
    return {"family": "layer", "layer": layer, "x": _randn((cfg.tokens, cfg.model_dim), seed + 1).to(torch.bfloat16),
            "logits": wl.make_logits(cfg, device="cuda").to(_DT[case["logits"]])}


def _quant_rows(w, in_dtype):
    """One scale per row: (codes, f32 scales)."""
    if in_dtype == "fp8":
        q, s = wl.quant_groups(w)
        return q, s.squeeze(-1)
    s = w.abs().amax(dim=-1, keepdim=True) / 127.0
    return torch.round(w / s).to(torch.int8), s.squeeze(-1)


def _prepare_pertoken(case, seed):
    """Weights and launchers of one layer; one batch's routing, activations and, for the 8-bit types, the
    quantised stage-2 input (the caller quantises between the stages); the buffers a caller keeps."""
    T, H, I, E, k = (case[n] for n in ("tokens", "model_dim", "inter_dim", "experts", "topk"))
    U, kind = case["tile_m"], case["in_dtype"]
    half = {"bf16": torch.bfloat16, "fp16": torch.float16}.get(kind)
    wdt = half or (FP8 if kind == "fp8" else torch.int8)
    i32, f32, dev = torch.int32, torch.float32, "cuda"
    empty = torch.empty(0, dtype=f32, device=dev)
    w1, w2 = torch.empty((E, 2 * I, H), dtype=wdt, device=dev), torch.empty((E, H, I), dtype=wdt, device=dev)
    s1 = s2 = sx = sa2 = empty
    if half is None:
        s1, s2 = torch.empty((E, 2 * I), dtype=f32, device=dev), torch.empty((E, H), dtype=f32, device=dev)
    for e in range(E):
        for j, (w, s) in enumerate(((w1, s1), (w2, s2))):
            r = _randn(w.shape[1:], seed + 7919 * (2 * e + j) + 3, 0.02)
            if half is not None:
                w[e] = r.to(half)
            else:
                w[e], s[e] = _quant_rows(r, kind)
    x = _randn((T, H), seed + 1)
    if half is not None:
        x, a2 = x.to(half), None
    else:
        x, sx = _quant_rows(x, kind)
        a2, sa2 = _quant_rows(_randn((T * k, I), seed + 2, 0.5), kind)
    ids_w = torch.topk(torch.softmax(wl.make_logits(_config(case, seed), device=dev), dim=-1), k, dim=-1)
    rows = T * k + E * U - k
    blocks = (rows + U - 1) // U
    odt = _DT[case["out"]]
    dims = dict(model_dim=H, inter_dim=I, experts=E, topk=k, tile_m=U, tile_k=128, in_dtype=kind, out_dtype=case["out"],
                w_layout="plain")
    return {"family": "pertoken", "T": T, "H": H, "I": I, "E": E, "U": U, "blocks": blocks,
            "gemm1": compile_moe_gemm1(tile_n=128, doweight_stage1=False, **dims),
            "gemm2": compile_moe_gemm2(tile_n=256, doweight_stage2=True, **dims),
            "ids": ids_w.indices.to(i32).contiguous(),
            "weights": (ids_w.values / ids_w.values.sum(-1, keepdim=True)).contiguous(),
            "w1": w1, "w2": w2, "s1": s1.view(-1), "s2": s2.view(-1), "x": x, "sx": sx, "a2": a2, "sa2": sa2,
            "sorted": (torch.empty(rows, dtype=i32, device=dev), torch.empty(rows, dtype=f32, device=dev),
                       torch.empty(blocks, dtype=i32, device=dev), torch.empty(2, dtype=i32, device=dev)),
            "sort_ws": torch.empty(max(1, ((T * k + 127) // 128 + 1) * E), dtype=i32, device=dev),
            "out1": torch.empty((T * k, I), dtype=odt, device=dev), "out2": torch.empty((T, H), dtype=odt, device=dev)}


def _prepare_dense(case, seed):
    """A preshuffled weight, converted at load time, and one batch of already-quantised activations."""
    m, n, k = case["m"], case["n"], case["k"]
    pad = (n + 127) // 128 * 128
    w, sw = wl.quant_weight_128x128(torch.nn.functional.pad(_randn((n, k), seed + 3, 0.02), (0, 0, 0, pad - n)))
    w = shuffle_weight(w[:n].contiguous(), n, k)
    prepare_weight(w, n, k)
    xq, xs = wl.quant_act_1x128(_randn((m, k), seed + 1))
    out = {"bf16": torch.bfloat16, "fp16": torch.float16}[case["out"]]
    return {"family": "dense", "m": m, "n": n, "w": w, "sw": sw, "x": xq, "sx": xs.t().contiguous(),
            "gemm": compile_blockscale_preshuffle_gemm(M=m, N=n, K=k, tile_m=_tile_m(m, 1, 1), tile_n=128, tile_k=128,
                                                       out_dtype=case["out"]),
            "c": torch.empty((m, n), dtype=out, device="cuda")}


# ----------------------------------------------------------------------------------------- one pass
def run(state):
    if state["family"] == "layer":
        xq, xs_t = quant_act_1x128(state["x"])
        return state["layer"](state["logits"], xq, xs_t)
    s = state
    if s["family"] == "dense":
        s["gemm"](s["c"], s["x"], s["w"], s["sx"], s["sw"], s["m"], s["n"])
        return s["c"]
    s_ids, s_w, s_e, nv = s["sorted"]
    moe_sorting_flydsl(s["ids"], s["weights"], s_ids, s_w, s_e, nv, s["out2"], s["E"], s["U"], workspace=s["sort_ws"])
    s["gemm1"](s["out1"], s["x"], s["w1"], s["sx"], s["s1"], s_ids, s_e, s_w, nv, s["T"], s["I"], s["H"], s["blocks"])
    a2 = s["out1"] if s["a2"] is None else s["a2"]
    s["gemm2"](s["out2"], a2, s["w2"], s["sa2"], s["s2"], s_ids, s_e, s_w, nv, s["T"], s["H"], s["I"], s["blocks"])
    return {"stage1": s["out1"], "stage2": s["out2"]}


# ----------------------------------------------------------------------------------------- work
def work(case):
    """Bytes: the routed experts' weights and scales, the inputs and the outputs, once each; intermediates that stay
    inside the framework are not counted.  Operations: those of the real (token, slot) pairs, without padding."""
    if case["family"] == "dense":
        m, n, k = case["m"], case["n"], case["k"]
        scales = 4.0 * (m * (k // 128) + ((n + 127) // 128) * (k // 128))
        return {"bytes": float(m * k + n * k + 2 * m * n) + scales, "flops": 2.0 * m * n * k}
    T, H, I, E, k = (case[n] for n in ("tokens", "model_dim", "inter_dim", "experts", "topk"))
    # experts that receive a token under this routing (one seeded sample of it)
    ids = torch.topk(wl.make_logits(_config(case, 1)), k, dim=-1).indices
    active = float(torch.unique(ids).numel())
    flops = 6.0 * T * k * H * I
    if case["family"] == "layer":
        weights = active * 3.0 * H * I * (1 + 4.0 / (128 * 128))
        return {"bytes": weights + T * H * 4.0 + T * E * (4.0 if case["logits"] == "f32" else 2.0), "flops": flops}
    half = case["in_dtype"] in ("bf16", "fp16")
    eb, sc = (2.0, 0.0) if half else (1.0, 4.0)
    weights = active * (3.0 * H * I * eb + (2 * I + H) * sc)
    acts = T * (H * eb + sc) + T * k * 2.0 * I + (0.0 if half else T * k * (I + sc)) + T * H * 2.0
    return {"bytes": weights + acts + 8.0 * T * k, "flops": flops}


def tolerance(case):
    """About four times what each path differs by from itself in 64-bit arithmetic on the same quantised inputs.
    Seen (2-norm, largest): the 16-bit rounding of the result, 1.7e-3 / 4e-3 (bf16), 2.1e-4 / 5e-4 (f16); with the
    experts' terms added up in bf16 memory 2.4e-3 / 2e-2 for 2 of them and 4.1e-3 / 2.9e-2 for 8, in f16 5e-4 / 4e-3."""
    bf16 = case["out"] == "bf16"
    if case["family"] == "dense":
        return {"rel": 7e-3, "max": 1.6e-2} if bf16 else {"rel": 9e-4, "max": 2e-3}
    if not bf16:
        return {"rel": 2e-3, "max": 1.6e-2}
    summed_in_memory = case["family"] == "pertoken" or case["mode"] == "atomic"
    return {"rel": 1.6e-2 if summed_in_memory and case["topk"] > 2 else 1e-2, "max": 0.12 if case["topk"] > 2 else 8e-2}
