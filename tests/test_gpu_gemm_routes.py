"""Edges of the GEMM kernels' routes, through the launchers: dense shapes on the cluster (row blocks of 16-64, few
tiles) and one-CTA kernels, and routed ones with enough rows per expert for merged row blocks and, with per-token scales
and row blocks of 64 and 128, for CTA pairs.  Routed launches on the cluster kernel: test_gpu_gemm_split.py.

References: the CPU oracle for dense shapes (16-bit results: one rounding step, 2^-8 / 2^-11 relative, plus fp32 sums
in another order), and the CUDA-core implementation for routed ones."""
import pytest
import torch

from flydsl_b200 import _lib
from flydsl_b200 import workloads as wl
from flydsl_b200.kernels import moe_blockscale_2stage as bs
from flydsl_b200.kernels import moe_gemm_2stage as pt
from flydsl_b200.kernels.blockscale_preshuffle_gemm import compile_blockscale_preshuffle_gemm
from flydsl_b200.kernels.moe_sorting_kernel import moe_sorting_flydsl
from oracle import moe_oracle as orc
from tests.gpu_common import assert_close

pytestmark = pytest.mark.gpu
FP8 = torch.float8_e4m3fn
EPS = {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11}


# K = 128 (nothing to split), 256, 1152 (9 K blocks: uneven shares), 7168; N = 64 mod 128, 128 mod 256, whole tiles;
# M around the row blocks, and around one and two 128-row blocks (which never share K)
@pytest.mark.parametrize("N,K", [(192, 128), (64, 256), (384, 1152), (2112, 7168)])
@pytest.mark.parametrize("M,tile_m", [(1, 16), (16, 16), (17, 32), (64, 64), (96, 128), (128, 128), (129, 128),
                                      (257, 128), (640, 128)])
def test_dense_edges(M, tile_m, N, K):
    g = torch.Generator().manual_seed(M * 31 + N)
    x, xs = wl.quant_act_1x128(torch.randn((M, K), generator=g))
    pad = (N + 127) // 128 * 128
    w, ws = wl.quant_weight_128x128(torch.nn.functional.pad(torch.randn((N, K), generator=g), (0, 0, 0, pad - N)))
    w = w[:N].contiguous()
    ref = orc.blockscale_gemm(x, xs, w, ws)
    exe = compile_blockscale_preshuffle_gemm(M=M, N=N, K=K, tile_m=tile_m, tile_n=128, tile_k=128, out_dtype="fp16",
                                             w_layout="plain")
    c = torch.full((M + 1, N), 7.0, dtype=torch.float16, device="cuda")
    exe(c, x.cuda(), w.cuda(), xs.t().contiguous().cuda(), ws.cuda(), M, N)
    torch.cuda.synchronize()
    assert _lib.device_status() == 0
    # fp32 sums in another order differ by at most a few ulp of the largest partial sum, well under 1e-5 of it
    assert_close(c[:M], ref, 2 * EPS[torch.float16], 1e-5 * float(ref.abs().max()), f"dense {M}x{N}x{K}")
    assert bool((c[M] == 7.0).all())


# rows per expert: none, one, exactly a block, one more, three blocks (odd), two blocks
COUNTS = (0, 1, 128, 129, 300, 256)


def _routing(k=1):
    ids = torch.cat([torch.full((c,), e, dtype=torch.int32) for e, c in enumerate(COUNTS)])
    ids = ids[torch.randperm(ids.numel(), generator=torch.Generator().manual_seed(3))].view(-1, k)
    w = torch.rand(ids.shape, generator=torch.Generator().manual_seed(4)) + 0.1
    return ids.cuda(), w.cuda()


def _sort(ids, w, E, unit):
    T, k = ids.shape
    cap = T * k + E * unit - k
    nblk = (cap + unit - 1) // unit
    i32 = dict(dtype=torch.int32, device="cuda")
    s = (torch.empty(cap, **i32), torch.empty(cap, dtype=torch.float32, device="cuda"), torch.empty(nblk, **i32),
         torch.empty(2, **i32))
    moe_sorting_flydsl(ids, w, *s, None, E, unit)
    return s, nblk


@pytest.mark.parametrize("tile_m", [16, 32, 64, 128])
@pytest.mark.parametrize("H,I,out", [(384, 256, "bf16"), (1024, 128, "f16")])
def test_routed_blockscale_against_cuda_cores(H, I, out, tile_m):
    ids, tw = _routing(2)
    T, k = ids.shape
    E = len(COUNTS)
    cfg = wl.MoEConfig("routes", T, H, I, E, k, 5)
    w1q, w1s, w2q, w2s = wl.make_weights(cfg, device="cuda")
    _x, xq, xs = wl.make_activations(cfg, device="cuda")
    xs_t = xs.t().contiguous()
    (s_ids, s_w, s_e, nv), nblk = _sort(ids, tw, E, tile_m)
    got = {}
    for impl in ("simt", "tcgen05"):
        common = dict(model_dim=H, inter_dim=I, experts=E, topk=k, tile_m=tile_m, tile_k=128, w_layout="plain", impl=impl)
        a2 = torch.full((T * k, I), 0x55, dtype=torch.uint8, device="cuda")
        a2s = torch.full((I // 128, T * k), -1.0, device="cuda")
        bs.compile_moe_blockscale_gemm1(tile_n=128, doweight_stage1=False, out_dtype="fp8", **common)(
            a2, xq, w1q, xs_t, w1s.view(-1), s_ids, s_e, s_w, nv, T, I, H, nblk, None, arg_out_scale=a2s)
        if impl == "simt":
            ref_a2, ref_a2s = a2, a2s                   # both implementations run stage 2 on the same input
        pair = torch.full((T * k, H), 7.0, dtype={"bf16": torch.bfloat16, "f16": torch.float16}[out], device="cuda")
        bs.compile_moe_blockscale_gemm2(tile_n=256, doweight_stage2=True, out_dtype=out, accumulate=False, **common)(
            pair, ref_a2, w2q, ref_a2s, w2s.view(-1), s_ids, s_e, s_w, nv, T, H, I, nblk)
        acc = torch.zeros((T, H), device="cuda")
        bs.compile_moe_blockscale_gemm2(tile_n=256, doweight_stage2=True, out_dtype="f32", accumulate=True, **common)(
            acc, ref_a2, w2q, ref_a2s, w2s.view(-1), s_ids, s_e, s_w, nv, T, H, I, nblk)
        torch.cuda.synchronize()
        assert _lib.device_status() == 0
        got[impl] = (a2, a2s, pair, acc)
    (ra, rs, rp, rc), (a, s, p, c) = got["simt"], got["tcgen05"]
    # stage 1 differs by the fast exp2/rcp of the activation (a few fp32 ulp): codes within one e4m3 step
    step = orc.e4m3_ulp_distance(a.view(FP8).cpu(), ra.view(FP8).cpu())
    assert int(step.max()) <= 1 and float((step != 0).float().mean()) < 0.01
    assert torch.allclose(s, rs, rtol=1e-5, atol=0)
    assert_close(p, rp, 2 * EPS[p.dtype], 1e-5 * float(rp.abs().max()), "stage 2 rows")
    assert_close(c, rc, 1e-5, 1e-5 * float(rc.abs().max()), "stage 2 sums")


@pytest.mark.parametrize("tile_m", [16, 32, 64, 128])
@pytest.mark.parametrize("in_dtype", ["fp8", "int8"])
def test_routed_pertoken_against_cuda_cores(in_dtype, tile_m):
    ids, tw = _routing(2)
    T, k = ids.shape
    E, H, I = len(COUNTS), 384, 256
    g = torch.Generator().manual_seed(8)
    dt = FP8 if in_dtype == "fp8" else torch.int8
    xq, sx = orc.quant_rows(torch.randn((T, H), generator=g), dt)
    w1, sw1 = orc.quant_rows(torch.randn((E * 2 * I, H), generator=g) * 0.05, dt)
    aq, sa = orc.quant_rows(torch.randn((T * k, I), generator=g), dt)
    w2, sw2 = orc.quant_rows(torch.randn((E * H, I), generator=g) * 0.05, dt)
    flat = [t.float().reshape(-1).cuda() for t in (sx, sw1, sa, sw2)]
    xq, w1, aq, w2 = (t.cuda() for t in (xq, w1, aq, w2))
    (s_ids, s_w, s_e, nv), nblk = _sort(ids, tw, E, tile_m)
    got = []
    for impl in ("simt", "tcgen05"):
        common = dict(model_dim=H, inter_dim=I, experts=E, topk=k, tile_m=tile_m, tile_k=128, in_dtype=in_dtype,
                      w_layout="plain", impl=impl)
        o1 = torch.full((T * k, I), 7.0, dtype=torch.float16, device="cuda")
        pt.compile_moe_gemm1(tile_n=128, doweight_stage1=True, out_dtype="f16", **common)(
            o1, xq, w1, flat[0], flat[1], s_ids, s_e, s_w, nv, T, I, H, nblk)
        o2 = torch.zeros((T, H), device="cuda")
        pt.compile_moe_gemm2(tile_n=256, doweight_stage2=True, out_dtype="f32", **common)(
            o2, aq, w2, flat[2], flat[3], s_ids, s_e, s_w, nv, T, H, I, nblk)
        torch.cuda.synchronize()
        assert _lib.device_status() == 0
        got.append((o1, o2))
    (r1, r2), (o1, o2) = got
    assert_close(o1, r1, 2 * EPS[torch.float16], 1e-5 * float(r1.abs().max()), "stage 1")
    assert_close(o2, r2, 1e-5, 1e-5 * float(r2.abs().max()), "stage 2")
