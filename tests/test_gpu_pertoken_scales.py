"""16-bit operands: each of the two scale pointers may be null by itself and then stands for ones, whichever kernel
a launch takes (C ABI: the Python launchers pass none).

Outputs are the fp32 ones of both stages, compared with float64 on the same operands: bf16 products are exact in fp32,
and sums of 1152 of them in another order differ by well under 1e-5 of the largest."""
import pytest
import torch

from flydsl_b200 import _lib
from flydsl_b200.kernels.moe_sorting_kernel import moe_sorting_flydsl
from tests.gpu_common import assert_close

pytestmark = pytest.mark.gpu
E, K, N = 4, 1152, 256
# route -> tokens, row block: few tiles of long K share K in a cluster; 128-row blocks do not; 120 rows per expert and
# more run on CTA pairs
ROUTES = {"split": (5, 16), "one-cta": (40, 128), "pair": (300, 64)}


@pytest.mark.parametrize("scales", ["both", "x", "w", "none"])
@pytest.mark.parametrize("route", sorted(ROUTES))
def test_scale_pointers_are_independent(route, scales):
    T, U = ROUTES[route]
    k = 2
    g = torch.Generator().manual_seed(21)
    ids = torch.stack([torch.randperm(E, generator=g)[:k] for _ in range(T)]).to(torch.int32).cuda()
    tw = (torch.rand((T, k), generator=g) + 0.1).cuda()
    blocks = (T * k + E * U - k + U - 1) // U
    rows = blocks * U
    i32 = dict(dtype=torch.int32, device="cuda")
    s_ids, s_e, nv = torch.empty(rows, **i32), torch.empty(blocks, **i32), torch.empty(2, **i32)
    s_w = torch.empty(rows, device="cuda")
    moe_sorting_flydsl(ids, tw, s_ids, s_w, s_e, nv, None, E, U)
    r = torch.arange(rows, device="cuda")
    tok, slot = (s_ids & 0xFFFFFF).long(), (s_ids >> 24).long()
    real = (r < nv[0]) & (tok < T)

    def rnd(*shape, std=1.0):
        return (torch.randn(shape, generator=g) * std).to(torch.bfloat16).cuda()

    def scale(n):
        return (torch.rand(n, generator=g) + 0.5).cuda()

    x, w1, a2, w2 = rnd(T, K), rnd(E, 2 * N, K, std=0.05), rnd(T * k, K), rnd(E, N, K, std=0.05)
    sx, sw1, sa, sw2 = scale(T), scale(E * 2 * N), scale(T * k), scale(E * N)
    xs, a2s = torch.zeros((rows, K), dtype=x.dtype, device="cuda"), torch.zeros((rows, K), dtype=x.dtype, device="cuda")
    xs[real] = x[tok[real]]
    a2s[real] = a2[tok[real] * k + slot[real]]
    with_x, with_w = scales in ("both", "x"), scales in ("both", "w")
    lib, p, st = _lib.load(), _lib.ptr, torch.cuda.current_stream().cuda_stream
    out1 = torch.zeros((T * k, 2 * N), device="cuda")
    _lib.check(lib.flymoe_moe_gemm1_pertoken(
        p(out1), p(xs), p(sx) if with_x else None, p(w1), p(sw1) if with_w else None, p(s_ids), p(s_e), p(s_w), p(nv), T, N, K,
        blocks, E, k, U, 0, _lib.BF16, _lib.F32, _lib.ROWS_SORTED, _lib.ROWS_BY_TOKEN, _lib.ROWS_BY_PAIR,
        _lib.IMPL_TCGEN05, st), "gemm1")
    out2 = torch.zeros((T, N), device="cuda")
    _lib.check(lib.flymoe_moe_gemm2_pertoken(
        p(out2), p(a2s), p(sa) if with_x else None, p(w2), p(sw2) if with_w else None, p(s_ids), p(s_e), p(s_w), p(nv), T, N, K,
        blocks, E, k, U, 0, _lib.BF16, _lib.F32, 1, _lib.ROWS_SORTED, _lib.ROWS_BY_PAIR, _lib.IMPL_TCGEN05, st), "gemm2")
    torch.cuda.synchronize()
    assert _lib.device_status() == 0

    def ref(a, sa_, w, sw_, rows_of):                       # [T*k, columns] in float64
        n = w.shape[1]
        y = torch.empty((T * k, n), dtype=torch.float64, device="cuda")
        for e in range(E):
            sel = torch.nonzero(ids.view(-1) == e).view(-1)
            f = a[rows_of(sel)].double() @ w[e].double().t()
            if with_x:
                f = f * sa_[rows_of(sel)].double()[:, None]
            y[sel] = f * sw_.view(E, n)[e].double() if with_w else f
        return y

    r1 = ref(x, sx, w1, sw1, lambda s: s // k)
    assert_close(out1, r1, 1e-5, 1e-5 * float(r1.abs().max()), f"stage 1 {route} {scales}")
    r2 = ref(a2, sa, w2, sw2, lambda s: s).view(T, k, N).sum(1)
    assert_close(out2, r2, 1e-5, 1e-5 * float(r2.abs().max()), f"stage 2 {route} {scales}")
