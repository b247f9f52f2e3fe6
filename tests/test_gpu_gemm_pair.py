"""The two-CTA GEMM kernel (256-row tiles) at the edges of its tiles, against 64-bit products."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

PAIR = 1024         # + tile columns: the kernel is chosen whatever the rule by sizes says


def _k():
    from miles_b200.ops import cuda

    return cuda


def _check(y, ref, out_dtype=torch.bfloat16):
    # bf16 results: one rounding, 2^-9 relative; fp32 results: the order of up to 4096 fp32 sums
    limit = 2 ** -8.5 if out_dtype == torch.bfloat16 else 1e-5
    assert torch.isfinite(y).all()
    assert ((y.double() - ref).norm() / ref.norm()).item() < limit
    assert _k().check_error_flag(y) == 0


@pytest.mark.parametrize("cols", [128, 256])
@pytest.mark.parametrize("M,N,Kd", [(256, 256, 64), (129, 8, 64), (304, 264, 72), (512, 1000, 1000), (2504, 2304, 320)])
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True), (True, False)])
def test_dense_layouts(cols, M, N, Kd, a_mn, b_mn):
    K = _k()
    M = -(-M // 8) * 8 if a_mn else M
    g = torch.Generator(device="cuda").manual_seed(2)
    a = torch.randn(M, Kd, device="cuda", generator=g).bfloat16()
    b = torch.randn(N, Kd, device="cuda", generator=g).bfloat16()
    ref = a.double() @ b.double().t()
    stored_a, stored_b = (a.t().contiguous() if a_mn else a), (b.t().contiguous() if b_mn else b)
    for dtype in (torch.bfloat16, torch.float32):
        y = torch.full((M, N), math.nan, device="cuda", dtype=dtype)
        K.C.gemm(stored_a, stored_b, y, M, N, Kd, stored_a.shape[1], stored_b.shape[1], N, a_mn, b_mn, False, None, PAIR + cols)
        _check(y, ref, dtype)
    start = torch.randn(M, N, device="cuda", generator=g)
    y, bias = start.clone(), torch.randn(N, device="cuda", generator=g).bfloat16()
    K.C.gemm(stored_a, stored_b, y, M, N, Kd, stored_a.shape[1], stored_b.shape[1], N, a_mn, b_mn, True, bias, PAIR + cols)
    _check(y, ref + start.double() + bias.double(), torch.float32)


@pytest.mark.parametrize("cols", [128, 256])
@pytest.mark.parametrize("T,k,E,H,F2", [(40, 1, 8, 128, 256), (500, 2, 4, 256, 528), (777, 8, 16, 512, 1536)])
def test_grouped(cols, T, k, E, H, F2):
    """Segments end anywhere in a 256-row tile: the tile's halves may belong to two experts, or to none; some experts get no rows."""
    K = _k()
    g = torch.Generator(device="cuda").manual_seed(3)
    scores = torch.rand(T, E, device="cuda", generator=g)
    scores[:, E // 2] = 0.0
    idx = scores.topk(k).indices.to(torch.int32).contiguous()
    rows = K.moe_max_rows(T * k, E)
    seg, tile, _, _ = K.C.moe_align(idx.view(-1), E, 0, rows, None)
    x = torch.randn(rows, H, device="cuda", generator=g).bfloat16()
    w = torch.randn(E, F2, H, device="cuda", generator=g).bfloat16()
    dy = torch.randn(rows, F2, device="cuda", generator=g).bfloat16()
    s = seg.tolist()
    parts = [slice(s[e], s[e + 1]) for e in range(E)]
    y = torch.zeros(rows, F2, device="cuda", dtype=torch.bfloat16)
    K.C.gemm_grouped(x, w, y, rows, F2, H, E, tile, False, PAIR + cols)
    _check(y[:s[E]], torch.cat([x[p].double() @ w[e].double().t() for e, p in enumerate(parts)]))
    assert not y[s[E]:].any()                                     # rows behind the last segment are left alone
    dx = torch.zeros(rows, H, device="cuda", dtype=torch.bfloat16)
    K.C.gemm_grouped(dy, w, dx, rows, H, F2, E, tile, True, PAIR + cols)
    _check(dx[:s[E]], torch.cat([dy[p].double() @ w[e].double() for e, p in enumerate(parts)]))
    dw = torch.full((E, F2, H), math.nan, device="cuda", dtype=torch.bfloat16)
    K.C.gemm_grouped_wgrad(dy, x, dw, rows, F2, H, E, seg, False, PAIR + cols)
    _check(dw, torch.stack([dy[p].double().t() @ x[p].double() for p in parts]))
