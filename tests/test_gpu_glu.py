"""silu(gate) · up in the product's epilogue: the same bits as the two kernels', dense and per expert."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _two_kernels(K, x, w):
    with torch.no_grad():
        return K.swiglu(K.linear(x, w))


@pytest.mark.parametrize("M,F,H", [(7000, 1536, 256), (9000, 1032, 264), (5001, 2008, 512), (40000, 128, 64)])
def test_dense(M, F, H):
    from miles_b200.ops import cuda as K

    g = torch.Generator(device="cuda").manual_seed(M)
    x = torch.randn(M, H, device="cuda", generator=g).bfloat16()
    w = (torch.randn(2 * F, H, device="cuda", generator=g) * 3 / H ** 0.5).bfloat16()
    act = torch.full((M, F), math.nan, device="cuda", dtype=torch.bfloat16)
    assert K.C.gemm_glu(x, w, act, None)
    assert torch.equal(act, _two_kernels(K, x, w))
    with torch.no_grad():
        assert torch.equal(K.linear_swiglu(x.view(1, M, H), w)[0], act)
    assert K.check_error_flag(x) == 0


@pytest.mark.parametrize("M,F", [(64, 768), (257, 104), (3000, 16)])
def test_few_rows_or_columns(M, F):
    from miles_b200.ops import cuda as K

    x, w = torch.randn(M, 256, device="cuda").bfloat16(), torch.randn(2 * F, 256, device="cuda").bfloat16()
    with torch.no_grad():
        assert torch.equal(K.linear_swiglu(x, w), _two_kernels(K, x, w))


def test_ragged_columns_stay_refused():
    from miles_b200.ops import cuda as K

    x, w = torch.randn(9000, 256, device="cuda").bfloat16(), torch.randn(2 * 1028, 256, device="cuda").bfloat16()
    assert not K.C.gemm_glu(x, w, torch.empty(9000, 1028, device="cuda", dtype=torch.bfloat16), None)
    with torch.no_grad(), pytest.raises(RuntimeError):
        K.linear_swiglu(x, w)


@pytest.mark.parametrize("T,k,E,H,F", [(4000, 8, 16, 256, 768), (9001, 2, 4, 512, 520)])
def test_experts(T, k, E, H, F):
    from miles_b200.ops import cuda as K
    from miles_b200.ops import cuda_more as M

    g = torch.Generator(device="cuda").manual_seed(T)
    x = torch.randn(T, H, device="cuda", generator=g).bfloat16()
    w13 = (torch.randn(E, 2 * F, H, device="cuda", generator=g) / H ** 0.5).bfloat16()
    w2 = (torch.randn(E, H, F, device="cuda", generator=g) / F ** 0.5).bfloat16()
    idx = torch.rand(T, E, device="cuda", generator=g).topk(k).indices.to(torch.int32)
    w = torch.rand(T, k, device="cuda", generator=g)
    xp, seg, tile, _ = M.sort_by_expert(x, idx, E, 128)
    none, fused = M.experts_forward(xp, w13, w2, seg, tile, keep=False)
    h1, apart = M.experts_forward(xp, w13, w2, seg, tile)
    rows = int(seg[-1])
    assert none is None and h1 is not None and torch.equal(fused[:rows], apart[:rows])
    with torch.no_grad():
        inference = K.moe_ffn(x, w13, w2, w, idx)
    training = K.moe_ffn(x.requires_grad_(), w13, w2, w, idx)
    assert training.requires_grad and torch.equal(inference, training.detach())
