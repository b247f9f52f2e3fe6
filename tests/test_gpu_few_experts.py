"""The experts of a handful of tokens (two matrix-vector kernels) at the edges of their items, pieces and tables, against fp32."""
import pytest
import torch

from miles_b200.ops import reference as ref

pytestmark = pytest.mark.gpu


def _inputs(T, E, k, H, F, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    rand = lambda *s: torch.randn(*s, device="cuda", generator=g)
    x, w13, w2 = rand(T, H).bfloat16(), (rand(E, 2 * F, H) / H ** 0.5).bfloat16(), (rand(E, H, F) / F ** 0.5).bfloat16()
    tw, ti = rand(T, E).softmax(-1).topk(k, dim=-1)
    return x, w13, w2, tw / tw.sum(-1, keepdim=True), ti.int()


# pieces of 1024 columns and a rest, widths off a multiple of 64, more and fewer experts than pairs, shares that end inside an expert, one CTA's worth
@pytest.mark.parametrize("T,E,k,H,F", [(1, 1, 1, 32, 32), (1, 16, 8, 2048, 768), (7, 16, 8, 2048, 768), (8, 256, 8, 1056, 1056), (8, 8, 8, 4096, 96), (2, 40, 32, 96, 160),
                                       (5, 3, 2, 8192, 64), (8, 64, 6, 2080, 1376)])
def test_against_fp32(T, E, k, H, F):
    from miles_b200.ops import cuda as K, cuda_more

    x, w13, w2, tw, ti = _inputs(T, E, k, H, F, T + E)
    want = ref.moe_ffn(x.float(), w13.float(), w2.float(), tw, ti.long())
    with torch.no_grad():
        assert cuda_more.few_token_experts(x, w13, T, k)
        y = K.moe_ffn(x, w13, w2, tw, ti)
    # operands and sums as in fp32; gate, up, the weighted activation and the output are rounded to bf16 (2^-9 relative each, 2-norm below 4 · 2^-9 together)
    assert ((y.float() - want).norm() / want.norm()).item() < 8e-3
    assert K.check_error_flag(x) == 0


def test_choices_that_are_none_and_other_ranks_experts():
    from miles_b200.ops import cuda as K

    x, w13, w2, tw, ti = _inputs(6, 12, 4, 256, 96, 5)
    ti[2] = -1                                                       # a token without experts
    ti[4, 1:] = torch.tensor([3, 9, 11], device="cuda")
    with torch.no_grad():
        y = K.moe_ffn(x, w13[4:8], w2[4:8], tw, ti, 4)
    keep = (ti >= 4) & (ti < 8)
    want = ref.moe_ffn(x.float(), w13.float(), w2.float(), tw * keep, ti.long().clamp(min=0))
    assert (y[2] == 0).all() and ((y.float() - want).norm() / want.norm()).item() < 8e-3
    with torch.no_grad():
        none = K.moe_ffn(x, w13[4:8], w2[4:8], tw, torch.full_like(ti, -1), 4)
    assert (none == 0).all() and K.check_error_flag(x) == 0
