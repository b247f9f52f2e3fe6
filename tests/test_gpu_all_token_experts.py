"""The experts of 9 to 64 tokens without a sort, at the edges of their tiles and tables, against fp32."""
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


# token tiles of 16, 32 and 64 at both ends; one feature tile; rows off a multiple of 128 and 64; more tiles than CTAs; more experts than pairs
@pytest.mark.parametrize("T,E,k,H,F", [(9, 16, 8, 2048, 768), (16, 16, 8, 2048, 768), (17, 16, 8, 2048, 768), (61, 16, 8, 2048, 768), (64, 1, 1, 8, 64), (33, 5, 2, 328, 64),
                                       (64, 128, 8, 1000, 192), (32, 256, 3, 264, 128), (12, 40, 1, 2304, 320)])
def test_against_fp32(T, E, k, H, F):
    from miles_b200.ops import cuda as K, cuda_more

    x, w13, w2, tw, ti = _inputs(T, E, k, H, F, T + E)
    want = ref.moe_ffn(x.float(), w13.float(), w2.float(), tw, ti.long())
    y = torch.empty_like(x)
    K.C.moe_rows(x, w13, w2, ti, tw, y, 0)
    with torch.no_grad():
        through = K.moe_ffn(x, w13, w2, tw, ti)
        if cuda_more.all_token_experts(x, w13, w2, T, k):
            n0 = K.launch_count()
            assert torch.equal(y, K.moe_ffn(x, w13, w2, tw, ti)) and K.launch_count() - n0 == 2
        else:
            assert (T, E) == (64, 128)
    assert ((through.float() - want).norm() / want.norm()).item() < 8e-3
    # gate, up, the weighted activation and the output are rounded to bf16 (2^-9 relative each, 2-norm below 4 · 2^-9 together); sums in fp32
    assert ((y.float() - want).norm() / want.norm()).item() < 8e-3
    assert K.check_error_flag(x) == 0


def test_choices_that_are_none_and_other_ranks_experts():
    from miles_b200.ops import cuda as K

    x, w13, w2, tw, ti = _inputs(20, 12, 4, 256, 128, 5)
    ti[2] = -1                                                       # a token without experts
    w13[9] = float("nan")                                            # an expert of another rank
    with torch.no_grad():
        y = K.moe_ffn(x, w13[4:8], w2[4:8], tw, ti, 4)
    keep = (ti >= 4) & (ti < 8)
    want = ref.moe_ffn(x.float(), w13.float().nan_to_num(), w2.float(), tw * keep, ti.long().clamp(min=0))
    assert (y[2] == 0).all() and ((y.float() - want).norm() / want.norm()).item() < 8e-3
    with torch.no_grad():
        none = K.moe_ffn(x, w13[4:8], w2[4:8], tw, torch.full_like(ti, -1), 4)
    assert (none == 0).all() and K.check_error_flag(x) == 0
