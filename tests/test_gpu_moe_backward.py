"""The experts' activation in the backward pass (weighted activation, gradients of the pre-activation and of the gate weights) against 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# widths: one lane's piece, a part of a round of three pieces per lane, exactly one, more than one
@pytest.mark.parametrize("F", [8, 264, 768, 1544])
@pytest.mark.parametrize("T,k,E", [(1, 1, 1), (70, 4, 6)])
def test_moe_glu_bwd(T, k, E, F):
    from miles_b200.ops.cuda import C
    from miles_b200.ops import cuda_more as M

    g = torch.Generator(device="cuda").manual_seed(F + T)
    rand = lambda *s: torch.randn(*s, device="cuda", generator=g)
    idx = rand(T, E).topk(k, -1).indices.int()
    rows = M.moe_max_rows(T * k, E)
    seg, tile, src, dst = C.moe_align(idx.view(-1), E, 0, rows, None, 128, True)
    total = int(seg[-1])
    h1, d, w = (rand(rows, 2 * F) * 2).bfloat16(), rand(rows, F).bfloat16(), torch.rand(T * k, device="cuda", generator=g)
    act, dh1, dw = d.clone(), torch.full_like(h1, 7.0), torch.zeros(T * k, device="cuda")
    C.moe_glu_bwd(h1, act, dh1, w, src, seg, dw)

    real = src[:total] >= 0
    row_w = torch.where(real, w[src[:total].clamp(min=0).long()], torch.zeros((), device="cuda")).double()[:, None]
    gate, up = h1[:total].double().chunk(2, -1)
    e, s = d[:total].double(), torch.sigmoid(gate)
    a = gate * s * up
    close = lambda got, want: torch.allclose(got.double(), want, rtol=2 ** -8 + 1e-5, atol=1e-30)       # one rounding to bf16 of a value good to 1e-5
    assert close(act[:total], row_w * a)
    assert close(dh1[:total], row_w * torch.cat([e * up * s * (1 + gate * (1 - s)), e * gate * s], -1))
    rounded = a.float().bfloat16().double()
    want = (e * rounded).sum(-1)
    # a rounding of the activation that falls the other way: 2^-8 of single terms; sums of F of them
    bound = (e.abs() * a.abs()).sum(-1) * 2e-5 + (e * a).abs().amax(-1) * 2 ** -8
    got = torch.zeros(total, device="cuda", dtype=torch.float64)
    got[real] = dw[src[:total][real].long()].double()
    assert ((got - torch.where(real, want, torch.zeros_like(want))).abs() <= bound).all()
    assert (act[:total][~real] == 0).all() and (dh1[:total][~real] == 0).all() and (dh1[total:] == 7).all()
