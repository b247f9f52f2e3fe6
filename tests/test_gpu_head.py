"""The vocabulary head whose statistics and gradients come out of the product's epilogue, against 64-bit softmax."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("R,H,V", [(65, 64, 1000), (128, 72, 128), (129, 256, 8), (300, 1024, 16384 + 136), (257, 512, 40000)])
@pytest.mark.parametrize("temperature,with_entropy", [(1.0, True), (0.7, False)])
def test_logprob_entropy_and_gradients(R, H, V, temperature, with_entropy):
    from miles_b200.ops import cuda as K
    from miles_b200.ops import cuda_more

    assert cuda_more._head_in_place(R, torch.empty(R, H, dtype=torch.bfloat16), torch.empty(V, H, dtype=torch.bfloat16))
    g = torch.Generator(device="cuda").manual_seed(R)
    h = torch.randn(R, H, device="cuda", generator=g).bfloat16().requires_grad_()
    w = (torch.randn(V, H, device="cuda", generator=g) * 3 / H ** 0.5).bfloat16().requires_grad_()
    t = torch.randint(0, V, (R,), device="cuda", generator=g)
    t[0], t[1] = 0, V - 1
    g_lp, g_ent = torch.randn(R, device="cuda", generator=g), torch.randn(R, device="cuda", generator=g)
    lp, ent = K.logprob_entropy(h, w, t, temperature, with_entropy)
    hd, wd = h.detach().double().requires_grad_(), w.detach().double().requires_grad_()
    logp = torch.log_softmax(hd @ wd.t() / temperature, -1)
    want_lp, want_ent = logp.gather(1, t[:, None])[:, 0], -(logp.exp() * logp).sum(-1)
    # fp32 logits of magnitude ~10 summed over H products: 1e-5 absolute and relative covers the order of the sums
    assert (lp.double() - want_lp).abs().max().item() < 5e-5
    loss, want = (lp * g_lp).sum(), (want_lp * g_lp.double()).sum()
    if with_entropy:
        assert (ent.double() - want_ent).abs().max().item() < 5e-5
        loss, want = loss + (ent * g_ent).sum(), want + (want_ent * g_ent.double()).sum()
    loss.backward()
    want.backward()
    for a, b in ((h.grad, hd.grad), (w.grad, wd.grad)):
        # d logits and the results are rounded to bf16 (2^-9 relative each)
        assert ((a.double() - b).norm() / b.norm()).item() < 2 ** -7.5
    assert K.check_error_flag(h) == 0


def test_targets_outside_the_shard_and_no_finite_logit():
    from miles_b200.ops import cuda as K

    h = torch.randn(70, 64, device="cuda").bfloat16()
    w = torch.randn(300, 64, device="cuda").bfloat16()
    t = torch.full((70,), -5, device="cuda")
    lp, _, lse = K.logprob_entropy(h, w, t, 1.0, False, 0, return_lse=True)
    assert torch.allclose(lp, -lse)                                       # as before: no target here, its logit counts 0
    h[3] = float("nan")
    lp, ent = K.logprob_entropy(h, w, t, 1.0, True)
    assert torch.isnan(lp[3]) and torch.isnan(ent[3]) and torch.isfinite(lp[4:]).all()
