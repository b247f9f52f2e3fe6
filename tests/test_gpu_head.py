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


@pytest.mark.parametrize("sign", [1, -1])
def test_infinite_logits(sign):
    """A logit of −∞ has no weight and its row stays a number, one of +∞ makes its row none; other rows see nothing of either."""
    from miles_b200.ops import cuda as K

    g = torch.Generator(device="cuda").manual_seed(3)
    h, w = torch.randn(70, 64, device="cuda", generator=g).bfloat16(), torch.randn(304, 64, device="cuda", generator=g).bfloat16()
    t = torch.randint(8, 304, (70,), device="cuda", generator=g)
    h[:, 0], w[:, 0] = 0, 0
    h[3, 0], w[7, 0] = 1e30, sign * 1e30                                  # their product is beyond fp32
    h = h.requires_grad_()
    lp, _ = K.logprob_entropy(h, w, t, 1.0, False)
    z = h.detach().double() @ w.double().t()
    z[3, 7] = sign * float("inf")
    want = torch.log_softmax(z, -1).gather(1, t[:, None])[:, 0]
    assert torch.equal(torch.isnan(lp), torch.isnan(want)) and torch.isnan(lp[3]).item() == (sign > 0)
    ok = ~torch.isnan(want)
    assert (lp.double() - want)[ok].abs().max().item() < 5e-5             # as above
    lp[ok].sum().backward()
    rows = ok.clone()
    rows[3] = False                                                       # its gradient is 0 · w with an element of 1e30: left out
    assert torch.isfinite(h.grad[rows]).all() and K.check_error_flag(h) == 0


def test_backward_launches_nothing_beside_its_products():
    """Several vocabulary chunks: the targets of each are found in the kernel, not by a subtraction in front of it."""
    from miles_b200.ops import cuda as K

    h = torch.randn(70, 64, device="cuda").bfloat16().requires_grad_()
    w = torch.randn(40000, 64, device="cuda").bfloat16().requires_grad_()
    lp, _ = K.logprob_entropy(h, w, torch.arange(70, device="cuda") * 500, 1.0, False)
    total = lp.sum()
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CPU]) as prof:
        total.backward()
    assert not any(e.key in ("aten::sub", "aten::add") for e in prof.key_averages())
