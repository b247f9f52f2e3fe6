"""Recorded routing choices: weights and gradients from the current scores, against the plain statement in 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,E,k", [(1, 8, 2), (700, 16, 8), (333, 128, 8), (65, 256, 32), (9, 40, 1)])
@pytest.mark.parametrize("normalize", [True, False])
def test_router_replay(T, E, k, normalize):
    from miles_b200.ops import cuda as K
    from miles_b200.ops import reference as ref

    g = torch.Generator(device="cuda").manual_seed(T)
    logits = torch.randn(T, E, device="cuda", generator=g).requires_grad_()
    records = torch.rand(T, 3, E, device="cuda", generator=g).topk(k).indices.to(torch.int32)     # [T, layers, k]
    records[T // 2] = -1                                                                          # a token without a record
    idx = records[:, 1]
    w, chosen, probs = K.router_replay(logits, idx, normalize)
    exact = logits.detach().double().requires_grad_()
    p = torch.softmax(exact, -1)
    want_idx = torch.where((idx < 0).all(-1)[:, None], ref.router_topk(logits.detach(), k, normalize)[1], idx)
    want = p.gather(1, want_idx.long())
    if normalize:
        want = want / want.sum(-1, keepdim=True)
    assert torch.equal(chosen, want_idx)
    assert (w.double() - want).abs().max().item() < 1e-6 and (probs.double() - p).abs().max().item() < 1e-6
    gw = torch.randn(T, k, device="cuda", generator=g)
    (w * gw).sum().backward()
    (want * gw.double()).sum().backward()
    assert (logits.grad.double() - exact.grad).abs().max().item() < 1e-5
