"""Recorded routing choices: weights and gradients from the current scores, against the plain statement in 64 bits."""
import numpy as np
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


@pytest.mark.parametrize("E,k", [(16, 8), (128, 8), (40, 1), (256, 32)])
@pytest.mark.parametrize("bad", ["past the last", "far past", "partly negative"])
def test_invalid_records_raise_the_error_flag(E, k, bad):
    """Without gradients too, and with nothing read or written out of range behind the router."""
    from miles_b200.ops import cuda as K

    if bad == "partly negative" and k == 1:
        pytest.skip("one choice: a negative one is a row without a record")
    g = torch.Generator(device="cuda").manual_seed(E)
    logits = torch.randn(65, E, device="cuda", generator=g)
    idx = torch.rand(65, E, device="cuda", generator=g).topk(k).indices.to(torch.int32)
    with torch.no_grad():
        w0, i0, _ = K.router_replay(logits, idx)
        assert K.check_error_flag(logits) == 0
        wrong = idx.clone()
        wrong[40, k - 1] = {"past the last": E, "far past": 2 ** 31 - 1, "partly negative": -1}[bad]
        w, i, _ = K.router_replay(logits, wrong)
        try:
            assert K.check_error_flag(logits) == 72
        finally:
            K.C.error_flag(logits).zero_()
    assert w[40, k - 1] == 0 and ((i >= 0) & (i < E)).all()
    others = torch.arange(65, device="cuda") != 40
    assert torch.equal(w[others], w0[others]) and torch.equal(i[others], i0[others])


def test_records_on_the_host_are_refused():
    from miles_b200.ops import cuda as K

    logits = torch.randn(4, 16, device="cuda")
    with pytest.raises(RuntimeError, match="logits on cuda"):
        K.router_replay(logits, torch.zeros(4, 2, dtype=torch.int32))


def test_training_refuses_invalid_records():
    from miles_b200.args import parse_args
    from miles_b200.models.config import ModelConfig
    from miles_b200.ops import cuda as K
    from miles_b200.train.actor import TrainActor
    from miles_b200.train.data import convert_samples_to_train_data
    from miles_b200.types import Sample, Status

    cfg = ModelConfig(name="tiny-moe", vocab_size=512, hidden_size=256, num_layers=1, num_heads=2, num_kv_heads=1, head_dim=128, ffn_hidden_size=256,
                      num_experts=8, moe_topk=2, moe_ffn_hidden_size=128)
    args = parse_args("--rollout-batch-size 1 --n-samples-per-prompt 2 --rollout-max-response-len 8 --num-rollout 1 --rm-type even_fraction --lr 1e-5 "
                      "--colocate --use-rollout-routing-replay".split())
    actor = TrainActor(args, device="cuda:0")
    actor.init(cfg)
    before = {n: p.detach().clone() for n, p in actor.model.named_parameters()}

    def data(worst):
        group = []
        for j in range(2):
            s = Sample(group_index=0, index=j, tokens=list(range(3, 11)))
            s.append_response(list(range(20 + j, 28 + j)), [-6.0] * 8)
            routed = np.tile(np.array([1, 2], dtype=np.int32), (15, 1, 1))
            routed[3, 0, 1] = worst
            s.rollout_routed_experts, s.status, s.reward = routed, Status.TRUNCATED, float(j)
            group.append(s)
        return convert_samples_to_train_data(args, [group])

    try:
        with pytest.raises(RuntimeError, match="72"):
            actor.train(0, data(8))
    finally:
        K.C.error_flag(torch.empty(0, device="cuda")).zero_()
    assert all(torch.equal(p, before[n]) for n, p in actor.model.named_parameters())
    assert actor.train(0, data(3))["train/grad_norm"] > 0
