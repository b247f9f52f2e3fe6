"""Layers run again in the backward pass: the values and gradients of `torch.utils.checkpoint`, and its place where the conditions do not hold."""
import pytest
import torch

from miles_b200.models import qwen3
from miles_b200.models.config import ModelConfig
from miles_b200.models.qwen3 import ForwardMeta, build_model

pytestmark = pytest.mark.gpu


def _model(moe: bool, **kw):
    cfg = ModelConfig(name="t", vocab_size=512, hidden_size=256, num_layers=3, num_heads=4, num_kv_heads=2, head_dim=128, ffn_hidden_size=384,
                      num_experts=8 if moe else 0, moe_topk=2 if moe else 0, moe_ffn_hidden_size=192 if moe else 0, **kw)
    model = build_model(cfg, dtype=torch.bfloat16, device="cuda", seed=3)
    with torch.no_grad():
        model.embed.mul_(50.0)
    return model


def _meta(lengths, recompute=True):
    cu = [0]
    for n in lengths:
        cu.append(cu[-1] + n)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    return ForwardMeta(positions=torch.cat([torch.arange(n, device="cuda") for n in lengths]).int(), cu_seqlens=i32(cu), max_seqlen=max(lengths), recompute=recompute)


def _step(model, tokens, meta, times=1):
    model.zero_grad(set_to_none=True)
    logp, _ = model.log_probs(model(tokens, meta), tokens.long(), 1.0)
    loss = (logp * torch.linspace(-1, 1, logp.numel(), device="cuda")).sum()
    for i in range(times):
        loss.backward(retain_graph=i + 1 < times)
    return logp.detach(), {n: p.grad for n, p in model.named_parameters()}


@pytest.mark.parametrize("moe", [False, True])
@pytest.mark.parametrize("lengths", [[129], [300, 7, 420]])
@pytest.mark.parametrize("freeze", [None, "embed", "attn", "ln"])
def test_same_as_checkpoint(monkeypatch, moe, lengths, freeze):
    model, tokens = _model(moe), torch.randint(0, 512, (sum(lengths),), device="cuda", dtype=torch.int32)
    for n, p in model.named_parameters():
        if freeze is not None and freeze in n:
            p.requires_grad_(False)
    calls = []
    apply = qwen3._RunAgain.apply
    monkeypatch.setattr(qwen3._RunAgain, "apply", lambda *a: (calls.append(1), apply(*a))[1])
    logp, grads = _step(model, tokens, _meta(lengths))
    assert len(calls) == 3
    monkeypatch.setattr(qwen3, "_runs_again", lambda *a: False)
    want, want_grads = _step(model, tokens, _meta(lengths))
    assert len(calls) == 3 and torch.equal(logp, want)
    plain, plain_grads = _step(model, tokens, _meta(lengths, recompute=False))
    assert torch.equal(logp, plain)
    for n, g in want_grads.items():
        assert (g is None) == (grads[n] is None)
        if g is not None:
            assert torch.equal(grads[n], g), n
            assert torch.equal(plain_grads[n], g), n


def test_backward_twice_adds_up():
    model, tokens = _model(True), torch.randint(0, 512, (200,), device="cuda", dtype=torch.int32)
    _, once = _step(model, tokens, _meta([200]))
    once = {n: g.clone() for n, g in once.items()}
    _, twice = _step(model, tokens, _meta([200]), times=2)
    for n, g in once.items():
        assert torch.equal(twice[n], g + g), n


def test_where_it_does_not_apply():
    model = _model(True)
    x, meta, layer = torch.randn(256, 256, device="cuda").bfloat16(), _meta([256]), model.layers[0]
    assert qwen3._runs_again(layer, x, meta)
    assert not qwen3._runs_again(layer, x[:64], _meta([64]))                          # rows that decode kernels take without gradients
    assert not qwen3._runs_again(layer, x.float(), meta)
    handle = layer.mlp.register_forward_hook(lambda *a: None)
    assert not qwen3._runs_again(layer, x, meta)
    handle.remove()
    meta.record_topk = []
    assert not qwen3._runs_again(layer, x, meta)
