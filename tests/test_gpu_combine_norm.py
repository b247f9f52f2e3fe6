"""The weighted sum of experts' rows, the residual stream's add and the next norm in one kernel: the bits of the kernels apart, in the op and through a model."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,E,k,H", [(64, 4, 1, 1024), (129, 16, 8, 2048), (300, 40, 9, 4096), (70, 48, 40, 1024), (65, 8, 2, 2560), (64, 8, 3, 520)])
def test_same_bits(T, E, k, H):
    from miles_b200.ops import cuda as K, cuda_more as M

    g = torch.Generator(device="cuda").manual_seed(T + E)
    rand = lambda *s: torch.randn(*s, device="cuda", generator=g)
    idx = rand(T, E).topk(k, -1).indices.int()
    idx[3] = -1                                                       # a token without experts
    rows = M.moe_max_rows(T * k, E)
    seg, tile, src, dst = K.C.moe_align(idx.view(-1), E, 0, rows, None, 128, True)
    y_perm, w, res, nw = rand(rows, H).bfloat16(), torch.rand(T, k, device="cuda", generator=g), rand(T, H).bfloat16(), (1 + 0.1 * rand(H)).bfloat16()
    x = M.Combine(y_perm, w, dst, k, res)
    with torch.no_grad():
        want, total = K.add_rmsnorm(x.value(), res, nw, 1e-6)
        got, got_total = M.combine_add_rmsnorm(x, res, nw, 1e-6)
        assert torch.equal(got, want) and torch.equal(got_total, total)
        odd = torch.cat([nw[:1], nw])[1:]                             # off a 16-byte boundary: the kernels apart
        assert torch.equal(M.combine_add_rmsnorm(x, res, odd.clone(), 1e-6)[0], want)


def test_through_a_model(monkeypatch):
    from miles_b200.models import qwen3
    from miles_b200.models.config import ModelConfig
    from miles_b200.models.qwen3 import ForwardMeta, build_model
    from miles_b200.ops import cuda_more as M

    cfg = ModelConfig(name="t", vocab_size=512, hidden_size=1024, num_layers=3, num_heads=4, num_kv_heads=2, head_dim=128, ffn_hidden_size=384, num_experts=8,
                      moe_topk=2, moe_ffn_hidden_size=192)
    model = build_model(cfg, dtype=torch.bfloat16, device="cuda", seed=3)
    T = 300
    meta = ForwardMeta(positions=torch.arange(T, device="cuda", dtype=torch.int32), cu_seqlens=torch.tensor([0, T], device="cuda", dtype=torch.int32), max_seqlen=T)
    tokens = torch.randint(0, 512, (T,), device="cuda", dtype=torch.int32)
    calls = []
    fused = M.combine_add_rmsnorm
    monkeypatch.setattr("miles_b200.ops.cuda.combine_add_rmsnorm", lambda *a: (calls.append(1), fused(*a))[1])
    with torch.no_grad():
        got = model(tokens, meta)
        assert len(calls) == 3
        handle = model.layers[1].register_forward_hook(lambda m, a, out: out)      # somebody looks on: tensors in and out of that layer
        assert torch.equal(model(tokens, meta), got) and len(calls) == 4
        handle.remove()
        monkeypatch.setattr(qwen3.Qwen3Model, "_hands_on_rows", lambda *a: False)
        assert torch.equal(model(tokens, meta), got) and len(calls) == 4
    taped = model(tokens, meta)
    assert taped.requires_grad and torch.equal(taped, got)
