"""Tile edges of the tcgen05 attention kernels (head_dim 128) against 64-bit softmax."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _softmax64(q, k, v, cu_q, cu_k, causal):
    """Outputs [T, Hq, D] and log-sum-exp [Hq, T]; the queries are the last positions of their keys."""
    out, lse = [], []
    group = q.shape[1] // k.shape[1]
    for a, e, ka, ke in zip(cu_q, cu_q[1:], cu_k, cu_k[1:]):
        qq = q[a:e].double().transpose(0, 1)
        kk, vv = (x[ka:ke].double().transpose(0, 1).repeat_interleave(group, 0) for x in (k, v))
        s = qq @ kk.transpose(1, 2) / math.sqrt(q.shape[2])
        if causal:
            hidden = torch.arange(ke - ka, device=q.device)[None] > torch.arange(ke - ka - (e - a), ke - ka, device=q.device)[:, None]
            s = s.masked_fill(hidden, -math.inf)
        out.append((torch.softmax(s, -1) @ vv).transpose(0, 1))
        lse.append(torch.logsumexp(s, -1))
    return torch.cat(out), torch.cat(lse, 1)


def _offsets(lens):
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    return cu


@pytest.mark.parametrize("heads", [(2, 1), (32, 4), (6, 2), (4, 4)])          # pairs of heads; an odd group and single heads: pairs of query tiles
@pytest.mark.parametrize("lens,key_lens,causal", [
    ([1], None, True), ([128], None, True), ([129], None, False), ([255, 256, 257, 0, 700], None, True),
    ([64] * 40 + [500], None, True),                                          # more sequences than a warp has lanes
    ([97, 300, 1, 129], [1000, 300, 777, 2500], True), ([97, 300], [1000, 640], False)])
def test_flash_forward_tiles(heads, lens, key_lens, causal):
    from miles_b200.ops import cuda as K

    g = torch.Generator(device="cuda").manual_seed(5)
    hq, hkv = heads
    cu_q, cu_k = _offsets(lens), _offsets(key_lens or lens)
    q = torch.randn(cu_q[-1], hq, 128, device="cuda", generator=g).bfloat16()
    k, v = (torch.randn(cu_k[-1], hkv, 128, device="cuda", generator=g).bfloat16() for _ in range(2))
    o = torch.full_like(q, math.nan)
    lse = torch.full((hq, cu_q[-1]), math.nan, device="cuda")
    i32 = dict(dtype=torch.int32, device="cuda")
    K.C.flash_fwd_tc(q, k, v, o, lse, torch.tensor(cu_q, **i32), max(lens), 1 / math.sqrt(128), causal, K.C.error_flag(q),
                     torch.tensor(cu_k, **i32) if key_lens else None)
    ref, ref_lse = _softmax64(q, k, v, cu_q, cu_k, causal)
    # weights and outputs are rounded to bf16 once each: 2^-9 relative, independent, so 2^-8 bounds the norm; the sums are fp32
    assert ((o.double() - ref).norm() / ref.norm()).item() < 2 ** -8
    assert (lse.double() - ref_lse).abs().max().item() < 1e-4
    assert K.check_error_flag(q) == 0


@pytest.mark.parametrize("heads", [(8, 1), (4, 4), (6, 2)])
@pytest.mark.parametrize("lens,causal", [([1], True), ([127, 128, 129], True), ([255, 257, 0, 64, 700], True), ([300, 1, 129], False), ([64] * 40 + [260], True)])
def test_flash_backward_tiles(heads, lens, causal):
    from miles_b200.ops import cuda_more as M
    from miles_b200.ops import cuda as K

    g = torch.Generator(device="cuda").manual_seed(6)
    hq, hkv = heads
    cu = _offsets(lens)
    q, k, v, do = (torch.randn(cu[-1], n, 128, device="cuda", generator=g).bfloat16() for n in (hq, hkv, hkv, hq))
    leaves = [t.clone().requires_grad_() for t in (q, k, v)]
    o = M._FlashAttn.apply(*leaves, torch.tensor(cu, dtype=torch.int32, device="cuda"), max(lens), causal)
    o.backward(do)
    exact = [t.double().requires_grad_() for t in (q, k, v)]
    _softmax64(*exact, cu, cu, causal)[0].backward(do.double())
    for a, b in zip(leaves, exact):
        # P and dS are rounded to bf16 before their products and the gradients after them, Δ comes from a rounded output: 2^-9 each
        assert (a.grad.double() - b.grad).norm().item() <= 2 ** -6.5 * b.grad.norm().item() + 1e-3 * (b.numel() ** 0.5 if max(lens) == 1 else 0.0)
        assert torch.isfinite(a.grad).all()
    assert K.check_error_flag(q) == 0
