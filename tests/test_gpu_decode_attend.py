"""Norm, rotation, cache write and attention of a decode step in one launch: the cache of the kernels it stands for, attention against 64-bit softmax."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _inputs(lens, hq, hkv, page, norm, seed=3):
    g = torch.Generator(device="cuda").manual_seed(seed)
    rand = lambda *s: torch.randn(*s, device="cuda", generator=g)
    pages = [max(1, -(-n // page)) for n in lens]
    total = sum(pages) + 1
    kc, vc = rand(total, page, hkv, 128).bfloat16(), rand(total, page, hkv, 128).bfloat16()
    order = torch.randperm(total - 1, generator=g, device="cuda").to(torch.int32)
    table = torch.zeros(len(lens), max(pages) + 1, dtype=torch.int32, device="cuda")
    slots, at = [], 0
    for b, n in enumerate(pages):
        table[b, :n] = order[at:at + n]
        at += n
        last = max(lens[b] - 1, 0)
        slots.append(int(table[b, last // page]) * page + last % page)
        kc[table[b, n - 1], last % page:] = math.nan           # the new token's row, and what lies behind it
        vc[table[b, n - 1], last % page:] = math.nan
    qkv = rand(len(lens), (hq + 2 * hkv) * 128 + 8).bfloat16()
    q, k, v, _ = qkv.split([hq * 128, hkv * 128, hkv * 128, 8], dim=-1)
    q, k, v = q.view(-1, hq, 128), k.view(-1, hkv, 128), v.view(-1, hkv, 128)
    w = [(1 + 0.2 * rand(128)).bfloat16() for _ in range(2)] if norm else [None, None]
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device="cuda")
    return [q, k, v, *w, i32([max(n - 1, 0) for n in lens]), 1e6, 1e-6, kc, vc, torch.tensor(slots, device="cuda"), table, i32(lens)]


def _want(args):
    """The cache after the step, and attention over it in 64 bits."""
    from miles_b200.ops import cuda as K

    q, k, v, qw, kw, positions, theta, eps, kc, vc, slots, table, lens = args
    kc, vc = kc.clone(), vc.clone()
    qr, _ = K.qk_norm_rope_cache(q, k, v, qw, kw, positions, theta, eps, kc, vc, slots)
    out = torch.zeros(qr.shape, dtype=torch.float64, device=q.device)
    group = qr.shape[1] // kc.shape[2]
    for b, n in enumerate(lens.tolist()):
        if n:
            pages = table[b, :-(-n // kc.shape[1])].long()
            kk, vv = (x[pages].flatten(0, 1)[:n].double().transpose(0, 1).repeat_interleave(group, 0) for x in (kc, vc))
            p = torch.softmax(qr[b].double()[:, None] @ kk.transpose(1, 2) / math.sqrt(128), -1)
            out[b] = (p @ vv)[:, 0]
    return kc, vc, out


def _check(args, split):
    from miles_b200.ops import cuda as K

    kc, vc, ref = _want(args)
    args[8:10] = [args[8].clone(), args[9].clone()]
    out = torch.full(ref.shape, 9.0, device="cuda").bfloat16()
    q, k, v, qw, kw, positions, theta, eps, kc2, vc2, slots, table, lens = args
    K.C.decode_attend(q, k, v, qw, kw, positions, theta, eps, kc2, vc2, slots, table, lens, out, 1 / math.sqrt(128), split, K.C.error_flag(q))
    bits = lambda t: t.view(torch.int16)
    assert torch.equal(bits(kc2), bits(kc)) and torch.equal(bits(vc2), bits(vc))
    # weights and outputs are rounded to bf16 once each: 2^-9 relative and independent
    assert torch.isfinite(out).all() and (out.double() - ref).norm().item() <= 2 ** -8 * ref.norm().item() + 1e-30
    assert K.check_error_flag(q) == 0


@pytest.mark.parametrize("split", [1, 3, 8, 16])
@pytest.mark.parametrize("hq,hkv,norm", [(32, 4, True), (8, 8, False), (4, 2, True)])
@pytest.mark.parametrize("lens,page", [([1], 64), ([1, 15, 16, 17, 64, 65, 0, 700], 64), ([1801], 64), ([9000, 33], 16), ([300, 129], 128)])
def test_against_the_kernels_apart(split, hq, hkv, norm, lens, page):
    _check(_inputs(lens, hq, hkv, page, norm), split)


def test_new_tokens_that_are_not_cached_or_elsewhere():
    args = _inputs([40, 65, 130], 16, 2, 64, True)
    args[8].nan_to_num_(0.5), args[9].nan_to_num_(0.5)
    args[10][0] = -1                                         # not cached: attention sees what the cache holds
    args[10][2] = int(args[11][2, 0]) * 64 + 5               # in the middle of the sequence
    _check(args, 8)


def test_through_the_rule():
    from miles_b200.ops import cuda as K, cuda_more

    args = _inputs([700, 33], 32, 4, 64, True)
    _, _, ref = _want(args)
    assert K.decode_attention(*args) is None                 # gradients may be recorded
    with torch.no_grad():
        graph = torch.cuda.CUDAGraph()
        first = K.decode_attention(*args)
        with torch.cuda.graph(graph):                        # two in a row: the second starts while the first still runs
            K.decode_attention(*args)
            again = K.decode_attention(*args)
        graph.replay()
        assert torch.equal(first, again) and (first.double() - ref).norm() <= 2 ** -8 * ref.norm()
        wide = _inputs([5] * (cuda_more._ATTEND_SEGMENTS // 4 + 1), 32, 4, 64, True)
        assert K.decode_attention(*wide) is None
        assert K.decode_attention(*_inputs([5], 16, 1, 64, True)) is None          # 16 heads to a KV head
        args[5] = args[5].long()
        assert K.decode_attention(*args) is None
