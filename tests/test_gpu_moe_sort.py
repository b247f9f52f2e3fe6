"""Sorting (token, choice) pairs by expert: exact, in order, for one CTA and for a cluster."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,E,offset,pad", [(1, 1, 0, 128), (31, 16, 0, 16), (488, 16, 0, 32), (4096, 128, 0, 128), (4097, 16, 0, 128), (60001, 256, 0, 128),
                                            (100003, 16, 4, 128), (5000, 3, -2, 16)])
def test_moe_align(n, E, offset, pad):
    from miles_b200.ops import cuda as K
    from miles_b200.ops import cuda_more as M

    g = torch.Generator(device="cuda").manual_seed(n)
    idx = torch.randint(-1, E + 6, (n,), device="cuda", generator=g).to(torch.int32)      # some belong to other ranks, some to nobody
    rows = M.moe_max_rows(n, E) if pad == 128 else M.moe_max_rows_pad(n, E, pad)
    for count in (None, torch.tensor([n // 2 + 1], dtype=torch.int32, device="cuda")):
        m = n if count is None else n // 2 + 1
        seg, tile, src, dst = K.C.moe_align(idx, E, offset, rows, count, pad)
        local = idx[:m].long() - offset
        inside = (local >= 0) & (local < E)
        counts = torch.bincount(local[inside], minlength=E)
        ends = (-(-counts // pad) * pad).cumsum(0)
        starts = torch.cat([ends.new_zeros(1), ends])
        assert torch.equal(seg.long(), starts)
        order = torch.arange(m, device="cuda")[inside][torch.sort(local[inside], stable=True).indices]
        want = torch.full((int(starts[-1]),), -1, device="cuda", dtype=torch.long)
        first = counts.cumsum(0) - counts
        e = local[order]
        at = starts[e] + torch.arange(len(order), device="cuda") - first[e]
        want[at] = order
        assert torch.equal(src[:len(want)].long(), want)
        back = torch.full((m,), -1, device="cuda", dtype=torch.long)
        back[order] = at
        assert torch.equal(dst[:m].long(), back)
        used = torch.arange(rows // pad, device="cuda") * pad
        owner = torch.searchsorted(starts[1:], used, right=True)
        assert torch.equal(tile.long(), torch.where(used < starts[-1], owner, torch.full_like(owner, -1)))


@pytest.mark.parametrize("n,E,offset,pad", [(1, 1, 0, 128), (31, 16, 0, 16), (488, 16, 2, 32), (4096, 32, 0, 128), (4097, 32, 0, 128), (2049, 33, 0, 16)])
def test_any_order_within_an_expert(n, E, offset, pad):
    """Inference may have a segment's rows in any order: the same segments, the same pairs in each."""
    from miles_b200.ops import cuda as K
    from miles_b200.ops import cuda_more as M

    g = torch.Generator(device="cuda").manual_seed(n)
    idx = torch.randint(-1, E + 6, (n,), device="cuda", generator=g).to(torch.int32)
    rows = M.moe_max_rows_pad(n, E, pad)
    for count in (None, torch.tensor([n // 2 + 1], dtype=torch.int32, device="cuda")):
        m = n if count is None else n // 2 + 1
        seg, tile, src, dst = K.C.moe_align(idx, E, offset, rows, count, pad)
        seg2, tile2, src2, dst2 = K.C.moe_align(idx, E, offset, rows, count, pad, False)
        assert torch.equal(seg, seg2) and torch.equal(tile, tile2)
        for e in range(E):
            a, b = int(seg[e]), int(seg[e + 1])
            assert torch.equal(src[a:b].sort().values, src2[a:b].sort().values)
        there = (dst2[:m] >= 0).nonzero()[:, 0]
        assert torch.equal(dst[:m] >= 0, dst2[:m] >= 0) and torch.equal(src2[dst2[:m][there].long()].long(), there)


@pytest.mark.parametrize("T", [9, 61, 300])
def test_order_does_not_change_the_sums(T):
    """A row's products and a token's sum over its choices are the same wherever the row is."""
    from miles_b200.ops import cuda as K

    g = torch.Generator(device="cuda").manual_seed(T)
    rand = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()
    x, w13, w2 = rand(T, 512), rand(16, 256, 512) * 0.05, rand(16, 512, 128) * 0.05
    idx = torch.rand(T, 16, device="cuda", generator=g).topk(4).indices.to(torch.int32)
    w = torch.rand(T, 4, device="cuda", generator=g)
    with torch.no_grad():
        outs = [K.moe_ffn(x, w13, w2, w, idx) for _ in range(4)]
    assert all(torch.equal(o, outs[0]) for o in outs)
