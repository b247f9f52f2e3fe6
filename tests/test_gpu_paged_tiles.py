"""Paged decode attention with an even share of all key tiles per CTA, against 64-bit softmax."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _inputs(lens, hq, hkv, d, page):
    g = torch.Generator(device="cuda").manual_seed(9)
    pages = [max(1, -(-n // page)) for n in lens]
    total = sum(pages) + 2
    k, v = (torch.randn(total, page, hkv, d, device="cuda", generator=g).bfloat16() for _ in range(2))
    order = torch.randperm(total, generator=g, device="cuda").to(torch.int32)
    table = torch.zeros(len(lens), max(pages) + 1, dtype=torch.int32, device="cuda")
    at = 0
    for b, n in enumerate(pages):
        table[b, :n] = order[at:at + n]
        at += n
        if lens[b] % page:                        # what a page holds behind its sequence's end may be no number
            k[table[b, n - 1], lens[b] % page:] = math.nan
            v[table[b, n - 1], lens[b] % page:] = math.nan
    q = torch.randn(len(lens), hq, d, device="cuda", generator=g).bfloat16()
    return q, k, v, table, torch.tensor(lens, dtype=torch.int32, device="cuda")


def _softmax64(q, k, v, table, lens):
    out = torch.zeros(q.shape, dtype=torch.float64, device=q.device)
    group = q.shape[1] // k.shape[2]
    for b, n in enumerate(lens.tolist()):
        if n:
            pages = table[b, :-(-n // k.shape[1])].long()
            kk, vv = (x[pages].flatten(0, 1)[:n].double().transpose(0, 1).repeat_interleave(group, 0) for x in (k, v))
            p = torch.softmax(q[b].double()[:, None] @ kk.transpose(1, 2) / math.sqrt(q.shape[2]), -1)
            out[b] = (p @ vv)[:, 0]
    return out


@pytest.mark.parametrize("hq,hkv,d", [(32, 4, 128), (16, 8, 128), (4, 4, 128), (8, 2, 64)])
@pytest.mark.parametrize("lens,page", [([1], 64), ([1, 63, 64, 65, 700, 0, 128], 64), ([0, 0, 5, 0], 64), ([6000, 1, 1, 3], 64), ([300] * 61, 128),
                                       ([7] * 300, 64), (list(range(1, 700, 9)), 64), ([9000] + [1] * 40, 64), ([0, 0], 64)])
@pytest.mark.parametrize("tiles_from", [0, None])           # every batch by tiles; as many segments as the rule asks for
def test_paged_decode_tiles(monkeypatch, hq, hkv, d, lens, page, tiles_from):
    from miles_b200.ops import cuda as K
    from miles_b200.ops import cuda_more

    if tiles_from is not None:
        monkeypatch.setattr(cuda_more, "_DECODE_TILES_FROM", tiles_from)
    args = _inputs(lens, hq, hkv, d, page)
    ref = _softmax64(*args)
    out = K.paged_attention(*args)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):                 # two in a row, the second one's kernels start while the first one's still run
        K.paged_attention(*args)
        again = K.paged_attention(*args)
    graph.replay()
    assert torch.isfinite(out).all() and torch.equal(out, again)
    # weights and outputs are rounded to bf16 once each: 2^-9 relative and independent
    assert (out.double() - ref).norm().item() <= 2 ** -8 * ref.norm().item()
    assert K.check_error_flag(out) == 0


@pytest.mark.parametrize("rows,hq,hkv", [(1, 32, 4), (8, 32, 4), (9, 32, 4), (4, 16, 8), (5, 16, 8), (32, 8, 1)])
def test_few_segments_are_split_as_they_always_were(rows, hq, hkv):
    """Up to 32 (request, KV head) segments the split form runs as one wave: it is the faster one, and its sums keep their order."""
    from miles_b200.ops import cuda as K

    q, k, v, table, lens = _inputs([1801 - 31 * b for b in range(rows)], hq, hkv, 128, 64)
    splits = max(1, min(8, -(-296 // (rows * hkv))))
    part = lambda n: torch.empty(rows * hq * splits * n, dtype=torch.float32, device="cuda")
    want, tiles = torch.empty_like(q), torch.empty_like(q)
    K.C.paged_decode(q, k, v, table, lens, want, part(128), part(2), 1 / math.sqrt(128), splits)
    K.C.paged_decode_tiles(q, k, v, table, lens, tiles, 1 / math.sqrt(128), K.C.error_flag(q))
    assert not torch.equal(want, tiles)
    assert torch.equal(K.paged_attention(q, k, v, table, lens), want if rows * hkv <= 32 else tiles)


def test_asked_for_splits_do_not_depend_on_the_batch():
    """MILES_DECODE_SPLITS pins where a request's sums are cut."""
    import os
    import subprocess
    import sys

    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    code = """
import sys
sys.path.insert(0, %r)
import torch
from tests.test_gpu_paged_tiles import _inputs
from miles_b200.ops import cuda as K
q, k, v, table, lens = _inputs([700, 64, 3001, 1], 32, 4, 128, 64)
out = K.paged_attention(q, k, v, table, lens)
for b in range(4):
    assert torch.equal(out[b], K.paged_attention(q[b:b + 1], k, v, table[b:b + 1], lens[b:b + 1])[0]), b
""" % root
    for splits in ("1", "4"):
        subprocess.run([sys.executable, "-c", code], check=True, cwd=root, env={**os.environ, "MILES_DECODE_SPLITS": splits})
