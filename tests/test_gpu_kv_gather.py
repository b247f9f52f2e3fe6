"""Rows of a paged cache by slot, keys and values in one launch, against index_select of each."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads,dim", [(1, 8), (1, 128), (3, 40), (4, 128), (8, 128)])
@pytest.mark.parametrize("n", [0, 1, 3, 4, 33, 1001])
def test_kv_gather(n, heads, dim):
    from miles_b200.ops import cuda as K
    torch.manual_seed(3)
    kc = torch.randn(7, 16, heads, dim, device="cuda").bfloat16()
    vc = torch.randn(7, 16, heads, dim, device="cuda").bfloat16()
    kc[1, 2] = float("nan")
    vc[0, 0] = float("-inf")
    slots = torch.randint(0, 7 * 16, (n,), device="cuda")
    slots[:1], slots[-1:] = 0, 7 * 16 - 1
    k, v = K.C.kv_gather(kc, vc, slots, K.C.error_flag(kc))
    assert k.shape == v.shape == (n, heads, dim)
    for got, cache in ((k, kc), (v, vc)):
        want = cache.view(-1, heads, dim).index_select(0, slots)
        assert torch.equal(got.view(torch.int16), want.view(torch.int16))
    assert K.check_error_flag() == 0


@pytest.mark.parametrize("bad", [-1, 64])
def test_slot_outside_the_cache(bad):
    """Zeros in its place and the error flag; the other rows as they are."""
    from miles_b200.ops import cuda as K
    kc = torch.randn(4, 16, 2, 128, device="cuda").bfloat16()
    slots = torch.tensor([5, bad, 63], device="cuda")
    k, v = K.C.kv_gather(kc, kc, slots, K.C.error_flag(kc))
    flag = K.C.error_flag(kc)
    torch.cuda.synchronize()
    assert int(flag.item()) == 73
    flag.zero_()
    for got in (k, v):
        assert torch.equal(got[0], kc.view(-1, 2, 128)[5]) and torch.equal(got[2], kc.view(-1, 2, 128)[63]) and not got[1].any()
