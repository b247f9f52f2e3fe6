"""Norm, router logits and top-k of a decode step in one launch, against 64 bits and against the kernels it stands for."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,H,E,k,residual,normalize", [
    (1, 2048, 16, 8, True, True), (7, 2048, 16, 8, True, True), (61, 2048, 16, 8, True, False), (3, 8, 1, 1, True, True), (2, 264, 13, 13, False, True),
    (5, 4096, 16, 8, True, True), (8, 4088, 9, 6, True, False), (64, 512, 15, 4, True, True)])
def test_against_64_bits(T, H, E, k, residual, normalize):
    from miles_b200.ops import cuda as K

    g = torch.Generator(device="cuda").manual_seed(T * H + E)
    rand = lambda *s: torch.randn(*s, device="cuda", generator=g)
    x, res = rand(T, H).bfloat16(), (rand(T, H) * 3).bfloat16() if residual else None
    nw = (1 + 0.2 * rand(H)).bfloat16()
    router = torch.nn.Parameter((rand(E, H) * 2 / H ** 0.5).bfloat16())
    with torch.no_grad():
        assert K.few_token_router(x, router)
        xn, total, w, idx = K.add_rmsnorm_router(x, res, nw, 1e-6, router, k, normalize)
        want_xn, want_total = K.add_rmsnorm(x, res, nw, 1e-6) if residual else (K.rmsnorm(x, nw, 1e-6), x)
    assert torch.equal(total, want_total)
    # the sum of squares may be added up in another order: rounding to bf16 may fall the other way, one step of 2^-8 of the value
    assert (xn.double() - want_xn.double()).abs().le(want_xn.double().abs() * 2 ** -7 + 1e-30).all()
    h = want_total.double()
    logits = (h * torch.rsqrt(h.pow(2).mean(-1, keepdim=True) + 1e-6) * nw.double()) @ router.detach().double().t()
    probs = torch.softmax(logits, -1)
    # logits of order one to ten: fp32 sums of up to 4096 terms are good to about 1e-6 of them, exp to 1e-6; a probability to a few 1e-5
    assert ((idx >= 0) & (idx < E)).all() and all(len(set(r)) == k for r in idx.tolist())
    top = probs.gather(1, idx.long())
    assert torch.allclose(top, probs.topk(k, -1).values, rtol=1e-4, atol=1e-9)        # a near tie may go either way
    want = top / top.sum(-1, keepdim=True) if normalize else top
    assert torch.allclose(w.double(), want, rtol=1e-4, atol=1e-9)


def test_rows_that_are_no_numbers():
    from miles_b200.ops import cuda as K

    x = torch.randn(4, 256, device="cuda").bfloat16()
    x[1] = float("nan")
    x[2, 5] = float("inf")
    router = torch.nn.Parameter(torch.randn(16, 256, device="cuda").bfloat16())
    nw = torch.ones(256, device="cuda").bfloat16()
    with torch.no_grad():
        _, _, w, idx = K.add_rmsnorm_router(x, torch.zeros_like(x), nw, 1e-6, router, 4)
        _, _, _, alone = K.add_rmsnorm_router(x[3:], torch.zeros_like(x[3:]), nw, 1e-6, router, 4)
    assert (idx[1] == -1).all() and (idx[2] == -1).all() and torch.equal(idx[3], alone[0]) and (idx[0] >= 0).all()


def test_where_it_applies():
    from miles_b200.ops import cuda as K

    x, router = torch.randn(4, 256, device="cuda").bfloat16(), torch.randn(16, 256, device="cuda").bfloat16()
    assert not K.few_token_router(x, router)                                          # a backward may follow
    with torch.no_grad():
        assert K.few_token_router(x, router)
        assert not K.few_token_router(x.float(), router) and not K.few_token_router(torch.cat([x] * 17), router)
        assert not K.few_token_router(x[:, :252].contiguous(), router[:, :252].contiguous())      # rows of the router off a 16-byte boundary
        assert not K.few_token_router(x, torch.cat([router, router[:1]])) and not K.few_token_router(x, torch.randn(256, 16, device="cuda").bfloat16().t())
