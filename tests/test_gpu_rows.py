"""Row kernels for many tokens: norms whose backward (and, at 1024, 2048 and 4096, whose forward) takes a row in the registers of a warp or
several, rotation of several heads by one warp."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,H", [(592, 512), (700, 1024), (601, 1536), (1000, 2048), (593, 2560), (777, 3072), (640, 3584), (911, 4096), (700, 520)])
def test_rmsnorm_widths(T, H):
    from miles_b200.ops import cuda as K

    g = torch.Generator(device="cuda").manual_seed(H)
    rand = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()
    x, r, dy, dr = rand(T, H), rand(T, H), rand(T, H), rand(T, H)
    w = (1 + 0.1 * torch.randn(H, device="cuda", generator=g)).bfloat16()
    ins = [t.clone().requires_grad_() for t in (x, r, w)]
    y, s = K.add_rmsnorm(*ins, 1e-6)
    torch.autograd.backward([y, s], [dy, dr])
    # the norm is taken of the sum as it is stored; every 16-bit result is then rounded once (2^-9 of its value), gradients of x from the stored sum
    assert torch.equal(s, (x.double() + r.double()).bfloat16())
    sd, wd = s.detach().double().requires_grad_(), w.double().requires_grad_()
    yd = sd * torch.rsqrt(sd.pow(2).mean(-1, keepdim=True) + 1e-6) * wd
    torch.autograd.backward([yd, sd], [dy.double(), dr.double()])
    for got, want in ((y, yd), (ins[0].grad, sd.grad), (ins[1].grad, sd.grad), (ins[2].grad, wd.grad)):
        assert ((got.double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-4 * want.abs().max()).all()


@pytest.mark.parametrize("T", [1183, 1184, 1191])
@pytest.mark.parametrize("H", [512, 520, 1536, 2560, 3072, 3584])
def test_a_token_is_normed_alike_in_every_batch(T, H):
    """Widths with one kernel: the same bits for a token among 16 and among all (trainer and engine batch differently)."""
    from miles_b200.ops import cuda as K

    g = torch.Generator(device="cuda").manual_seed(H)
    rand = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()
    x, r, w = rand(T, H), rand(T, H), rand(H)
    with torch.no_grad():
        y, (ya, total) = K.rmsnorm(x, w, 1e-6), K.add_rmsnorm(x, r, w, 1e-6)
        few = [(K.rmsnorm(x[i:i + 16], w, 1e-6), *K.add_rmsnorm(x[i:i + 16], r[i:i + 16], w, 1e-6)) for i in range(0, T, 16)]
        assert all(torch.equal(all_rows, torch.cat(f)) for all_rows, f in zip((y, ya, total), zip(*few)))
        assert torch.equal(y[-1:], K.rmsnorm(x[-1:], w, 1e-6))


@pytest.mark.parametrize("T,Hq,Hk,D,norm", [(1184, 4, 4, 128, True), (601, 32, 4, 128, True), (500, 40, 8, 128, False), (3001, 6, 1, 128, True), (700, 32, 8, 64, True)])
def test_rotation_of_many_tokens(T, Hq, Hk, D, norm):
    from miles_b200.ops import cuda as K

    g = torch.Generator(device="cuda").manual_seed(T)
    rand = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()
    qkv = rand(T, (Hq + 2 * Hk) * D)
    q, k, v = (t.view(T, -1, D) for t in qkv.split([Hq * D, Hk * D, Hk * D], -1))
    qw, kw = (rand(D), rand(D)) if norm else (None, None)
    pos = torch.randint(0, 30000, (T,), device="cuda", generator=g, dtype=torch.int32)
    cache = rand(2, T + 5, Hk, D)
    slots = torch.randperm(T + 5, device="cuda", generator=g)[:T]
    slots[3::7] = -1
    with torch.no_grad():
        few = [K.qk_norm_rope(q[i:i + 16], k[i:i + 16], qw, kw, pos[i:i + 16], 1e6, 1e-6) for i in range(0, T, 16)]     # one warp per head
        q1, k1 = (torch.cat(t) for t in zip(*few))
        q2, k2 = K.qk_norm_rope(q, k, qw, kw, pos, 1e6, 1e-6)
        kc, vc = cache.clone().unsqueeze(1)
        q3, k3 = K.qk_norm_rope_cache(q, k, v, qw, kw, pos, 1e6, 1e-6, kc, vc, slots)
    # both forms round the normalised head to bf16 before they rotate it, and the result: 2^-9 of the pair's length each; sums of other order
    # may flip the first rounding (2^-8)
    def close(got, want):
        pair = want.float().view(*want.shape[:-1], 2, D // 2).norm(dim=-2, keepdim=True).expand(*want.shape[:-1], 2, D // 2).reshape(want.shape)
        return ((got.float() - want.float()).abs() <= 2.0 ** -6.5 * pair).all()

    assert close(q2, q1) and close(k2, k1) and torch.equal(q3, q2) and torch.equal(k3, k2)
    want = cache.clone()
    want[0, slots[slots >= 0]], want[1, slots[slots >= 0]] = k3[slots >= 0], v[slots >= 0]
    assert torch.equal(kc[0], want[0]) and torch.equal(vc[0], want[1])
