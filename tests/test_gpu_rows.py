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


@pytest.mark.parametrize("T,Hq,Hk,D,norm,offset", [(1184, 4, 4, 128, True, 0), (601, 32, 4, 128, True, 0), (500, 40, 8, 128, False, 0), (3001, 6, 1, 128, True, 0),
                                                   (700, 32, 8, 64, True, 0), (601, 32, 4, 128, True, 2), (601, 32, 4, 128, False, 1), (77, 4, 4, 64, True, 1)])
def test_rotation_of_many_tokens(T, Hq, Hk, D, norm, offset):
    from miles_b200.ops import cuda as K

    g = torch.Generator(device="cuda").manual_seed(T)
    rand = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()
    width = (Hq + 2 * Hk) * D
    qkv = rand(T * width + offset)[offset:].view(T, width)               # an offset of one or two elements: no 8-byte pieces
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
    # a token is rotated alike in every batch: the engine's few rows, its prefill and the trainer's pack
    assert torch.equal(q2, q1) and torch.equal(k2, k1) and torch.equal(q3, q2) and torch.equal(k3, k2)
    pair = lambda x: x.double().view(*x.shape[:-1], 2, D // 2)
    for x, wn, got in ((q, qw, q2), (k, kw, k2)):
        # against 64 bits: the normalised head and the result are rounded to bf16 once each (2^-9 of the pair's length); an angle of up to 30 000
        # is a product of fp32 numbers (2^-24 of it) whose second one is an exp2f of a rounded exponent (2^-22), taken in turns by another (2^-24)
        xd = x.double()
        if norm:
            xd = xd * torch.rsqrt(xd.pow(2).mean(-1, keepdim=True) + 1e-6) * wn.double()
        angle = pos.double()[:, None] * 1e6 ** (-2 * torch.arange(D // 2, device="cuda").double() / D)
        c, s = angle.cos()[:, None], angle.sin()[:, None]
        a, b = pair(xd).unbind(-2)
        want = torch.stack([a * c - b * s, b * c + a * s], -2)
        assert ((pair(got) - want).norm(dim=-2) <= (2.0 ** -8 + 30000 * (2.0 ** -22 + 2.0 ** -23)) * want.norm(dim=-2) + 1e-6).all()
    want = cache.clone()
    want[0, slots[slots >= 0]], want[1, slots[slots >= 0]] = k3[slots >= 0], v[slots >= 0]
    assert torch.equal(kc[0], want[0]) and torch.equal(vc[0], want[1])


@pytest.mark.parametrize("T,heads", [(1, 4), (37, 32), (700, 8)])
@pytest.mark.parametrize("offset", [0, 2])                 # rows off an 8-byte boundary take a warp per head
def test_qk_norm_rope_backward_four_heads_at_a_time(T, heads, offset):
    """Gradients of norm and rotation against 64 bits."""
    from miles_b200.ops import cuda as K

    g = torch.Generator(device="cuda").manual_seed(T + heads)
    rand = lambda *s: torch.randn(*s, device="cuda", generator=g)
    wide = rand(T, (heads + 2) * 128 + 4).bfloat16()
    x = wide[:, offset:offset + heads * 128].view(T, heads, 128)
    w, dy, pos = (1 + 0.2 * rand(128)).bfloat16(), rand(T, heads, 128).bfloat16(), torch.randint(0, 5000, (T,), device="cuda", dtype=torch.int32)
    x64 = x.double().requires_grad_()
    w64 = w.double().requires_grad_()
    rstd = torch.rsqrt(x64.pow(2).mean(-1, keepdim=True) + 1e-6)
    n = x64 * rstd * w64
    ang = pos.double()[:, None] * 1e6 ** (-torch.arange(0, 128, 2, device="cuda", dtype=torch.float64) / 128)
    c, s = ang.cos()[:, None], ang.sin()[:, None]
    y = torch.cat([n[..., :64] * c - n[..., 64:] * s, n[..., 64:] * c + n[..., :64] * s], -1)
    y.backward(dy.double())
    dx = torch.empty(T, heads, 128, dtype=torch.bfloat16, device="cuda")
    dw = K.C.qk_norm_rope_bwd(x, w, rstd.detach().float().view(-1), dy, pos, dx, 1e6)
    # one rounding to bf16 each (2^-9), angles of up to 5000 in fp32 (5000 · 2^-24 = 3e-4 of a turn's radius)
    assert ((dx.double() - x64.grad).norm() / x64.grad.norm()).item() < 3e-3
    assert ((dw.double() - w64.grad).norm() / w64.grad.norm()).item() < 5e-3


@pytest.mark.parametrize("add", [False, True])
@pytest.mark.parametrize("H", [8, 264, 512, 520, 1024, 2048, 2560, 4096, 4104, 6152, 8192, 8200, 16392])
def test_rmsnorm_of_any_width(H, add):
    """Widths around the edges of its pieces and threads; a row's result does not depend on the rows beside it.  y is rounded to bf16 once behind fp32 sums:
    half a unit in the last of 8 bits, and the norm's own error (squares and their sum in fp32, rsqrt) far below it."""
    from miles_b200.ops import cuda as K

    g = torch.Generator(device="cuda").manual_seed(H)
    x, r = (torch.randn(70, H, device="cuda", generator=g).bfloat16() for _ in range(2))
    w = (1 + 0.1 * torch.randn(H, device="cuda", generator=g)).bfloat16()
    x[5, 0], x[6] = float("nan"), 0
    r[6] = 0
    with torch.no_grad():
        run = (lambda s: K.add_rmsnorm(x[s], r[s], w, 1e-6)) if add else (lambda s: (K.rmsnorm(x[s], w, 1e-6), x[s]))
        y, total = run(slice(0, 70))
        few, few_total = run(slice(60, 63))
    h = (x.double() + r.double()).bfloat16() if add else x
    assert torch.equal(total[[0, 69]], h[[0, 69]])
    want = h.double() * (h.double().pow(2).mean(-1, keepdim=True) + 1e-6).rsqrt() * w.double()
    ok = torch.arange(70, device="cuda") != 5
    assert y[5].isnan().all() and ((y.double() - want)[ok].abs() <= want[ok].abs() * 2.0 ** -8 * 1.01).all()
    assert torch.equal(few, y[60:63]) and torch.equal(few_total, total[60:63])
