"""Without gradients the forward passes run outside of autograd: the same results, and forward mode is refused as before."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _ops():
    from miles_b200.ops import cuda as K

    g = torch.Generator(device="cuda").manual_seed(2)
    rand = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()
    x, w, v = rand(70, 256), rand(64, 256), rand(256)
    q, k = rand(70, 4, 128), rand(70, 2, 128)
    pos = torch.arange(70, device="cuda", dtype=torch.int32)
    cu = torch.tensor([0, 30, 70], device="cuda", dtype=torch.int32)
    return {
        "linear": (lambda x: K.linear(x, w), x), "linear_fp32": (lambda x: K.linear_fp32(x, w), x), "rmsnorm": (lambda x: K.rmsnorm(x, v), x),
        "add_rmsnorm": (lambda x: K.add_rmsnorm(x, x, v)[1], x), "swiglu": (K.swiglu, x), "rope": (lambda q: K.rope(q, pos, 1e6), q),
        "qk_norm_rope": (lambda q: K.qk_norm_rope(q, k, None, None, pos, 1e6, 1e-6)[0], q),
        "attention": (lambda q: K.attention_varlen(q, k, k, cu, 40), q), "router": (lambda x: K.router_topk(x.float(), 8)[0], x),
    }


@pytest.mark.parametrize("name", ["linear", "linear_fp32", "rmsnorm", "add_rmsnorm", "swiglu", "rope", "qk_norm_rope", "attention", "router"])
def test_same_without_gradients(name):
    import torch.autograd.forward_ad as fwd

    f, x = _ops()[name]
    taped = f(x.clone().requires_grad_())
    assert taped.requires_grad
    with torch.no_grad():
        plain = f(x.clone().requires_grad_())
        assert not plain.requires_grad and torch.equal(plain, taped)
        with fwd.dual_level(), pytest.raises((RuntimeError, NotImplementedError)):
            f(fwd.make_dual(x, torch.ones_like(x)))
