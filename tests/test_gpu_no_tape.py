"""Without gradients the forward passes run outside of autograd: the same results, forward mode is refused and traces run the kernels as before."""
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


@pytest.mark.filterwarnings("ignore")
@pytest.mark.parametrize("name", ["linear", "linear_fp32", "rmsnorm", "add_rmsnorm", "swiglu", "rope", "qk_norm_rope", "attention", "router"])
def test_trace_without_gradients(name):
    """A trace made under no_grad computes: it holds the function, not the memory that its kernels wrote while it was made."""
    f, x = _ops()[name]
    with torch.no_grad():
        traced = torch.jit.trace(f, x.clone(), check_trace=False)
        other = (x.float() * 0.5 + 0.25).to(x.dtype)
        assert torch.equal(traced(other), f(other))


@pytest.mark.filterwarnings("ignore")
def test_trace_of_gate_and_up():
    from miles_b200.ops import cuda_more

    g = torch.Generator(device="cuda").manual_seed(3)
    rand = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()
    x, w = rand(9000, 1024), rand(4096, 1024) * 0.03                 # sizes of the fused product
    with torch.no_grad():
        traced = torch.jit.trace(lambda x: cuda_more.linear_swiglu(x, w), x, check_trace=False)
        other = rand(9000, 1024)
        assert torch.equal(traced(other), cuda_more.linear_swiglu(other, w))
