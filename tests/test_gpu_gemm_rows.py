"""Projections of up to 64 tokens with the reduction cut over a cluster of CTAs, against 64-bit products."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [1, 16, 17, 33, 64])
@pytest.mark.parametrize("N,Kd", [(16, 2048), (200, 328), (2048, 64), (2176, 4096)])
@pytest.mark.parametrize("split", [1, 2, 4, 8])
def test_gemm_rows(M, N, Kd, split):
    from miles_b200.ops import cuda as K

    g = torch.Generator(device="cuda").manual_seed(11)
    x = torch.randn(M, Kd, device="cuda", generator=g).bfloat16()
    w = (torch.randn(N, Kd, device="cuda", generator=g) * 0.05).bfloat16()
    bias = torch.randn(N, device="cuda", generator=g).bfloat16()
    ref = x.double() @ w.double().t()
    for dtype, limit in ((torch.bfloat16, 2 ** -8.5), (torch.float32, 1e-5)):      # one rounding to bf16; the order of fp32 sums
        for b, early in ((None, True), (bias, False)):
            y = torch.full((M, N + 8), math.nan, device="cuda", dtype=dtype)
            K.C.gemm_rows(x, w, y, M, N, Kd, N + 8, b, split, early)
            want = ref if b is None else ref + bias.double()
            assert ((y[:, :N].double() - want).norm() / want.norm()).item() < limit
            assert torch.isnan(y[:, N:]).all()
    assert K.check_error_flag(x) == 0


def test_split_fits_the_gpu():
    from miles_b200.ops import cuda as K

    for M in (9, 32, 33, 64):
        for N in (1, 128, 1024, 2048, 2560, 5120, 18944, 18945, 37888, 37889, 151936):
            for Kd in (8, 64, 100, 2048, 9728):
                s, tiles = K._row_split(M, N, Kd), -(-N // 128)
                assert (s == 0) == (tiles > (296 if M <= 32 else 148))
                assert s == 0 or (tiles * s <= 296 and (s == 1 or -(-Kd // 64) >= 2 * s))


@pytest.mark.parametrize("M,N", [(8, 640), (9, 640), (16, 640), (17, 640), (1, 12288), (1, 12289), (8, 12416)])
def test_from_matrix_vector_to_clusters(M, N):
    from miles_b200 import ops
    from miles_b200.ops import cuda as K

    g = torch.Generator(device="cuda").manual_seed(M)
    x, w = torch.randn(M, 1024, device="cuda", generator=g).bfloat16(), torch.randn(N, 1024, device="cuda", generator=g).bfloat16()
    with torch.no_grad():
        assert ops.few_token_decode(x, w) == (M <= 16)
        assert (M <= K._gemv_rows(K._row_split(M, N, 1024), N, 1024)) == (M <= 8 and N <= 12288)
        y = K.linear(x, w)
    want = x.double() @ w.double().t()
    assert ((y.double() - want).norm() / want.norm()).item() < 2 ** -8.5          # one rounding to bf16


@pytest.mark.parametrize("M,N,Kd", [(1, 640, 2048), (8, 640, 2048), (9, 640, 2048), (16, 16, 2048), (16, 5120, 2048), (1, 6144, 2560), (4, 6144, 2560),
                                    (13, 19456, 2560), (8, 12416, 1024), (9, 200, 4064)])
@pytest.mark.parametrize("ones", [True, False])
@pytest.mark.parametrize("with_residual", [True, False])
def test_few_rows_behind_a_norm(M, N, Kd, ones, with_residual):
    """Whichever kernel takes the projection: with norm weights of one its operand is the sum itself, not a rounded quotient."""
    from miles_b200 import ops
    from miles_b200.ops import cuda as K

    g = torch.Generator(device="cuda").manual_seed(M + N)
    rand = lambda *s: torch.randn(*s, device="cuda", generator=g)
    x, r, w = rand(M, Kd).bfloat16(), rand(M, Kd).bfloat16() if with_residual else None, (rand(N, Kd) * 0.05).bfloat16()
    nw = torch.ones(Kd, device="cuda").bfloat16() if ones else (1 + 0.1 * rand(Kd)).bfloat16()
    bias = rand(N).bfloat16()
    h = (x.double() + r.double()).bfloat16() if with_residual else x
    quotient = h.double() * torch.rsqrt(h.double().pow(2).mean(-1, keepdim=True) + 1e-6)
    want = quotient * nw.double() @ w.double().t() + bias.double()
    rel = lambda a, b: ((a.double() - b).norm() / b.norm()).item()
    with torch.no_grad():
        assert ops.few_token_decode(x, w)                 # what a decoder layer asks; else it norms first and multiplies then
        y, total, normed = K.add_rmsnorm_linear(x, r, nw, 1e-6, w, bias, want_normed=True)
        y32, _, none = K.add_rmsnorm_linear(x, r, nw, 1e-6, w, bias, out_fp32=True)
    assert none is None and ((total is None) if r is None else torch.equal(total, h))
    assert rel(normed, quotient * nw.double()) < 2 ** -9                          # one rounding to bf16: 2^-9 of each value at most
    # fp32: the order of sums of up to 4064 terms; times norm weights, one rounding of the operand on the way (2^-9 of each term, independent)
    assert rel(y32, want) < (1e-5 if ones else 2 ** -9)
    assert rel(y, want) < (2 ** -9 if ones else 2 ** -8.5)                        # … and one of the result
    assert K.check_error_flag(x) == 0


@pytest.mark.parametrize("which", ["x", "residual", "norm weights"])
def test_rows_off_a_16_byte_boundary_are_refused(which):
    """By the host, whichever kernel the projection goes to (the matrix-vector one at 8 rows looks at the rows alone, as it always did)."""
    from miles_b200.ops import cuda as K

    off = lambda *s: torch.zeros(math.prod(s) + 1, device="cuda", dtype=torch.bfloat16)[1:].view(*s)
    on = lambda *s: torch.zeros(*s, device="cuda", dtype=torch.bfloat16)
    make = lambda name: off if name == which else on
    w = on(640, 2048)
    for M in (8, 9) if which == "x" else (9,):
        x, r, nw = make("x")(M, 2048), make("residual")(M, 2048), make("norm weights")(2048)
        assert (K._row_split(M, 640, 2048) > 0 and M > K._gemv_rows(K._row_split(M, 640, 2048), 640, 2048)) == (M == 9)
        with torch.no_grad(), pytest.raises(RuntimeError):
            K.add_rmsnorm_linear(x, r, nw, 1e-6, w)


def test_weights_ahead_of_the_rows():
    """Weights that nothing on the stream writes are requested before the kernel in front, which makes the rows, has finished."""
    from miles_b200.ops import cuda as K

    g = torch.Generator(device="cuda").manual_seed(5)
    x, nw = torch.randn(16, 2560, device="cuda", generator=g).bfloat16(), torch.ones(2560, device="cuda").bfloat16()
    ws = [torch.nn.Parameter((torch.randn(2560, 2560, device="cuda", generator=g) * 0.02).bfloat16()) for _ in range(6)]
    with torch.no_grad():
        def chain():
            y = x
            for w in ws:                                  # norm and product in turn: each kernel reads what the one in front writes
                y = K.add_rmsnorm_linear(y, None, nw, 1e-6, w)[0]
            return y
        first = chain()
        stepwise = x
        for w in ws:
            torch.cuda.synchronize()
            stepwise = K.add_rmsnorm_linear(stepwise, None, nw, 1e-6, w)[0]
            torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            captured = chain()
        for _ in range(20):
            captured.zero_()
            graph.replay()
            assert torch.equal(captured, stepwise)
    assert torch.equal(first, stepwise) and K.check_error_flag(x) == 0


@pytest.mark.parametrize("T", [1, 9, 16, 17, 32, 33, 64])
@pytest.mark.parametrize("F,K", [(64, 256), (3072, 1024), (320, 328), (9472, 512)])
@pytest.mark.parametrize("split", [1, 2, 4, 8])
def test_gate_and_up_in_one_product(T, F, K, split):
    """silu(gate) · up where the sums are: the bits of the product and the activation apart, with and without factors on the rows."""
    from miles_b200.ops.cuda import C

    if split > 1 and K // 64 < split:
        pytest.skip("fewer steps than slices")
    g = torch.Generator(device="cuda").manual_seed(T + F)
    x, w = torch.randn(T, K, device="cuda", generator=g).bfloat16(), (torch.randn(2 * F, K, device="cuda", generator=g) / K ** 0.5 * 2).bfloat16()
    for scale in (None, torch.rand(T, device="cuda", generator=g) + 0.5):
        h, want, got = (torch.empty(T, n, dtype=torch.bfloat16, device="cuda") for n in (2 * F, F, F))
        C.gemm_rows(x, w, h, T, 2 * F, K, 2 * F, None, split, False, scale)
        C.swiglu_fwd(h, want, None)
        C.gemm_rows(x, w, got, T, 2 * F, K, F, None, split, False, scale, True)
        assert torch.equal(got, want)


@pytest.mark.parametrize("T", [1, 8, 12, 16, 19, 32, 50])
@pytest.mark.parametrize("F,K", [(3072, 1024), (9728, 2560), (72, 512)])
def test_gate_and_up_behind_a_norm(T, F, K):
    """Through the functions that models call: what the norm, the projection and the activation give one after another."""
    from miles_b200.ops import cuda as K_

    g = torch.Generator(device="cuda").manual_seed(T + F)
    x, r = (torch.randn(T, K, device="cuda", generator=g).bfloat16() for _ in range(2))
    w, nw = torch.nn.Parameter((torch.randn(2 * F, K, device="cuda", generator=g) / K ** 0.5 * 2).bfloat16()), (1 + 0.1 * torch.randn(K, device="cuda", generator=g)).bfloat16()
    with torch.no_grad():
        assert torch.equal(K_.linear_swiglu(x, w), K_.swiglu(K_.linear(x, w)))
        if K_.gemv_ok(x, w):
            y, res = K_.add_rmsnorm_swiglu(x, r, nw, 1e-6, w)
            h13, want_res, _ = K_.add_rmsnorm_linear(x, r, nw, 1e-6, w)
            assert torch.equal(y, K_.swiglu(h13)) and torch.equal(res, want_res)
    assert K_.check_error_flag(x) == 0
