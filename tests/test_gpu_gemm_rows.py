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
        assert ops.few_token_decode(x, w) == (M <= 8 and N <= 12288)
        y = K.linear(x, w)
    want = x.double() @ w.double().t()
    assert ((y.double() - want).norm() / want.norm()).item() < 2 ** -8.5          # one rounding to bf16
