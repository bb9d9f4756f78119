"""float32 products on the tensor cores (operands as three bfloat16 values) against float64: around the tiles'
edges (16, 32, 64, 128, 256), with weights that are bfloat16 values and that are not, with infinities and NaN, and the rule that
chooses the product."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def inputs(T, N, K, exact_weights, seed=0):
    g = torch.Generator(device=DEV).manual_seed(seed)
    x, w = torch.randn((T, K), generator=g, device=DEV), torch.randn((N, K), generator=g, device=DEV)
    return x, (w.bfloat16().float() if exact_weights else w)


def bound(x, w):
    """What a result may be off by, of the sum of |x| |w|: products left out 2^-21; the tensor cores cut bits off (2^-23 each) at 4
    additions of 16 products and inside each, 8 in all; K / 64 + 1 rounded additions of 2^-24."""
    return (x.double().abs() @ w.double().abs().t()) * (2.0 ** -21 + 8 * 2.0 ** -23 + (x.shape[1] / 64 + 1) * 2.0 ** -24)


@pytest.mark.parametrize("T,N,K,tokens", [(1, 1, 4, 0), (16, 256, 32, 0), (17, 257, 36, 16), (31, 255, 60, 32), (128, 128, 64, 0), (129, 300, 100, 96),
                                          (256, 512, 2048, 0), (257, 513, 2052, 0), (600, 100, 68, 256), (700, 2048, 2048, 0)])
@pytest.mark.parametrize("exact_weights", [True, False])
def test_gemm_f32(T, N, K, tokens, exact_weights):
    from turboquant_cpp_b200.kernels.gemm_f32 import MIN_K, gemm_f32
    from turboquant_cpp_b200.kernels.gemm_tc import check_status
    x, w = inputs(T, N, K, exact_weights)
    y = gemm_f32(x, w, tokens)
    want = x.double() @ w.double().t()
    assert bool(((y.double() - want).abs() <= bound(x, w)).all())
    library = torch.mm(x, w.t())
    if K >= MIN_K:                        # as accurate as a float32 sum wherever it is chosen; a sum of 32 has fewer roundings than this has parts
        assert (y.double() - want).norm() <= 1.05 * (library.double() - want).norm() + 1e-12
    # rows of a wider tensor, infinities and NaN: where they are, and nowhere else
    wide = torch.zeros((T, K + 8), device=DEV)
    wide[:, 4:K + 4] = x
    wide[T // 2, 5] = math.inf
    wide[T - 1, 4 + K // 2] = math.nan
    w[N // 2, 0] = -math.inf
    y, library = gemm_f32(wide[:, 4:K + 4], w, tokens), torch.mm(wide[:, 4:K + 4], w.t())
    assert torch.equal(y.isnan(), library.isnan()) and torch.equal(y[y.isinf()], library[library.isinf()])
    check_status()


def test_which_products_it_takes():
    from turboquant_cpp_b200.kernels import gemm_f32 as KF
    from turboquant_cpp_b200.kernels.linear import linear
    x, w = inputs(256, 1024, 64, False)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    assert KF.pays(x, w) and torch.equal(linear(x, w, status=status), KF.gemm_f32(x, w))
    assert torch.equal(linear(x, w), torch.mm(x, w.t()))                     # no status word: the library's
    strided = torch.randn((256, 130), device=DEV)[:, 1:65]                   # rows off 16-byte boundaries
    for a, b in ((x[:100], w), (x[:, :62], w[:, :62]), (strided, w), (x.t().contiguous().t(), w), (x, w.t().contiguous().t()), (x.clone().requires_grad_(), w)):
        assert not KF.pays(a, b)
        torch.testing.assert_close(linear(a, b, status=status), torch.mm(a, b.t()), rtol=0, atol=0)
    assert int(status) == 0
