"""float32 products and float32 prompt attention on the tensor cores (operands as three bfloat16 values) against float64: around the tiles'
edges (16, 32, 64, 128, 256), with weights that are bfloat16 values and that are not, with infinities and NaN, and the rule that
chooses the product."""
import math

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def inputs(T, N, K, exact_weights, seed=0):
    g = torch.Generator(device=DEV).manual_seed(seed)
    x, w = torch.randn((T, K), generator=g, device=DEV), torch.randn((N, K), generator=g, device=DEV)
    return x, (w.bfloat16().float() if exact_weights else w)


def bound(x, w):
    """What a result may be off by, of the sum of |x| |w|: products left out 2^-26; the tensor cores cut bits off (2^-23 each) at 4
    additions of 16 products and inside each, 8 in all, and at every product of the smaller ones (2^-8 of the sum, five a block of 16);
    K / 64 + 1 rounded additions of 2^-24."""
    K = x.shape[1]
    return (x.double().abs() @ w.double().abs().t()) * (2.0 ** -26 + (8 + 5 * K / 16 * 2.0 ** -8) * 2.0 ** -23 + (K / 64 + 1) * 2.0 ** -24)


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
    if K >= MIN_K:                        # as accurate as a float32 sum wherever it is chosen; sums of fewer elements have as few roundings as this
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
    for (T, N, K), taken in {(16, 20480, 128): False, (64, 20480, 128): False, (65, 20480, 128): True, (16, 20480, 256): True, (4096, 64, 64): True,
                             (8, 30000, 512): False}.items():
        assert KF.pays(torch.empty((T, K), device=DEV), torch.empty((N, K), device=DEV)) == taken, (T, N, K)
    assert int(status) == 0


def test_a_build_that_cannot_launch_leaves_the_products_to_the_library(monkeypatch):
    from turboquant_cpp_b200.kernels import gemm_f32 as KF
    from turboquant_cpp_b200.kernels.linear import linear
    x, w = inputs(256, 1024, 512, False)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    assert KF.runs() and KF.pays(x, w)
    monkeypatch.setattr(KF, "runs", lambda: False)
    assert not KF.pays(x, w) and torch.equal(linear(x, w, status=status), torch.mm(x, w.t()))


CASES = [  # H, G, head size, page, runs, held, window
    (4, 2, 128, 64, [1, 31, 32, 33, 64, 65], [0, 0, 31, 40, 0, 7], 0),
    (6, 3, 64, 64, [127, 300], [0, 100], 0),
    (4, 1, 64, 48, [200, 20], [13, 0], 70),              # a tile of keys lies in two pages
    (2, 2, 128, 16, [129, 65], [0, 500], 33),
    (16, 16, 128, 64, [700], [0], 0),
    (4, 2, 128, 64, [1, 1, 200, 1, 1], [300, 5, 0, 64, 1000], 0),                # a prompt beside sequences that bring one token
    (8, 2, 64, 64, [1] * 9 + [70], [40 * i + 1 for i in range(9)] + [3], 50),
]


@pytest.mark.parametrize("case", range(len(CASES)))
@pytest.mark.parametrize("spread", [1.0, 6.0])
def test_attention_f32(case, spread):
    from test_attention_prefill_gpu import attend
    from turboquant_cpp_b200.kernels import attention as KA
    H, G, hd, page, runs, held, window = CASES[case]
    g = torch.Generator(device=DEV).manual_seed(case)
    r = lambda *s: torch.randn(s, generator=g, device=DEV)
    i32 = lambda a: torch.tensor(np.asarray(a), dtype=torch.int32, device=DEV)
    T, cu = sum(runs), np.concatenate([[0], np.cumsum(runs)])
    counts = [-(-(a + b) // page) for a, b in zip(runs, held)]
    order, table, at = np.random.RandomState(0).permutation(sum(counts)), np.full((len(runs), max(counts)), -1), 0
    cache = torch.full((sum(counts), 2, G, page, hd), 1e30, device=DEV)         # what lies behind a sequence's end
    q, rows = spread * r(T, H, hd), []
    for i, c in enumerate(counts):
        table[i, :c] = order[at:at + c]
        at += c
        n = runs[i] + held[i]
        rows.append((r(n, G, hd), r(n, G, hd)))
        pos = torch.arange(n, device=DEV)
        where = i32(table[i]).long()[pos // page]
        cache[where, 0, :, pos % page], cache[where, 1, :, pos % page] = rows[i]
    out = torch.full((T, H * hd), math.nan, device=DEV)
    run = lambda: KA.attention_tiled(q, cache, i32(cu), i32(held), i32(table), page, window, hd ** -0.5, out, len(runs), H, G, hd)
    run()
    tf32, torch.backends.cuda.matmul.allow_tf32 = torch.backends.cuda.matmul.allow_tf32, False

    def compare(first_row=0):
        """The whole step's error beside that of the same formulas in float32: a part of the operands or a product left out is ten times it."""
        ours = theirs = size = 0.0
        for i in range(len(runs)):
            skip = first_row if i == 0 else 0
            mine = slice(cu[i] + skip, cu[i + 1])
            args = (held[i] + skip, hd ** -0.5, window, 0, 0, 0.0, None, None)
            want, _ = attend(q[mine].double(), rows[i][0].double(), rows[i][1].double(), *args)
            single, _ = attend(q[mine], rows[i][0], rows[i][1], *args)
            got = out[mine].view(-1, H, hd).double()
            ours, theirs, size = ours + (got - want).square().sum(), theirs + (single.double() - want).square().sum(), size + want.square().sum()
        assert float(ours) ** 0.5 <= 2 * float(theirs) ** 0.5 + 2.0 ** -25 * float(size) ** 0.5, (float(ours / size) ** 0.5, float(theirs / size) ** 0.5)

    try:
        compare()
        # a key of -inf has no weight (the row that sees no other key has no result)
        first, alone = int(table[0, 0]), 1 if held[0] == 0 else 0
        cache[first, 0, 0, 0, 1] = -math.inf
        rows[0][0][0, 0, 1] = -math.inf
        q[..., 1] = q[..., 1].abs() + 0.1
        run()
        compare(alone)
        assert bool(out[alone:].isfinite().all())
    finally:
        torch.backends.cuda.matmul.allow_tf32 = tf32
    # a value of inf shows in the rows that see it, and in no others
    was, key = out.clone(), 1 if len(runs) == 1 else 0           # not the key that has no weight
    cache[int(table[-1, 0]), 1, 0, key, 0] = math.inf
    run()
    pos = torch.arange(runs[-1], device=DEV) + held[-1]
    sees = (pos >= key) & (pos - key < window if window else pos >= 0)
    met = torch.zeros((T, H, hd), dtype=torch.bool, device=DEV)
    met[cu[-2]:, :H // G, 0] = sees[:, None]
    got, rest = out.view(T, H, hd), ~met
    rest[:alone] = False
    assert bool((got[met] == math.inf).all())
    torch.testing.assert_close(got[rest], was.view(T, H, hd)[rest], rtol=1e-5, atol=1e-5)      # rows that met it are summed again, key by key
