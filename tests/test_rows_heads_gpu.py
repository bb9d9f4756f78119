"""The tensor-core token form of the attention over rows at the edges of its tiles: 16 keys a tile, 8 or 16 heads a product."""
import math

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"
PAGE = 64


# heads per key/value head on both sides of 8 and 16, a last chunk of one head among them
@pytest.mark.parametrize("per_kv,dk,dv", [(2, 128, 128), (7, 64, 128), (8, 32, 32), (9, 64, 64), (16, 128, 32), (17, 32, 64)])
@pytest.mark.parametrize("window,keep,cap", [(0, 0, 0.0), (37, 20, 8.0)])
def test_tokens_of_several_sequences_against_float64(per_kv, dk, dv, window, keep, cap):
    from turboquant_cpp_b200.kernels import bias_attention as KB
    rng = np.random.default_rng(per_kv * 100 + dk + window)
    lens = [1, 15, 16, 17, 64, 65, 129, 300]                 # tiles, pages and warps (4 tiles) just full and just begun
    G, H, T, far = 2, 2 * per_kv, len(lens), 50
    assert KB.heads_form(torch.bfloat16, dk, dv, per_kv, PAGE)
    columns = -(-max(lens) // PAGE)
    table = torch.tensor(rng.permutation(T * columns).reshape(T, columns), dtype=torch.int32, device=DEV)
    bf = lambda *shape: torch.tensor(rng.standard_normal(shape), dtype=torch.bfloat16, device=DEV)
    cache, q = bf(T * columns, G, PAGE, dk + dv), bf(T, H, dk)
    bias = torch.tensor(rng.standard_normal((far + 1, H)), dtype=torch.float32, device=DEV)
    sink = torch.tensor(rng.standard_normal(H), dtype=torch.float32, device=DEV)
    scale = 1 / math.sqrt(dk)
    want = torch.empty((T, H, dv), dtype=torch.float64, device=DEV)
    for t, n in enumerate(lens):
        rows = torch.cat([cache[p] for p in table[t].tolist()], dim=1)[:, :n].double().repeat_interleave(per_kv, dim=0)
        score = torch.einsum("hd,hnd->hn", q[t].double(), rows[:, :, :dk]) * scale
        if cap:
            score = cap * torch.tanh(score / cap)
        d = n - 1 - torch.arange(n, device=DEV)
        score = score + bias.double()[d.clamp(max=far)].t()
        if window:
            score[:, (d >= window) & (torch.arange(n, device=DEV) >= keep)] = -math.inf
        p = torch.softmax(torch.cat([score, sink.double()[:, None]], dim=1), dim=1)[:, :n]
        want[t] = torch.einsum("hn,hnd->hd", p, rows[:, :, dk:])
    positions = torch.tensor([n - 1 for n in lens], dtype=torch.int32, device=DEV)
    seqs = torch.arange(T, dtype=torch.int32, device=DEV)
    for n_splits in (1, 2, 3, KB.heads_splits_for(T, G * -(-per_kv // 16), max(lens), dk + dv, q.device)):
        out = torch.full((T, H * dv), float("nan"), dtype=torch.bfloat16, device=DEV)
        KB.attention(q, cache, bias, sink, positions, seqs, table, PAGE, window, keep, scale, out, H, G, dk, dv, n_splits=n_splits,
                     bias_t=bias.t().contiguous(), softcap=cap)
        # the weights and the result are rounded to bfloat16 (2^-9 each, the weights' errors averaging out), sums are float32
        err = (out.view(T, H, dv).double() - want).norm() / want.norm()
        assert err < 2 * 2.0 ** -9, (n_splits, float(err))


@pytest.mark.parametrize("per_kv,dk,dv", [(4, 128, 128), (16, 64, 64)])
@pytest.mark.parametrize("n_splits", [1, 3])
def test_infinite_and_nan_values_stay_in_their_column(per_kv, dk, dv, n_splits):
    """A value of infinity makes its own element of the sums that infinity, a NaN a NaN, and nothing else changes: the weights reach the
    product in two parts, neither of which may turn an infinity round or meet it with a zero."""
    from turboquant_cpp_b200.kernels import bias_attention as KB
    g = torch.Generator(device=DEV).manual_seed(per_kv)
    n, G, H = 200, 2, 2 * per_kv
    cache = torch.randn((4, G, PAGE, dk + dv), generator=g, device=DEV).to(torch.bfloat16)
    q = torch.randn((1, H, dk), generator=g, device=DEV).to(torch.bfloat16)
    q[0, 0] = 0                                              # weights of exactly one: their second part is nothing
    i32 = lambda a: torch.tensor(a, dtype=torch.int32, device=DEV)

    def run():
        out = torch.empty((1, H * dv), dtype=torch.bfloat16, device=DEV)
        KB.attention(q, cache, None, None, i32([n - 1]), i32([0]), i32([[2, 0, 3, 1]]), PAGE, 0, 0, dk ** -0.5, out, H, G, dk, dv, n_splits=n_splits)
        return out.view(H, dv)

    clean = run()
    cache[0, :, 5, dk + 1], cache[0, :, 5, dk + 2], cache[0, :, 5, dk + 3] = math.inf, -math.inf, math.nan
    got = run()
    assert bool((got[:, 1] == math.inf).all()) and bool((got[:, 2] == -math.inf).all()) and bool(got[:, 3].isnan().all())
    assert torch.equal(got[:, 4:], clean[:, 4:]) and torch.equal(got[:, 0], clean[:, 0])
