"""The rotating writer of cache rows and the gate that turns values back, over the shapes their launches split differently: a head a
warp over several blocks, a block per token with sixteen or eight warps, heads in registers and in shared memory, values too long
for either, with and without norms; against float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
SHAPES = [  # tokens, heads, key/value heads, key size, value size, rotated elements, halves, values turned, norms
    (1, 64, 8, 128, 128, 128, True, True, True),
    (3, 5, 1, 128, 64, 32, False, True, True),
    (2, 3, 3, 36, 20, 6, False, False, False),
    (16, 33, 11, 64, 64, 64, True, True, False),
    (60, 64, 8, 128, 128, 64, False, True, True),          # 4,800 heads: more than a warp each
    (592, 16, 4, 128, 128, 128, True, True, True),
    (593, 16, 4, 128, 128, 128, True, True, True),
    (700, 20, 2, 200, 130, 40, True, True, True),          # through shared memory
    (650, 3, 1, 33, 7, 10, False, False, True),            # unaligned rows
    (2, 2, 1, 64, 300, 64, True, True, False),
    (2, 2, 1, 64, 12800, 64, False, True, True),           # 50 KB a value
]


def turned(x, pos, freq, halves):
    """x float64 [T, heads, n]: its first 2 len(freq) elements turned by the float32 products pos * freq."""
    n = freq.shape[0]
    a = (pos.float()[:, None] * freq).double()[:, None]
    i = torch.arange(n, device=x.device)
    u, v = (i, i + n) if halves else (2 * i, 2 * i + 1)
    y = x.clone()
    y[..., u], y[..., v] = x[..., u] * torch.cos(a) - x[..., v] * torch.sin(a), x[..., v] * torch.cos(a) + x[..., u] * torch.sin(a)
    return y


def close(got, want):
    # a norm, a rotation and a factor in float32: some ten roundings of 2^-24, the sine's and cosine's two of 2^-23
    mag = want.abs().amax(-1, keepdim=True)
    assert bool(((got.double() - want).abs() <= 2.0 ** -20 * mag + 1e-7).all()), float(((got.double() - want).abs() / mag.clamp_min(1e-30)).max())


@pytest.mark.parametrize("shape", SHAPES)
def test_rotating_writer(shape):
    from turboquant_cpp_b200.kernels import bias_attention as KB
    T, H, G, dk, dv, dims, halves, turn, norms = shape
    g = torch.Generator(device=DEV).manual_seed(T + H)
    rand = lambda *s: torch.randn(s, generator=g, device=DEV)
    rows, pos = rand(T, H * dk + G * (dk + dv)), torch.randint(0, 300, (T,), generator=g, device=DEV, dtype=torch.int32)
    freq, v_freq = torch.rand(dims // 2, generator=g, device=DEV), torch.rand(dv // 2, generator=g, device=DEV) if turn else None
    qw, kw = (1 + 0.1 * rand(dk), 1 + 0.1 * rand(dk)) if norms else (None, None)
    page = torch.randperm(5 * T, generator=torch.Generator().manual_seed(1)).to(DEV)       # five pages of 64 a token
    q, cache = torch.empty((T, H, dk), device=DEV), torch.zeros((5 * T, 1, G, 64, dk + dv), device=DEV) if dv < 12800 else None
    table = page.to(torch.int32).view(T, 5)
    if cache is None:                      # one page: all tokens at different places of it
        pos = torch.arange(T, device=DEV, dtype=torch.int32)
        table, cache = torch.zeros((T, 1), dtype=torch.int32, device=DEV), torch.zeros((1, 1, G, 64, dk + dv), device=DEV)
    KB.kv_write_rot(rows, q, cache, freq, dims, halves, 1e-5, pos, torch.arange(T, device=DEV, dtype=torch.int32), table, 64, H, G, dk, dv,
                    mag=1.1, q_norm=qw, k_norm=kw, norm_eps=1e-5, v_freq=v_freq)
    x = rows.double()
    heads = [x[:, :H * dk].view(T, H, dk), x[:, H * dk:(H + G) * dk].view(T, G, dk)]
    for i, w in enumerate((qw, kw)):
        if norms:
            heads[i] = heads[i] / torch.sqrt(heads[i].square().mean(-1, keepdim=True) + 1e-5) * w.double()
        rest = heads[i][..., dims:]
        heads[i] = torch.cat([turned(heads[i], pos, freq, halves)[..., :dims] * 1.1, rest], -1)
        heads[i] = heads[i] / torch.sqrt(heads[i].square().mean(-1, keepdim=True) + 1e-5)
    v = x[:, (H + G) * dk:].view(T, G, dv)
    close(q, heads[0])
    at = cache[table.long()[torch.arange(T, device=DEV), pos.long() // 64], 0, :, pos.long() % 64]
    close(at[..., :dk], heads[1])
    close(at[..., dk:], turned(v, pos, v_freq, halves) if turn else v)


@pytest.mark.parametrize("shape", [s for s in SHAPES if s[4] <= 256])
def test_values_turned_back(shape):
    from turboquant_cpp_b200.kernels import bias_attention as KB
    T, H, _, _, dv, _, halves, turn, _ = shape
    g = torch.Generator(device=DEV).manual_seed(T + H)
    o, gates = torch.randn((T, H * dv), generator=g, device=DEV), torch.randn((T, H + 3), generator=g, device=DEV)
    pos = torch.randint(0, 300, (T,), generator=g, device=DEV, dtype=torch.int32)
    freq = torch.rand(dv // 2, generator=g, device=DEV) if turn else None
    want = o.double().view(T, H, dv)
    want = (turned(want, -pos, freq, halves) if turn else want) * torch.sigmoid(gates[:, 2:2 + H].double())[..., None]
    close(KB.heads_unrotate_gate(o, gates, 2, freq, halves, pos, o, H, dv).view(T, H, dv), want)
