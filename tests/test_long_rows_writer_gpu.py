"""The rotating writer and the turned-back gate on long steps, where a warp has a token's heads or some of them: numbers of heads that are
no multiple of four, shared values, values that are the keys, a temperature, no cache, short heads; against float64."""
import pytest
import torch

from test_rows_writer_gpu import DEV, close, turned

pytestmark = pytest.mark.gpu
SHAPES = [  # tokens, heads, key/value heads, key size, value size, rotated elements, halves, value heads shared by, values are keys
    (1, 700, 9, 128, 128, 128, True, 1, False),
    (600, 11, 3, 64, 128, 32, False, 3, False),
    (2049, 5, 1, 128, 128, 64, True, 1, True),
    (8200, 6, 2, 100, 36, 16, True, 2, False),
]


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("cached", [True, False])
def test_writer(shape, cached):
    from turboquant_cpp_b200.kernels import bias_attention as KB
    T, H, G, dk, dv, dims, halves, share, v_is_k = shape
    g = torch.Generator(device=DEV).manual_seed(T)
    rand = lambda *s: torch.randn(s, generator=g, device=DEV)
    n_v = 0 if v_is_k else G // share * dv
    rows, pos = rand(T, H * dk + G * dk + n_v + 4), torch.randperm(T, generator=g, device=DEV).to(torch.int32) + 3
    turn = dv % 8 == 0 and not v_is_k
    freq, v_freq = torch.rand(dims // 2, generator=g, device=DEV), torch.rand(dv // 2, generator=g, device=DEV) if turn else None
    qw, kw = 1 + 0.1 * rand(dk), 1 + 0.1 * rand(dk)
    pages = -(-(T + 3) // 64)
    table = torch.randperm(pages, generator=torch.Generator().manual_seed(1)).to(DEV, torch.int32).view(1, pages)
    q, cache = torch.empty((T, H, dk), device=DEV), torch.zeros((pages, 1, G, 64, dk + dv), device=DEV)
    KB.kv_write_rot(rows, q, cache if cached else None, freq, dims, halves, 1e-5, pos, torch.zeros(T, device=DEV, dtype=torch.int32), table, 64, H, G, dk, dv,
                    mag=1.1, q_norm=qw, k_norm=kw, norm_eps=1e-5, v_freq=v_freq, v_share=share, values_are_keys=v_is_k, temperature=(0.1, 50))
    x = rows.double()
    heads = [x[:, :H * dk].view(T, H, dk), x[:, H * dk:(H + G) * dk].view(T, G, dk)]
    raw = heads[1]
    for i, w in enumerate((qw, kw)):
        heads[i] = heads[i] / torch.sqrt(heads[i].square().mean(-1, keepdim=True) + 1e-5) * w.double()
        heads[i] = torch.cat([turned(heads[i], pos, freq, halves)[..., :dims] * 1.1, heads[i][..., dims:]], -1)
        heads[i] = heads[i] / torch.sqrt(heads[i].square().mean(-1, keepdim=True) + 1e-5)
    close(q, heads[0] * (1 + 0.1 * torch.log(((pos + 1) // 50).double() + 1))[:, None, None])
    if cached:
        v = raw if v_is_k else x[:, (H + G) * dk:(H + G) * dk + n_v].view(T, G // share, dv).repeat_interleave(share, 1)
        at = cache[table[0].long()[pos.long() // 64], 0, :, pos.long() % 64]
        close(at[..., :dk], heads[1])
        close(at[..., dk:], turned(v, pos, v_freq, halves) if turn else v)


@pytest.mark.parametrize("T,H,dv,halves", [(1792, 7, 128, True), (2000, 3, 36, False), (5000, 18, 64, True)])
def test_values_turned_back(T, H, dv, halves):
    from turboquant_cpp_b200.kernels import bias_attention as KB
    g = torch.Generator(device=DEV).manual_seed(T)
    o, gates, freq = torch.randn((T, H * dv), generator=g, device=DEV), torch.randn((T, H + 3), generator=g, device=DEV), torch.rand(dv // 2, generator=g, device=DEV)
    pos = torch.randint(0, 300, (T,), generator=g, device=DEV, dtype=torch.int32)
    want = turned(o.double().view(T, H, dv), -pos, freq, halves) * torch.sigmoid(gates[:, 2:2 + H].double())[..., None]
    close(KB.heads_unrotate_gate(o, gates, 2, freq, halves, pos, o, H, dv).view(T, H, dv), want)


@pytest.mark.parametrize("halves", [True, False])
@pytest.mark.parametrize("dk,dv,dims", [(128, 128, 128), (96, 64, 32)])
def test_a_token_s_rows_do_not_depend_on_the_step_s_size(halves, dk, dv, dims):
    """The kernels of long steps and of small ones write the same bits."""
    from turboquant_cpp_b200.kernels import bias_attention as KB
    H, G, T, part = 6, 2, 1800, 50
    g = torch.Generator(device=DEV).manual_seed(dk)
    rand = lambda *s: torch.randn(s, generator=g, device=DEV)
    rows, pos = rand(T, (H + G) * dk + G * dv), torch.arange(T, device=DEV, dtype=torch.int32)
    freq, v_freq, qw, kw = rand(dims // 2).abs(), rand(dv // 2).abs(), 1 + 0.1 * rand(dk), 1 + 0.1 * rand(dk)
    o, gates = rand(T, H * dv), rand(T, H)
    pages = -(-T // 64)
    table = torch.arange(pages, device=DEV, dtype=torch.int32).view(1, pages)

    def run(steps):
        cache, out = torch.zeros((pages, 1, G, 64, dk + dv), device=DEV), []
        for a in range(0, T, steps):
            n = slice(a, a + steps)
            q = torch.empty((rows[n].shape[0], H, dk), device=DEV)
            KB.kv_write_rot(rows[n], q, cache, freq, dims, halves, 1e-5, pos[n], torch.zeros_like(pos[n]), table, 64, H, G, dk, dv, mag=1.1, q_norm=qw,
                            k_norm=kw, norm_eps=1e-5, v_freq=v_freq, temperature=(0.1, 50))
            out.append(torch.cat([q.flatten(1), KB.heads_unrotate_gate(o[n], gates[n], 0, v_freq, halves, pos[n], torch.empty_like(o[n]), H, dv)], 1))
        return torch.cat(out), cache

    for a, b in zip(run(T), run(part)):
        assert torch.equal(a, b)
