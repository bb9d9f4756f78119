"""Latent attention's prompts over keys and values built from the cached rows, beside the path over the rows themselves: both
against float64, for ragged steps that hold earlier positions, with and without rotated parts, windows and sinks."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
CASES = [  # heads, dim, rot, vdim, rank, window, sink, runs, held
    (16, 128, 64, 128, 512, 0, True, [300], [0]),
    (4, 128, 64, 128, 256, 100, True, [129, 64, 1, 260], [0, 500, 70, 63]),
    (3, 64, 64, 64, 128, 0, False, [33, 128], [90, 0]),
    (8, 128, 0, 128, 512, 0, False, [257, 40], [0, 129]),
    (2, 64, 0, 128, 64, 64, False, [200], [200]),
]


def reference(m, x, held_rows, runs, held, weights, eps):
    """float64 layer output, from the weights by name."""
    H, R = m.heads, m.kv_rank
    w = lambda n: weights[n].double()
    freq = None if m.position is None else m.position._freq64.to(x.device)

    def turn(a, pos):
        if freq is None:
            return a
        ang = pos.double()[:, None, None] * freq
        c, s = torch.cos(ang) * m.position.mag, torch.sin(ang) * m.position.mag
        out = a.clone()
        n = 2 * freq.shape[0]
        out[..., 0:n:2], out[..., 1:n:2] = a[..., 0:n:2] * c - a[..., 1:n:2] * s, a[..., 1:n:2] * c + a[..., 0:n:2] * s
        return out
    outs, at = [], 0
    for n, h, old in zip(runs, held, held_rows):
        xs, pos = x[at:at + n].double(), torch.arange(h, h + n, device=x.device)
        at += n
        q = (xs @ w("q").t()).view(n, H, m.q_dim)
        q = torch.cat([q[..., :m.dim], turn(q[..., m.dim:], pos)], -1)
        d = xs @ w("dkv").t()
        c = d[:, :R] / torch.sqrt(d[:, :R].square().mean(1, keepdim=True) + eps) * w("dkv.norm")
        rows = torch.cat([old.double(), torch.cat([c, turn(d[:, None, R:], pos)[:, 0]], 1)])
        k = torch.cat([(rows[:, :R] @ w("uk").t()).view(-1, H, m.dim), rows[:, None, R:].expand(-1, H, -1)], -1)
        v = (rows[:, :R] @ w("uv").t()).view(-1, H, m.vdim)
        i, j = pos[:, None], torch.arange(h + n, device=x.device)[None]
        see = (j <= i) & ((i - j < m.window) if m.window else True)
        s = torch.einsum("nhd,mhd->hnm", q, k) * m.scale
        s = s.masked_fill(~see, -float("inf"))
        if m.has_sink:
            p = torch.softmax(torch.cat([s, w("sink")[:, None, None].expand(H, n, 1)], 2), 2)[..., :-1]
        else:
            p = torch.softmax(s, 2)
        outs.append(torch.einsum("hnm,mhd->nhd", p, v).reshape(n, -1) @ w("o").t())
    return torch.cat(outs)


def layer_and_step(case, seed, unused=0.0):
    """(mixer, weights by name, input rows, the held rows, the step, its cache, whose slots that no position has taken hold `unused`)."""
    from turboquant_cpp_b200.parts import LayerCache, StepContext, make_mixer, make_position_encoding
    from turboquant_cpp_b200.weights import RandomSource, WeightStore
    H, dim, rot, vdim, R, window, sink, runs, held = case
    pe = make_position_encoding("rotary_scaled", dims=rot, base=10000.0, factor=2.0, original=128, fast=8.0, slow=1.0) if rot else None
    m = make_mixer("latent_attention", prefix="", hidden=256, heads=H, dim=dim, rot_dim=rot, vdim=vdim, kv_rank=R, scale=(dim + rot) ** -0.5,
                   eps=1e-5, window=window, position=pe, sink=sink)
    m.run_dtype = torch.bfloat16
    source = RandomSource(m.weight_specs(), seed, std=0.06)
    m.bind(WeightStore(source, m.weight_specs(), DEV, torch.bfloat16))
    weights = {s.name: source.read(s.name, DEV) for s in m.weight_specs()}
    g = torch.Generator(device=DEV).manual_seed(seed)
    total = [n + h for n, h in zip(runs, held)]
    counts = [-(-t // 64) for t in total]
    order = torch.randperm(sum(counts), generator=torch.Generator().manual_seed(seed)).split(counts)
    kv = torch.full((sum(counts), 1, 1, 64, R + rot), unused, dtype=torch.bfloat16, device=DEV)
    table = torch.full((len(runs), max(counts)), -1, dtype=torch.int32)
    old = []
    for i, h in enumerate(held):
        table[i, :counts[i]] = order[i].to(torch.int32)
        old.append(torch.randn((h, R + rot), generator=g, device=DEV).to(torch.bfloat16))
        at = torch.arange(h, device=DEV)
        kv[order[i].to(DEV)[at // 64], 0, 0, at % 64] = old[i]
    x = torch.randn((sum(runs), 256), generator=g, device=DEV).to(torch.bfloat16)
    cu = np.concatenate([[0], np.cumsum(runs)])
    seq_of = np.repeat(np.arange(len(runs)), runs)
    pos = np.arange(cu[-1]) - cu[:-1][seq_of] + np.asarray(held)[seq_of]
    i32 = lambda a: torch.tensor(np.asarray(a), dtype=torch.int32, device=DEV)
    ctx = StepContext(n_tokens=int(cu[-1]), n_seqs=len(runs), tokens=i32(pos), positions=i32(pos), seq_of_token=i32(seq_of), cu_seqlens=i32(cu),
                      seq_start=i32(held), slots=i32(range(len(runs))), want_rows=i32([]), n_want=0, max_q_len=max(runs), max_kv_len=max(total),
                      act_dtype=torch.bfloat16, device=torch.device(DEV), host_q_lens=runs, host_seq_start=held,
                      status=torch.zeros(1, dtype=torch.int32, device=DEV))
    return m, weights, x, old, ctx, LayerCache(kv=kv, page_table=table.to(DEV), page_size=64)


@pytest.mark.parametrize("case", range(len(CASES)))
def test_expanded_prompts(case, monkeypatch):
    runs, held = CASES[case][-2:]
    m, weights, x, old, ctx, cache = layer_and_step(CASES[case], case)
    want = reference(m, x, old, runs, held, weights, 1e-5)
    err = {}
    for per_token in (1 << 20, 0):       # always expanded, never
        monkeypatch.setattr(type(m), "EXPAND_KEYS_PER_TOKEN", per_token)
        assert m._expands(ctx, cache) == bool(per_token)
        err[per_token] = float((m.forward(x, ctx, cache).double() - want).norm() / want.norm())
    assert int(ctx.status.item()) == 0
    # the same number of roundings to bfloat16 on either path (queries, keys, values and weights here; queries in the latent
    # space, weights and weighted latents there): neither may be further off than half as much again
    assert err[1 << 20] < 1.5 * err[0] and err[1 << 20] < 8e-3, err


@pytest.mark.parametrize("case", range(len(CASES)))
@pytest.mark.parametrize("unused", [float("nan"), float("inf"), 3e38])
def test_slots_that_no_position_has_taken_are_never_seen(case, unused, monkeypatch):
    """A page keeps what its last owner left behind the new one's end: the same bits whatever that is."""
    got = []
    for fill in (0.0, unused):
        m, _, x, _, ctx, cache = layer_and_step(CASES[case], case, fill)
        monkeypatch.setattr(type(m), "EXPAND_KEYS_PER_TOKEN", 1 << 20)
        assert m._expands(ctx, cache)
        got.append(m.forward(x, ctx, cache))
    assert torch.equal(got[0], got[1]) and bool(torch.isfinite(got[0]).all())


def test_sequences_without_new_tokens(monkeypatch):
    """Host and kernel count the same pages where a run is empty: the others' rows are those of the step without it."""
    got = []
    for runs, held in (([130, 70], [0, 40]), ([0, 130, 0, 70], [0, 0, 100, 40]), ([0, 130, 0, 70, 0], [0, 0, 0, 40, 0])):
        m, _, x, old, ctx, cache = layer_and_step((4, 128, 64, 128, 128, 0, False, runs, held), 5)
        live = [i for i, n in enumerate(runs) if n]
        if not got:
            rows, inputs = [old[i] for i in live], x
        else:                              # the same held rows and inputs in the wider step's pages
            for i, r in zip(live, rows):
                at = torch.arange(r.shape[0], device=DEV)
                cache.kv[cache.page_table[i].long()[at // 64], 0, 0, at % 64] = r
        monkeypatch.setattr(type(m), "EXPAND_KEYS_PER_TOKEN", 1 << 20)
        assert m._expands(ctx, cache)
        got.append(m.forward(inputs, ctx, cache))
    assert all(torch.equal(got[0], g) for g in got[1:])


@pytest.mark.parametrize("n_seqs", [33, 70])
def test_many_sequences(n_seqs, monkeypatch):
    """More sequences than a warp has lanes: each finds its own pages among the gathered ones."""
    runs = [(1, 40, 3, 70)[s % 4] for s in range(n_seqs)]
    held = [(0, 64, 129, 5, 63)[s % 5] for s in range(n_seqs)]
    m, weights, x, old, ctx, cache = layer_and_step((3, 64, 64, 128, 128, 0, True, runs, held), n_seqs)
    monkeypatch.setattr(type(m), "EXPAND_KEYS_PER_TOKEN", 1 << 20)
    assert m._expands(ctx, cache)
    want = reference(m, x, old, runs, held, weights, 1e-5)
    got = m.forward(x, ctx, cache).double()
    assert float((got - want).norm() / want.norm()) < 8e-3        # as above
    # no sequence may hide behind the others' rows
    for a, b in zip(got.split(runs), want.split(runs)):
        assert float((a - b).norm() / b.norm()) < 2e-2
