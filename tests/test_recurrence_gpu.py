"""Recurrences in chunks of 64 tokens beside the token-by-token kernels, both against float64: runs around the chunks' edges,
sequences together, states that are not zero, decays from none to nearly total."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
RUNS = [[1], [63, 64, 65], [130, 2, 200, 64], [513]]


def i32(a):
    return torch.tensor(np.asarray(a), dtype=torch.int32, device=DEV)


def memory_reference(q, k, v, gates, S, n):
    """float64 over one run: outputs, n . q, final S [H, dk, dv] and n [H, dk]."""
    ys, ds = [], []
    for t in range(q.shape[0]):
        a, b = torch.exp(gates[t, :, 0]), torch.exp(gates[t, :, 1])
        S = S * a[:, None, None] + (b[:, None] * k[t])[:, :, None] * v[t][:, None]
        n = n * a[:, None] + b[:, None] * k[t]
        ys.append(torch.einsum("hkv,hk->hv", S, q[t]))
        ds.append((n * q[t]).sum(-1))
    return torch.stack(ys), torch.stack(ds), S, n


@pytest.mark.parametrize("dk,dv", [(64, 64), (64, 128), (128, 64), (128, 128)])
@pytest.mark.parametrize("runs", range(len(RUNS)))
@pytest.mark.parametrize("decay", [0.01, 3.0])
def test_memory_in_chunks(dk, dv, runs, decay):
    from turboquant_cpp_b200.kernels import recurrence as KR, ssm as KS
    H, lens = 3, RUNS[runs]
    T, g = sum(lens), torch.Generator(device=DEV).manual_seed(dk + dv + runs)
    rand = lambda *s: torch.randn(s, generator=g, device=DEV)
    rows = rand(T, H * (2 * dk + dv) + 8)
    gates = torch.stack([-decay * torch.rand((T, H), generator=g, device=DEV), -2.0 * rand(T, H).abs()], -1).contiguous()
    first = rand(len(lens), H, dv + 1, dk)
    cu, slots = i32(np.concatenate([[0], np.cumsum(lens)])), i32(np.arange(len(lens))[::-1].copy())
    out = {}
    for how in ("chunks", "tokens"):
        state, y, dots = first.clone(), torch.empty((T, H * dv), device=DEV), torch.empty((T, H), device=DEV)
        if how == "chunks":
            KR.memory_chunks(rows, 4, 4 + H * dk, 4 + 2 * H * dk, gates, state, y, dots, KR.chunks_of(lens, T, len(lens)) + 2, H, dk, dv, cu, slots)
        else:
            KS.memory_scan(rows, 4, 4 + H * dk, 4 + 2 * H * dk, gates, state, y, dots, H, dk, dv, cu, slots)
        out[how] = (y.view(T, H, dv), dots, state)
    err = {how: [0.0, 0.0, 0.0] for how in out}
    at = 0
    for s, n in enumerate(lens):
        r = rows[at:at + n].double()
        q, k, v = r[:, 4:4 + H * dk].view(n, H, dk), r[:, 4 + H * dk:4 + 2 * H * dk].view(n, H, dk), r[:, 4 + 2 * H * dk:4 + H * (2 * dk + dv)].view(n, H, dv)
        slot = int(slots[s])
        y, d, S, nn = memory_reference(q, k, v, gates[at:at + n].double(), first[slot, :, :dv].transpose(1, 2).double(), first[slot, :, dv].double())
        want = (y, d, torch.cat([S.transpose(1, 2), nn[:, None]], 1))
        for how, (gy, gd, gs) in out.items():
            for i, (a, b) in enumerate(zip((gy[at:at + n], gd[at:at + n], gs[slot]), want)):
                err[how][i] = max(err[how][i], float((a.double() - b).norm() / b.norm()))
        at += n
    for a, b in zip(err["chunks"], err["tokens"]):
        assert a < max(1.5 * b, 1e-6), err       # float32 sums in another order


def test_an_infinite_value_reaches_no_earlier_token():
    from turboquant_cpp_b200.kernels import recurrence as KR
    H, d, T = 1, 64, 100
    g = torch.Generator(device=DEV).manual_seed(5)
    rows = torch.randn((T, 3 * d), generator=g, device=DEV)
    gates = torch.full((T, H, 2), -0.1, device=DEV)
    res = []
    for bad in (False, True):
        if bad:
            rows[70, 2 * d:] = float("inf")
        state, y, dots = torch.zeros((1, H, d + 1, d), device=DEV), torch.empty((T, d), device=DEV), torch.empty((T, H), device=DEV)
        KR.memory_chunks(rows, 0, d, 2 * d, gates, state, y, dots, 2, H, d, d, i32([0, T]), i32([0]))
        res.append(y)
    assert torch.equal(res[0][:70], res[1][:70]) and not bool(torch.isfinite(res[1][70:]).any())


def memory_step(lens, H=2, dk=64, dv=64, scratch=None, monkeypatch=None):
    """(y, dots, state) of runs in chunks, and the bytes a step's scratch may take."""
    from turboquant_cpp_b200.kernels import recurrence as KR
    if scratch is not None:
        monkeypatch.setattr(KR, "SCRATCH_BYTES", scratch)
    T, g = sum(lens), torch.Generator(device=DEV).manual_seed(11)
    rows = torch.randn((T, H * (2 * dk + dv)), generator=g, device=DEV)
    gates = torch.stack([-0.2 * torch.rand((T, H), generator=g, device=DEV), -torch.rand((T, H), generator=g, device=DEV)], -1).contiguous()
    state = torch.randn((len(lens), H, dv + 1, dk), generator=g, device=DEV)
    y, dots = torch.empty((T, H * dv), device=DEV), torch.empty((T, H), device=DEV)
    torch.cuda.synchronize()
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.memory_allocated()
    KR.memory_chunks(rows, 0, H * dk, 2 * H * dk, gates, state, y, dots, KR.chunks_of(lens, T, len(lens)), H, dk, dv,
                     i32(np.concatenate([[0], np.cumsum(lens)])), i32(range(len(lens))))
    return (y, dots, state), torch.cuda.max_memory_allocated() - before


@pytest.mark.parametrize("lens", [[700], [64, 130, 1, 300, 63], [1] * 40 + [200]])
@pytest.mark.parametrize("at_once", [1, 2, 3, 7])
def test_groups_of_chunks(lens, at_once, monkeypatch):
    """The states of a few chunks at a time: the same bits, in as little scratch."""
    whole, _ = memory_step(lens)
    parts, _ = memory_step(lens, scratch=at_once * 4 * 2 * (65 * 64 + 1), monkeypatch=monkeypatch)
    assert all(torch.equal(a, b) for a, b in zip(whole, parts))


def test_the_scratch_of_a_long_run_is_bounded():
    from turboquant_cpp_b200.kernels import recurrence as KR
    _, used = memory_step([20000], H=8, dk=128, dv=128)           # 313 chunks of 0.5 MB
    assert used <= KR.SCRATCH_BYTES + (1 << 20), used


@pytest.mark.parametrize("n_seqs", [33, 70])
def test_many_sequences(n_seqs):
    """More sequences than a warp has lanes, some of one token and some of none: the token-by-token kernel's outputs and states."""
    from turboquant_cpp_b200.kernels import recurrence as KR, ssm as KS
    H, d = 2, 64
    lens = [(1, 70, 0, 3, 129, 64)[s % 6] for s in range(n_seqs)]
    T, g = sum(lens), torch.Generator(device=DEV).manual_seed(n_seqs)
    rows = torch.randn((T, 3 * H * d), generator=g, device=DEV)
    gates = torch.stack([-0.2 * torch.rand((T, H), generator=g, device=DEV), -torch.rand((T, H), generator=g, device=DEV)], -1).contiguous()
    first = torch.randn((n_seqs, H, d + 1, d), generator=g, device=DEV)
    cu, slots = i32(np.concatenate([[0], np.cumsum(lens)])), i32(np.arange(n_seqs)[::-1].copy())
    out = []
    for how in ("chunks", "tokens"):
        state, y, dots = first.clone(), torch.empty((T, H * d), device=DEV), torch.empty((T, H), device=DEV)
        if how == "chunks":
            KR.memory_chunks(rows, 0, H * d, 2 * H * d, gates, state, y, dots, KR.chunks_of(lens, T, n_seqs), H, d, d, cu, slots)
        else:
            KS.memory_scan(rows, 0, H * d, 2 * H * d, gates, state, y, dots, H, d, d, cu, slots)
        out.append((y, dots, state))
    for a, b in zip(*out):
        assert float((a - b).norm() / b.norm()) < 1e-5            # float32 sums of some hundred terms in another order
    for s, n in enumerate(lens):
        if n == 0:
            assert torch.equal(out[0][2][slots[s]], first[slots[s]])


@pytest.mark.parametrize("d", [64, 128])
def test_a_memory_layer_continues_its_runs(d, monkeypatch):
    """The layer's own choice of form, in steps that follow one another: a chunked prompt goes on in another portion (walked or
    chunked) and in steps of single tokens as the walk alone does."""
    from turboquant_cpp_b200.parts import LayerCache, StepContext, chunks, make_mixer
    from turboquant_cpp_b200.weights import RandomSource, WeightStore
    H, n_seqs = 4, 3
    m = make_mixer("matrix_memory", prefix="", hidden=256, heads=H, dim=d, vdim=d, gate_cap=20.0, eps=1e-5)
    m.run_dtype = torch.float32
    m.bind(WeightStore(RandomSource(m.weight_specs(), d, std=0.05), m.weight_specs(), DEV, torch.float32))
    steps = [[700, 30, 1], [130, 1, 64], [200, 700, 700], [1, 1, 1], [90, 2, 60]]
    g = torch.Generator(device=DEV).manual_seed(d)
    xs = [torch.randn((sum(lens), 256), generator=g, device=DEV) for lens in steps]
    got, forms = {}, []
    for how in ("own", "walk"):
        if how == "walk":
            monkeypatch.setattr(type(m), "_in_chunks", lambda self, ctx, cuts: False)
        need = m.state_need()
        cache = LayerCache(page_size=64)
        cache.state = torch.zeros((n_seqs,) + tuple(need.shape), dtype=need.dtype, device=DEV)
        held, got[how] = np.zeros(n_seqs, dtype=np.int64), []
        for lens, x in zip(steps, xs):
            cu = np.concatenate([[0], np.cumsum(lens)])
            seq_of = np.repeat(np.arange(n_seqs), lens)
            pos = np.arange(cu[-1]) - cu[:-1][seq_of] + held[seq_of]
            ctx = StepContext(n_tokens=int(cu[-1]), n_seqs=n_seqs, tokens=i32(pos), positions=i32(pos), seq_of_token=i32(seq_of), cu_seqlens=i32(cu),
                              seq_start=i32(held), slots=i32(range(n_seqs)), want_rows=i32([]), n_want=0, max_q_len=max(lens),
                              max_kv_len=int((held + lens).max()), act_dtype=torch.float32, device=torch.device(DEV), host_q_lens=list(lens),
                              host_slots=list(range(n_seqs)), host_seq_start=[int(h) for h in held], status=torch.zeros(1, dtype=torch.int32, device=DEV))
            ctx.carry = {}
            if how == "own":
                forms.append(max(lens) > 1 and m._in_chunks(ctx, chunks.cut_size(ctx, H, d + 1) is not None))
            got[how].append(m.forward(x, ctx, cache))
            held = held + lens
        got[how].append(cache.state)
    assert forms[0] and forms[2] and not forms[3]
    for a, b in zip(got["own"], got["walk"]):
        assert float((a - b).norm() / b.norm()) < 2e-5            # float32 sums in another order, through norm and closing product
