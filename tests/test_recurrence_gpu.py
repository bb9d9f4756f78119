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
