"""The delta rule with one decay per head in chunks of 64 tokens as matrix products, beside the token-by-token kernels, both against float64:
runs around the chunks' edges, shared query/key heads, states that are not zero, keys that resemble each other, decays from none to
nearly total, steps in several groups of chunks, tokens that are not finite, and the rule that chooses the form."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
EPS = 1e-6
RUNS = [[1], [63, 64, 65], [130, 0, 2, 200], [513]]


def i32(a):
    return torch.tensor(np.asarray(a), dtype=torch.int32, device=DEV)


def data(lens, H, G, dk, dv, alike=0.0, decay=0.0, seed=0):
    """(rows of q | k | v behind four columns, projection with betas and raw decays, bias, rates, first states)"""
    g = torch.Generator(device=DEV).manual_seed(seed)
    r = lambda *s: torch.randn(s, generator=g, device=DEV)
    T, n = sum(lens), 2 * G * dk
    x = torch.cat([r(T, 4), alike * r(1, n) + (1 - alike) * r(T, n), r(T, H * dv)], 1).contiguous()
    return x, torch.cat([r(T, 3), 2 * r(T, H), decay + r(T, H)], 1).contiguous(), r(H), r(H), r(len(lens), H, dv, dk)


def reference(d, lens, H, G, dk, dv, slots):
    x, p, bias, rate, first = (t.double() for t in d)
    unit = lambda a: a / torch.sqrt(a.square().sum(-1, keepdim=True) + EPS)
    heads = lambda a: unit(a.reshape(-1, G, dk)).repeat_interleave(H // G, 1)
    q, k, v = heads(x[:, 4:4 + G * dk]) * dk ** -0.5, heads(x[:, 4 + G * dk:4 + 2 * G * dk]), x[:, 4 + 2 * G * dk:].reshape(-1, H, dv)
    beta, g = torch.sigmoid(p[:, 3:3 + H]), torch.exp(-torch.exp(rate) * torch.nn.functional.softplus(p[:, 3 + H:] + bias))
    y, state, at = torch.empty_like(v), first.clone(), 0
    for s, n in enumerate(lens):
        S = first[slots[s]]
        for t in range(at, at + n):
            S = S * g[t][:, None, None]
            u = beta[t][:, None] * (v[t] - torch.einsum("hvk,hk->hv", S, k[t]))
            S = S + u[:, :, None] * k[t][:, None]
            y[t] = torch.einsum("hvk,hk->hv", S, q[t])
        state[slots[s]] = S
        at += n
    return y.reshape(-1, H * dv), state


def run(form, d, lens, H, G, dk, dv, slots):
    from turboquant_cpp_b200.kernels import recurrence as KR, ssm as KS
    from turboquant_cpp_b200.kernels.gemm_tc import check_status
    x, p, bias, rate, first = d
    T, cu, state = sum(lens), i32(np.concatenate([[0], np.cumsum(lens)])), first.clone()
    y = torch.full((T, H * dv), float("nan"), device=DEV)
    args = (x, 4, 4 + G * dk, 4 + 2 * G * dk, p, 3, p, 3 + H, bias, rate, state, y)
    if form == "chunks":
        KR.delta_chunks(*args, KR.chunks_of(lens, T, len(lens)) + 2, H, G, dk, dv, EPS, dk ** -0.5, cu, i32(slots))
        check_status()
    else:
        KS.delta_scan_runs(*args, H, G, dk, dv, EPS, dk ** -0.5, cu, i32(slots))
    return y, state


@pytest.mark.parametrize("dk,dv", [(64, 64), (64, 128), (128, 64), (128, 128)])
@pytest.mark.parametrize("runs", range(len(RUNS)))
@pytest.mark.parametrize("alike,decay", [(0.0, -2.0), (0.7, -8.0), (0.0, 3.0)])
def test_against_float64(dk, dv, runs, alike, decay):
    lens, H, G = RUNS[runs], 4, 4 if dk == dv else 2
    slots = list(range(len(lens)))[::-1]
    d = data(lens, H, G, dk, dv, alike, decay, dk + dv + runs)
    want = reference(d, lens, H, G, dk, dv, slots)
    err = {form: [float((a.double() - b).norm() / b.norm()) for a, b in zip(run(form, d, lens, H, G, dk, dv, slots), want)] for form in ("chunks", "walk")}
    for a, b in zip(err["chunks"], err["walk"]):          # both are float32 sums in some order: of one size
        assert a <= 1.25 * b + 2.0 ** -25, err


def test_groups_of_chunks(monkeypatch):
    from turboquant_cpp_b200.kernels import recurrence as KR
    lens, H, G, dk, dv = [300, 70, 129], 2, 1, 128, 64
    d = data(lens, H, G, dk, dv)
    whole = run("chunks", d, lens, H, G, dk, dv, [2, 0, 1])
    monkeypatch.setattr(KR, "SCRATCH_BYTES", 2 * KR.delta_bytes(1, H, G, dk, dv))
    for a, b in zip(whole, run("chunks", d, lens, H, G, dk, dv, [2, 0, 1])):
        assert torch.equal(a, b)


@pytest.mark.parametrize("what", ["key", "value", "beta", "decay", "query"])
@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_a_token_that_is_not_finite(what, bad):
    """Earlier tokens and other heads are what they were; the token and, but for a query, all behind it and the state are not finite, of a
    value its own column alone.  Token by token the same places are lost."""
    lens, H, G, dk, dv, at = [200, 90], 2, 2, 64, 64, 77
    d = data(lens, H, G, dk, dv)
    clean = run("chunks", d, lens, H, G, dk, dv, [0, 1])
    x, p = d[0], d[1]
    if what == "beta" or what == "decay":
        p[at, 3 if what == "beta" else 3 + H] = float("nan")
    else:
        x[at, 4 + {"query": 0, "key": G * dk, "value": 2 * G * dk}[what] + 5] = bad
    y, state = run("chunks", d, lens, H, G, dk, dv, [0, 1])
    y, was = y.view(-1, H, dv), clean[0].view(-1, H, dv)
    assert torch.equal(y[:at], was[:at]) and torch.equal(y[:, 1], was[:, 1]) and torch.equal(y[200:], was[200:])
    assert torch.equal(state[0, 1], clean[1][0, 1]) and torch.equal(state[1], clean[1][1])
    lost, lost_state = torch.zeros_like(y[:, 0], dtype=torch.bool), torch.zeros_like(state[0, 0], dtype=torch.bool)
    tokens, columns = slice(at, at + 1 if what == "query" else 200), slice(5, 6) if what == "value" else slice(None)
    lost[tokens, columns] = True
    if what != "query":
        lost_state[columns] = True
    assert not bool(y[:, 0][lost].isfinite().any()) and torch.equal(y[:, 0][~lost], was[:, 0][~lost])
    assert not bool(state[0, 0][lost_state].isfinite().any()) and torch.equal(state[0, 0][~lost_state], clean[1][0, 0][~lost_state])
    walked, walked_state = run("walk", d, lens, H, G, dk, dv, [0, 1])
    assert torch.equal(walked.isfinite(), y.isfinite().view(walked.shape)) and torch.equal(walked_state.isfinite(), state.isfinite())


@pytest.mark.parametrize("dk,dv", [(64, 128), (128, 128)])
def test_values_that_are_not_finite_in_several_columns_and_chunks(dk, dv):
    """Both ends of a value, several tokens of one chunk and another chunk's first and last token."""
    lens, H, G = [330], 2, 1
    d = data(lens, H, G, dk, dv)
    clean = run("chunks", d, lens, H, G, dk, dv, [0])
    places = [(0, 1), (63, 0), (64, 17), (70, dv - 1), (66, 40), (100, 40), (127, 33), (329, 2)]
    for t, c in places:
        d[0][t, 4 + 2 * G * dk + dv + c] = float("nan")           # the second head
    y, state = run("chunks", d, lens, H, G, dk, dv, [0])
    y, was, lost = y.view(-1, H, dv), clean[0].view(-1, H, dv), torch.zeros((330, H, dv), dtype=torch.bool, device=DEV)
    for t, c in places:
        lost[t:, 1, c] = True
    assert bool(y[lost].isnan().all()) and torch.equal(y[~lost], was[~lost])
    assert bool(state[0][lost[-1]].isnan().all()) and torch.equal(state[0][~lost[-1]], clean[1][0][~lost[-1]])


def test_which_steps_go_in_chunks():
    from turboquant_cpp_b200.parts.delta import HeadDeltaMixer
    from types import SimpleNamespace
    m = HeadDeltaMixer("", 2048, 16, 16, 128, 128, 4, 1e-5)
    step = lambda lens: SimpleNamespace(host_q_lens=lens, n_tokens=sum(lens), n_seqs=len(lens), max_q_len=max(lens))
    assert m._in_chunks(step([2048])) and m._in_chunks(step([1000, 1048])) and m._in_chunks(step([8192]))
    assert not m._in_chunks(step([64])) and not m._in_chunks(step([200])) and not m._in_chunks(step([2048] + [1] * 63)) and not m._in_chunks(step([2] * 64))


@pytest.mark.parametrize("what", ["query", "key", "value"])
@pytest.mark.parametrize("dk,dv", [(64, 64), (128, 64), (128, 128)])
def test_a_matrix_memory_s_token_that_is_not_finite(what, dk, dv):
    """In chunks a token's output depends on no later token, other heads on neither, and a value reaches its own column only.  Token by
    token the same places are lost."""
    from turboquant_cpp_b200.kernels import recurrence as KR, ssm as KS
    H, lens, at, column = 2, [150, 70], 77, 35
    g = torch.Generator(device=DEV).manual_seed(1)
    rows, gates = torch.randn((220, H * (2 * dk + dv)), generator=g, device=DEV), -torch.rand((220, H, 2), generator=g, device=DEV)
    new = lambda: (torch.ones((2, H, dv + 1, dk), device=DEV), torch.empty((220, H * dv), device=DEV), torch.empty((220, H), device=DEV))
    offsets, cu, slots, out = (0, H * dk, 2 * H * dk), i32([0, 150, 220]), i32([0, 1]), []
    for bad in (0.5, float("nan"), float("inf")):
        rows[at, {"query": 0, "key": H * dk, "value": 2 * H * dk}[what] + column] = bad
        if bad != 0.5:
            rows[100, 2 * H * dk + 40] = bad                      # the same chunk, another column
        (state, y, dots), (w_state, w_y, w_dots) = new(), new()
        KR.memory_chunks(rows, *offsets, gates, state, y, dots, KR.chunks_of(lens, 220, 2), H, dk, dv, cu, slots)
        KS.memory_scan(rows, *offsets, gates, w_state, w_y, w_dots, H, dk, dv, cu, slots)
        for a, b in ((y, w_y), (dots, w_dots), (state, w_state)):
            assert torch.equal(a.isfinite(), b.isfinite())
        out.append((y.view(220, H, dv), dots, state))
    lost = torch.zeros_like(out[0][0], dtype=torch.bool)
    lost[at:at + 1 if what == "query" else 150, 0, slice(column, column + 1) if what == "value" else slice(None)] = True
    lost[100:150, 0, 40] = True
    lost_dots, lost_state = torch.zeros_like(out[0][1], dtype=torch.bool), torch.zeros_like(out[0][2], dtype=torch.bool)
    if what != "value":
        lost_dots[at:at + 1 if what == "query" else 150, 0] = True
    lost_state[0, 0, 40] = True
    if what == "value":
        lost_state[0, 0, column] = True
    if what == "key":
        lost_state[0, 0, :, column] = True
    for case in out[1:]:
        for got, was, where in zip(case, out[0], (lost, lost_dots, lost_state)):
            assert not bool(got[where].isfinite().any()) and torch.equal(got[~where], was[~where])
