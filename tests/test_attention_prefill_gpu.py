"""The tcgen05 prompt kernel over every way its query tiles are paired and every option, against float64: runs around the
tiles' edges (64, 128, 256 rows), sequences that hold earlier positions, grouped and ungrouped heads, windows with kept
positions, cells, caps (scores on both sides of a quarter of the cap), distance biases, sinks."""
import math

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def attend(q, k, v, first, scale, window, keep, cell, cap, bias, sink):
    """float64: (output, sum of weight * |value|) for queries q [n, H, dk] at positions first, …"""
    n, H, m = q.shape[0], q.shape[1], k.shape[0]
    i, j = torch.arange(first, first + n, device=q.device)[:, None], torch.arange(m, device=q.device)[None]
    see = j <= i
    if cell:
        see = see & (i // cell == j // cell)
    elif window:
        see = see & ((i - j < window) | (j < keep))
    o, mag = (torch.empty((n, H, v.shape[2]), dtype=torch.float64, device=q.device) for _ in range(2))
    for h in range(H):
        g = h * k.shape[1] // H
        s = q[:, h] @ k[:, g].t() * scale
        if cap:
            s = cap * torch.tanh(s / cap)
        if bias is not None:
            s = s + bias[h][torch.clamp(i - j, 0, bias.shape[1] - 1)]
        s = s.masked_fill(~see, -float("inf"))
        if sink is not None:
            p = torch.softmax(torch.cat([s, sink[h].expand(n, 1)], 1), 1)[:, :-1]
        else:
            p = torch.softmax(s, 1)
        o[:, h], mag[:, h] = p @ v[:, g], p @ v[:, g].abs()
    return o, mag


CASES = [  # H, G, dk, dv, planes, runs, held, window, keep, cell, cap, bias rows, sink
    (16, 16, 128, 128, 2, [1, 128, 129, 300], [0, 0, 0, 0], 0, 0, 0, 0.0, 0, False),
    (4, 4, 64, 64, 2, [257], [100], 0, 0, 0, 0.0, 0, False),
    (4, 2, 64, 64, 2, [65, 640], [0, 63], 200, 0, 0, 0.0, 0, False),
    (16, 2, 128, 128, 1, [700, 900, 512, 2, 640, 700], [0, 0, 0, 0, 0, 40], 0, 0, 0, 0.0, 0, True),      # head pairs
    (16, 2, 128, 128, 1, [1100, 900, 512, 60, 640, 700], [0, 7, 0, 0, 0, 40], 0, 0, 0, 30.0, 0, False),  # head pairs, capped
    (6, 2, 128, 64, 1, [200, 17], [500, 0], 0, 0, 0, 0.0, 0, True),
    (8, 2, 128, 128, 1, [500, 33], [0, 700], 256, 4, 0, 0.0, 700, True),
    (3, 1, 64, 128, 1, [383, 64], [0, 300], 100, 70, 0, 0.0, 90, False),
    (4, 2, 64, 128, 1, [400, 129], [11, 0], 0, 0, 96, 0.0, 0, False),
    (4, 2, 64, 128, 1, [300], [190], 0, 0, 64, 20.0, 50, True),
    (2, 1, 128, 128, 1, [640], [0], 128, 0, 0, 4.0, 0, True),
]


@pytest.mark.parametrize("case", range(len(CASES)))
@pytest.mark.parametrize("spread", [1.0, 6.0])       # 6: maxima grow by more than the rescaling threshold, scores pass the cap
def test_prompt_kernel(case, spread):
    from turboquant_cpp_b200.kernels import attention as KA
    from turboquant_cpp_b200.kernels.gemm_tc import check_status
    H, G, dk, dv, planes, runs, held, window, keep, cell, cap, rows, with_sink = CASES[case]
    g = torch.Generator(device=DEV).manual_seed(case * 31 + int(spread))
    rand = lambda *shape: torch.randn(shape, generator=g, device=DEV)
    bias = rand(H, rows) if rows else None
    sink = 2.0 * rand(H) if with_sink else None
    total = [n + h for n, h in zip(runs, held)]
    counts = [-(-t // 64) for t in total]
    order = torch.randperm(sum(counts), generator=torch.Generator().manual_seed(case)).split(counts)
    cache = torch.zeros((sum(counts), planes, G, 64, dk if planes == 2 else dk + dv), dtype=torch.bfloat16, device=DEV)
    table = torch.full((len(runs), max(counts)), -1, dtype=torch.int32)
    q = (spread * rand(sum(runs), H, dk)).to(torch.bfloat16)
    kv = []
    for i, t in enumerate(total):
        k, v = rand(t, G, dk).to(torch.bfloat16), rand(t, G, dv).to(torch.bfloat16)
        kv.append((k, v))
        table[i, :counts[i]] = order[i].to(torch.int32)
        at = torch.arange(t, device=DEV)
        page = order[i].to(DEV)[at // 64]
        if planes == 2:
            cache[page, 0, :, at % 64], cache[page, 1, :, at % 64] = k, v
        else:
            cache[page, 0, :, at % 64] = torch.cat([k, v], -1)
    i32 = lambda a: torch.tensor(a, dtype=torch.int32, device=DEV)
    out = torch.empty((sum(runs), H * dv), dtype=torch.bfloat16, device=DEV)
    scale = dk ** -0.5
    KA.prefill_rows(q, cache, planes, i32(np.concatenate([[0], np.cumsum(runs)])), i32(held), table.to(DEV), 64, window, scale, out,
                    len(runs), max(runs), H, G, dk, dv, keep_first=keep, cell=cell, softcap=cap, bias_t=bias, sink=sink)
    check_status()
    at = 0
    for (k, v), n, first in zip(kv, runs, held):
        got = out[at:at + n].view(n, H, dv).double()
        want, mag = attend(q[at:at + n].double(), k.double(), v.double(), first, scale, window, keep, cell, cap,
                           None if bias is None else bias.double(), None if sink is None else sink.double())
        at += n
        # weights rounded to bfloat16 (eight significant bits: at most 2^-8 of each; their sum is taken before), the output
        # too (2^-8 of it); the float32 scores, |s| up to about 40, add 2^-16 of relative weight
        bound = (2.0 ** -8 + 2.0 ** -16) * mag + 2.0 ** -8 * want.abs() + 1e-6
        assert bool(((got - want).abs() <= bound).all()), float(((got - want).abs() / bound).max())


def one_sequence(q, k, v, **options):
    """Attention over rows of one sequence whose positions all are new: q [T, H, dk], k [T, G, dk], v [T, G, dv] -> [T, H, dv]."""
    from turboquant_cpp_b200.kernels import bias_attention as KB
    T, H, dk = q.shape
    G, dv, pages = k.shape[1], v.shape[2], -(-T // 64)
    cache = torch.zeros((pages, 1, G, 64, dk + dv), dtype=torch.bfloat16, device=DEV)
    at = torch.arange(T, device=DEV)
    cache[at // 64, 0, :, at % 64] = torch.cat([k, v], -1).to(torch.bfloat16)
    i32 = lambda a: torch.tensor(a, dtype=torch.int32, device=DEV)
    out = torch.empty((T, H * dv), dtype=torch.bfloat16, device=DEV)
    bias, sink = options.pop("bias", None), options.pop("sink", None)
    KB.attention_runs(q.to(torch.bfloat16), cache, bias, sink, i32([0, T]), i32([0]), i32([list(range(pages))]), 64, options.pop("window", 0), 0,
                      options.pop("scale", 1.0), out, 1, T, H, G, dk, dv, **options)
    return out.view(T, H, dv)


@pytest.mark.parametrize("options", [{}, {"bias": True}, {"softcap": 1e4}, {"cell": 512}])
def test_the_largest_weight_is_not_rounded(options):
    """A row's largest weight is exactly one in the second product, also where a later tile brings it and the maximum grows by less
    than 2^8: with all other values zero the result is a float32 quotient, rounded once, but for the rounding of the one other weight
    that counts in the sum."""
    T, d, late = 400, 64, 300
    g = torch.Generator().manual_seed(3)
    q, k, v = torch.zeros(T, 1, d), torch.zeros(T, 1, d), torch.zeros(T, 1, d)
    q[:, 0, 0], q[:, 0, 1] = 3.0 + 2.4 * torch.rand(T, generator=g), 1.0
    k[late, 0, 0] = 1.0                                            # scores of 3 to 5.4
    k[1:, 0, 1], k[late, 0, 1] = -20.0, 0.0                        # position 0: zero, all others: -20
    v[late, 0] = 1.0 + torch.rand(d, generator=g)
    q, v = q.to(torch.bfloat16).float(), v.to(torch.bfloat16).float()
    options = dict(options)
    if options.pop("bias", False):
        options["bias"] = torch.zeros((1, 50), device=DEV)
    got = one_sequence(q.to(DEV), k.to(DEV), v.to(DEV), **options)[late:, 0].double().cpu()
    s = q[late:, 0, 0].double()
    s = options["softcap"] * torch.tanh(s / options["softcap"]) if "softcap" in options else s
    others = 1.0 + math.exp(-20) * (torch.arange(late, T, dtype=torch.float64) - 1)
    share = (torch.exp(s) / (torch.exp(s) + others))[:, None]
    want = share * v[late, 0].double()
    half = torch.exp2(torch.floor(torch.log2(want)) - 8)           # half a unit in the last place of bfloat16
    assert bool(((got - want).abs() <= half + (2.0 ** -8 * (1 - share) + 2.0 ** -18) * want).all()), float(((got - want).abs() / half).max())


def test_the_lowest_finite_bias_leaves_a_row_its_weights():
    """Where every key a row sees is biased by the type's lowest value the weights are equal, as they are after any other constant."""
    T, H, d = 200, 2, 64
    g = torch.Generator(device=DEV).manual_seed(4)
    v = torch.randn((T, H, d), generator=g, device=DEV).to(torch.bfloat16)
    zero = torch.zeros((T, H, d), device=DEV)
    got = one_sequence(zero, zero, v, bias=torch.full((H, 8), torch.finfo(torch.float32).min, device=DEV)).double()
    n = torch.arange(1, T + 1, device=DEV, dtype=torch.float64)[:, None, None]
    want, mag = v.double().cumsum(0) / n, v.double().abs().cumsum(0) / n
    assert bool(((got - want).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -20 * mag).all())


def test_the_cap_beyond_a_quarter_has_the_precision_of_tanhf():
    """Cells of two positions: an odd row's first weight is the logistic of the difference of two capped scores, and a cap of 1e6
    shows their relative errors.  tanhf was measured to be off by 7.8e-8 (root mean square) where |x| > 1/4, fast intrinsics by
    1.2e-7 and by more near the quarter."""
    T, d, cap = 8192, 64, 1e6
    g = torch.Generator().manual_seed(6)
    q, k, v = torch.zeros(T, 1, d), torch.zeros(T, 1, d), torch.zeros(T, 1, d)
    # scores 64 a + b / 64 of bfloat16 factors are exact in float32; a cell's two share a, its b give a difference of up to three
    q[:, 0, 0], q[:, 0, 1] = 64.0, 1.0 / 64
    k[:, 0, 0] = torch.round(512.0 * (0.26 + 0.1 * torch.rand(T // 2, generator=g))).repeat_interleave(2)
    k[:, 0, 1] = torch.randint(-3, 4, (T,), generator=g).float()
    v[0::2] = 1.0
    scale = cap / 32768
    got = one_sequence(q.to(DEV), k.to(DEV), v.to(DEV), scale=scale, softcap=cap, cell=2)[1::2, 0, 0].double().cpu()
    s = cap * torch.tanh((q.double() * k.double()).sum(-1)[:, 0] * float(np.float32(scale)) / cap)
    a, b = s[0::2], s[1::2]
    live = (a - b).abs() < 3                                       # weights that bfloat16 holds to 2^-9 of their logit's unit
    off = (torch.logit(got) - (a - b))[live] / (0.5 * (a + b))[live]
    assert int(live.sum()) > 1000 and float(off.square().mean().sqrt()) < 2 ** 0.5 * 1e-7, float(off.square().mean().sqrt())


def test_a_cap_too_small_for_the_series():
    """Scores of zero and scores far beyond a cap of 1e-7: all weights equal."""
    T, d = 100, 64
    g = torch.Generator(device=DEV).manual_seed(7)
    q, k = torch.ones((T, 1, d), device=DEV), torch.randint(0, 2, (T, 1, d), generator=g, device=DEV).float()
    k[::2] = 0
    v = torch.randn((T, 1, d), generator=g, device=DEV).to(torch.bfloat16)
    got = one_sequence(q, k, v, softcap=1e-7).double()
    n = torch.arange(1, T + 1, device=DEV, dtype=torch.float64)[:, None, None]
    want, mag = v.double().cumsum(0) / n, v.double().abs().cumsum(0) / n
    assert bool(((got - want).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -18 * mag).all())


@pytest.mark.parametrize("cap", [20.0, 7.3])
def test_infinite_scores_are_the_cap(cap):
    """Products that overflow float32 are capped like any other: weights e^cap and e^-cap."""
    T, d = 100, 64
    g = torch.Generator(device=DEV).manual_seed(10)
    q, k = torch.zeros((T, 1, d), device=DEV), torch.zeros((T, 1, d), device=DEV)
    q[:, 0, 0], k[:, 0, 0] = 3e38, 4.0 * (1 - 2 * torch.randint(0, 2, (T,), generator=g, device=DEV)).float()
    v = torch.randn((T, 1, d), generator=g, device=DEV).to(torch.bfloat16)
    got = one_sequence(q, k, v, softcap=cap).double()
    w = torch.exp(cap * torch.sign(k[:, 0, 0]).double() - cap)[:, None, None]
    want, mag = (w * v.double()).cumsum(0) / w.cumsum(0), (w * v.double().abs()).cumsum(0) / w.cumsum(0)
    assert bool(((got - want).abs() <= 2.0 ** -8 * want.abs() + (2.0 ** -7 + 1e-5) * mag).all())


def test_queries_and_results_at_any_element():
    """Contiguous views that begin off a 16-byte boundary, and a step without runs."""
    from turboquant_cpp_b200.kernels import bias_attention as KB
    T, H, d = 100, 2, 64
    g = torch.Generator(device=DEV).manual_seed(8)
    rand = lambda n: torch.randn(n, generator=g, device=DEV).to(torch.bfloat16)
    cache, q0, room = rand(2 * 64 * 2 * d).view(2, 1, 1, 64, 2 * d), rand(T * H * d + 2), torch.zeros(T * H * d + 2, dtype=torch.bfloat16, device=DEV)
    i32 = lambda a: torch.tensor(a, dtype=torch.int32, device=DEV)
    call = lambda q, out, run=T: KB.attention_runs(q, cache, None, None, i32([0, T]), i32([0]), i32([[0, 1]]), 64, 0, 0, 0.125, out, 1, run, H, 1, d, d)
    q = q0[2:].view(T, H, d)
    want = call(q.clone(), torch.empty((T, H * d), dtype=torch.bfloat16, device=DEV))
    out = room[2:].view(T, H * d)
    assert q.data_ptr() % 16 == 4 and out.data_ptr() % 16 == 4
    assert call(q, out) is out and torch.equal(out, want) and not bool(room[:2].any())
    assert call(q, out, run=0) is out and torch.equal(out, want)


def test_sizes_of_any_integer_type():
    """Counts as numpy gives them, such as the longest of an array of run lengths."""
    from turboquant_cpp_b200.kernels import bias_attention as KB
    T, H, d = 70, 2, 64
    g = torch.Generator(device=DEV).manual_seed(9)
    rand = lambda *s: torch.randn(s, generator=g, device=DEV)
    i32 = lambda a: torch.tensor(a, dtype=torch.int32, device=DEV)
    n = lambda *v: [np.int64(x) for x in v]
    rows, table, freq, gates = rand(T, 4 * d), i32([[0, 1]]), rand(d // 2), rand(T, H)
    got = []
    for f in (list, lambda v: n(*v)):
        sizes, run, page = f([H, 1, d, d]), f([T])[0], f([64])[0]
        q, cache, out = torch.empty((T, H, d), dtype=torch.bfloat16, device=DEV), torch.zeros((2, 1, 1, 64, 2 * d), dtype=torch.bfloat16, device=DEV), \
            torch.empty((T, H * d), dtype=torch.bfloat16, device=DEV)
        at = torch.arange(T, device=DEV, dtype=torch.int32), torch.zeros(T, device=DEV, dtype=torch.int32)
        KB.kv_write(rows, q, cache, None, None, 0.0, *at, table, page, *sizes)
        KB.attention_runs(q, cache, None, None, i32([0, T]), i32([0]), table, page, *f([0, 0]), 0.125, out, f([1])[0], run, *sizes, cell=f([0])[0])
        KB.kv_write_rot(rows, q, cache, freq, f([d])[0], True, 0.0, *at, table, page, *sizes, v_share=f([1])[0])
        KB.heads_unrotate_gate(out, gates, f([0])[0], None, True, at[0], out, f([H])[0], f([d])[0])
        got.append((q, cache, out))
    assert all(torch.equal(a, b) for a, b in zip(*got))
