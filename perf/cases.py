"""The work whose speed this framework answers for: decode steps of a whole model, and single layers of the designs on
prompts and on decode steps, from one token to steps of thousands, in bfloat16 and in true float32.

Most cases are one layer (a mixer or a feed-forward made through the registries of `parts`), run the way a model runs it:
bound weights, rows of a paged cache or per-sequence state, a StepContext.  Prompts call the layer's forward; decode layers
replay a CUDA graph of it, as the engine does with its decode steps.  Sizes are those of the framework's benchmark
(Qwen1.5-MoE-A2.7B layers, and the other designs' at width 2,048); drawn cases vary the tokens, the sequences, how many
positions they already hold, and for the smaller designs the width.
"""
import math

import numpy as np
import torch

import turboquant_cpp_b200 as tq
from turboquant_cpp_b200 import parts
from turboquant_cpp_b200.csrc.build import ensure_built
from turboquant_cpp_b200.weights import WeightStore
from turboquant_cpp_b200.weights.loader import WeightSource

PAGE = 64
EPS = 1e-5
DEVICE = "cuda:0"
VOCAB = 151936

MODEL = {
    "architectures": ["Qwen2MoeForCausalLM"], "model_type": "qwen2_moe", "num_hidden_layers": 4, "hidden_size": 2048,
    "num_attention_heads": 16, "num_key_value_heads": 16, "num_experts": 60, "num_experts_per_tok": 4,
    "moe_intermediate_size": 1408, "norm_topk_prob": False, "shared_expert_intermediate_size": 5632,
    "intermediate_size": 5632, "vocab_size": VOCAB, "rope_theta": 1000000.0, "rms_norm_eps": 1e-6,
    "max_position_embeddings": 4096, "use_sliding_window": False, "sliding_window": 0, "max_window_layers": 4,
    "tie_word_embeddings": False, "decoder_sparse_step": 1, "mlp_only_layers": [], "hidden_act": "silu",
    "torch_dtype": "bfloat16",
}


# ---- the cases ---------------------------------------------------------------------------------------------------
# seqs: sequences of the step; new: tokens they bring together (split unevenly); held: positions the longest of them holds
# from earlier steps
def listed():
    return [
        # one chat: a single sequence's next token, four layers and the head
        {"name": "model_decode_1", "kind": "model", "seqs": 1, "held": 700},
        # a server's decode step: 32 sequences of unequal lengths
        {"name": "model_decode_32", "kind": "model", "seqs": 32, "held": 2048},
        # the flagship's routed and shared experts on a prompt
        {"name": "experts_prompt", "kind": "experts", "new": 2048},
        # its attention layer on three prompts of unequal lengths in one step
        {"name": "attention_prompt", "kind": "attention", "dtype": "bfloat16", "seqs": 3, "new": 4096, "held": 0},
        # the same layer in the exact 32-bit run that users compare with
        {"name": "attention_float32", "kind": "attention", "dtype": "float32", "seqs": 1, "new": 700, "held": 0},
        # attention by distance bias inside a window, one prompt
        {"name": "window_prompt", "kind": "window", "width": 2048, "seqs": 1, "new": 2048, "held": 0},
        # attention with normed, rotated queries, keys and values and capped scores, over everything before
        {"name": "rotated_prompt", "kind": "rotated", "width": 2048, "seqs": 3, "new": 4096, "held": 0},
        # a decode step of the attention over rows: 64 sequences
        {"name": "rows_decode", "kind": "rows", "width": 2048, "seqs": 64, "held": 2048},
        # latent attention on a prompt
        {"name": "latent_prompt", "kind": "latent", "width": 2048, "seqs": 1, "new": 2048, "held": 0},
        # latent attention whose queries pass a latent too, a decode step of a small batch
        {"name": "latent_decode", "kind": "latent_q", "width": 2048, "seqs": 8, "held": 2048},
        # a recurrence that must take its tokens in order, on a prompt
        {"name": "delta_prompt", "kind": "delta", "width": 2048, "seqs": 1, "new": 2048},
        # a recurrence that is linear in its state, on two prompts
        {"name": "memory_prompt", "kind": "memory", "width": 2048, "seqs": 2, "new": 2048},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["model", "experts", "attention", "attention", "window", "rotated", "rows", "latent", "latent_q", "delta", "memory"])
    width = rng.choice([1024, 2048])
    if kind == "model":
        return {"kind": kind, "seqs": _log(rng, 1, 32), "held": _log(rng, 33, 2048)}
    if kind == "experts":
        return {"kind": kind, "new": _log(rng, 17, 2048)}
    if kind in ("rows", "latent_q"):
        return {"kind": kind, "width": width, "seqs": _log(rng, 1, 64 if kind == "rows" else 8), "held": _log(rng, 65, 2048)}
    if kind in ("delta", "memory"):
        new = _log(rng, 33, 2048)
        return {"kind": kind, "width": width, "seqs": rng.randint(1, max(1, min(4, new // 32))), "new": new}
    dtype = "bfloat16"
    if kind == "attention" and rng.random() < 0.3:
        dtype, new = "float32", _log(rng, 33, 700)
    else:
        new = _log(rng, 65, 4096 if kind in ("attention", "rotated") else 2048)
    held = rng.choice([0, 0, _log(rng, 16, 1024)]) if new <= 1024 and dtype == "bfloat16" else 0
    case = {"kind": kind, "seqs": rng.randint(1, max(1, min(4, new // 64))), "new": new, "held": held}
    return dict(case, dtype=dtype) if kind == "attention" else dict(case, width=width)


def _lens(case):
    """(tokens each sequence brings, positions it holds): unequal, from the case alone."""
    if case["kind"] == "experts":
        return [case["new"]], [0]
    n = case["seqs"]
    held = [max(0, case.get("held", 0) - (i * 37) % max(1, case.get("held", 0) // 3 + 1)) for i in range(n)]
    if "new" not in case:
        return [1] * n, held
    parts_of = [(i + 1) * case["new"] // (n * (n + 1) // 2) for i in range(n)]
    parts_of[-1] += case["new"] - sum(parts_of)
    return parts_of, held


def _sizes(case):
    """Sizes of the layer a case is about."""
    k = case["kind"]
    if k in ("model", "experts"):
        return {"W": 2048, "E": 60, "top": 4, "I": 1408, "S": 5632}
    if k == "attention":
        return {"W": 2048, "H": 16, "G": 16, "D": 128, "V": 128, "theta": 1000000.0}
    wide = case["width"] == 2048
    H, G = (16, 4) if wide else (8, 2)
    s = {"W": case["width"], "H": H, "G": G, "D": 128, "V": 128, "scale": 128 ** -0.5}
    if k == "window":
        return dict(s, window=1024, keep=4, far=2048, rows=32)
    if k == "rotated":
        return dict(s, base=500000.0, cap=50.0, factor=8.0, original=8192, fast=32.0, slow=1.0)
    if k == "latent":
        return dict(s, D=128 if wide else 64, R=64, V=128 if wide else 64, rank=512 if wide else 256, window=1024, base=1000000.0,
                    factor=4.0, original=4096, fast=32.0, slow=1.0, scale=(192 if wide else 128) ** -0.5, qr=0)
    if k == "latent_q":
        return dict(s, R=0, rank=512 if wide else 256, qr=768 if wide else 384, window=0)
    if k == "delta":
        return dict(s, taps=4)
    if k == "memory":
        return dict(s, D=128 if wide else 64, cap=20.0)
    return s


# ---- weights, drawn from the seed -----------------------------------------------------------------------------------
def _shapes(case):
    """Tensor name -> (shape, how its values are drawn)."""
    s, k = _sizes(case), case["kind"]
    W, H, G, D, V = (s.get(n, 0) for n in ("W", "H", "G", "D", "V"))
    m = "normal"
    if k == "experts":
        E, I, S = s["E"], s["I"], s["S"]
        t = {"gate.weight": ((E, W), m), "shared_expert_gate.weight": ((1, W), m)}
        for e in range(E):
            t.update({f"experts.{e}.gate_proj.weight": ((I, W), m), f"experts.{e}.up_proj.weight": ((I, W), m),
                      f"experts.{e}.down_proj.weight": ((W, I), m)})
        t.update({"shared_expert.gate_proj.weight": ((S, W), m), "shared_expert.up_proj.weight": ((S, W), m),
                  "shared_expert.down_proj.weight": ((W, S), m)})
        return t
    if k == "attention":
        t = {"o_proj.weight": ((W, H * D), m)}
        for n, rows in (("q", H * D), ("k", G * D), ("v", G * D)):
            t.update({n + "_proj.weight": ((rows, W), m), n + "_proj.bias": ((rows,), "wide")})
        return t
    if k in ("window", "rotated", "rows"):
        t = {"q": ((H * D, W), m), "k": ((G * D, W), m), "v": ((G * V, W), m), "o": ((W, H * V), m)}
        if k == "window":
            t["rel"] = ((s["rows"], H), "wide")
        if k == "rotated":
            t.update({"g": ((H, W), m), "q.norm": ((D,), "one"), "k.norm": ((D,), "one")})
        return t
    if k in ("latent", "latent_q"):
        R, rank = s["R"], s["rank"]
        t = {"uk": ((H * D, rank), m), "uv": ((H * V, rank), m), "o": ((W, H * V), m), "dkv": ((rank + R, W), m), "dkv.norm": ((rank,), "one")}
        if s["qr"]:
            t.update({"dq": ((s["qr"], W), m), "dq.norm": ((s["qr"],), "one"), "uq": ((H * (D + R), s["qr"]), m)})
        else:
            t.update({"q": ((H * (D + R), W), m), "sink": ((H,), "wide")})
        return t
    if k == "delta":            # one decay per head; as many query/key heads as value heads
        return {"q": ((H * D, W), m), "k": ((H * D, W), m), "v": ((H * V, W), m), "q.conv": ((H * D, s["taps"]), "taps"),
                "k.conv": ((H * D, s["taps"]), "taps"), "v.conv": ((H * V, s["taps"]), "taps"), "b": ((H, W), m), "a": ((H, W), m),
                "A_log": ((H,), "A_log"), "dt_bias": ((H,), "dt_bias"), "g": ((H * V, W), m), "norm": ((V,), "one"), "o": ((W, H * V), m)}
    return {"q": ((H * D, W), m), "k": ((H * D, W), m), "v": ((H * V, W), m), "g": ((H * V, W), m), "i": ((H, W), m),
            "i.b": ((H,), "in_gate"), "f": ((H, W), m), "f.b": ((H,), "forget"), "norm": ((H * V,), "one"), "o": ((W, H * V), m)}


def _tensor(shape, how, seed, index):
    """bfloat16 values as a trained model's initialisation has them: 0.02 for products, decays and gates over their usual ranges."""
    g = torch.Generator(device=DEVICE).manual_seed((seed * 1000003 + index) & 0x7FFFFFFF)
    z = torch.randn(shape, generator=g, device=DEVICE, dtype=torch.bfloat16 if how == "normal" else torch.float32)
    if how == "normal":
        return z.mul_(0.02)
    u = torch.rand(shape, generator=g, device=DEVICE)
    z = {"wide": lambda: 0.5 * z, "one": lambda: 1.0 + 0.02 * z, "taps": lambda: u - 0.5, "A_log": lambda: torch.log(1.0 + 15.0 * u),
         "dt_bias": lambda: torch.log(torch.expm1(torch.exp(math.log(0.001) + u * math.log(100.0)))),
         "in_gate": lambda: z - 2.0, "forget": lambda: 3.0 + 3.0 * u}[how]()
    return z.to(torch.bfloat16)


class _Weights(WeightSource):
    def __init__(self, shapes, seed):
        self.shapes, self.seed = shapes, int(seed)
        self.at = {n: i + 100 for i, n in enumerate(shapes)}

    def index(self):
        return {n: (torch.bfloat16, tuple(s)) for n, (s, _) in self.shapes.items()}

    def read(self, name, device):
        return _tensor(*self.shapes[name], self.seed, self.at[name])


def _inputs(case, seed):
    """The layer's input rows, normed as a block hands them over."""
    g = torch.Generator(device=DEVICE).manual_seed(seed * 7 + 1)
    x = torch.randn((sum(_lens(case)[0]), _sizes(case)["W"]), generator=g, device=DEVICE)
    return x if case.get("dtype") == "float32" else x.to(torch.bfloat16)


def _held_rows(case, seed, i, n):
    """The cached rows of sequence i's n earlier positions, [n, planes * heads, row]."""
    s, k = _sizes(case), case["kind"]
    g = torch.Generator(device=DEVICE).manual_seed(seed * 7919 + 13 + i)
    shape = (n, 2 * s["G"], s["D"]) if k == "attention" else (n, 1, s["rank"] + s["R"]) if k in ("latent", "latent_q") else (n, s["G"], s["D"] + s["V"])
    return (0.8 * torch.randn(shape, generator=g, device=DEVICE)).to(torch.float32 if case.get("dtype") == "float32" else torch.bfloat16)


# ---- what a program has in hand before the call ----------------------------------------------------------------------
def _mixer(case):
    s, k = _sizes(case), case["kind"]
    if k == "attention":
        pe = parts.make_position_encoding("rotary", head_dim=s["D"], theta=s["theta"], max_position=8192, pairing="half")
        return parts.make_mixer("attention", prefix="", hidden=s["W"], n_heads=s["H"], n_kv_heads=s["G"], head_dim=s["D"], qkv_bias=True, position=pe)
    one = dict(prefix="", hidden=s["W"], heads=s["H"], kv_heads=s["G"], dim=s["D"], vdim=s["V"])
    scaled = lambda dims, pairing: parts.make_position_encoding(
        "rotary_scaled", dims=dims, base=s["base"], factor=s["factor"], original=s["original"], fast=s["fast"], slow=s["slow"], pairing=pairing)
    if k == "window":
        return parts.make_mixer("window_bias_attention", **one, scale=s["scale"], window=s["window"], keep_first=s["keep"], bias_rows=s["rows"], bias_far=s["far"])
    if k == "rows":
        return parts.make_mixer("window_bias_attention", **one, scale=s["scale"])
    if k == "rotated":
        return parts.make_mixer("rotated_value_attention", **one, scale=s["scale"], eps=EPS, position=scaled(s["D"], "halves"),
                                value_base=s["base"], softcap=s["cap"])
    if k in ("latent", "latent_q"):
        return parts.make_mixer("latent_attention", prefix="", hidden=s["W"], heads=s["H"], dim=s["D"], rot_dim=s["R"], vdim=s["V"], kv_rank=s["rank"],
                                scale=s["scale"], eps=EPS, window=s["window"], position=scaled(s["R"], "neighbours") if s["R"] else None,
                                sink=k == "latent", q_rank=s["qr"])
    if k == "delta":
        return parts.make_mixer("head_delta", **dict(one, kv_heads=s["H"]), taps=s["taps"], eps=EPS)
    one.pop("kv_heads")
    return parts.make_mixer("matrix_memory", **one, gate_cap=s["cap"], eps=EPS)


def _context(case, dtype):
    new, held = _lens(case)
    cu = np.concatenate([[0], np.cumsum(new)])
    seq_of = np.repeat(np.arange(len(new)), new)
    pos = np.arange(cu[-1]) - cu[:-1][seq_of] + np.asarray(held)[seq_of]
    i32 = lambda a: torch.tensor(np.asarray(a), dtype=torch.int32, device=DEVICE)
    return parts.StepContext(
        n_tokens=int(cu[-1]), n_seqs=len(new), tokens=i32(np.zeros(cu[-1])), positions=i32(pos), seq_of_token=i32(seq_of), cu_seqlens=i32(cu),
        seq_start=i32(held), slots=i32(np.arange(len(new))), want_rows=i32([]), n_want=0, max_q_len=max(new),
        max_kv_len=max(a + b for a, b in zip(new, held)), act_dtype=dtype, device=torch.device(DEVICE), host_q_lens=list(new),
        host_slots=list(range(len(new))), host_seq_start=list(held), status=torch.zeros(1, dtype=torch.int32, device=DEVICE))


def _pages(case):
    """Each sequence's pages, scattered over the pool as they are after some traffic."""
    new, held = _lens(case)
    counts = [-(-(a + b) // PAGE) for a, b in zip(new, held)]
    order = np.random.RandomState(1).permutation(sum(counts))
    return np.split(order, np.cumsum(counts)[:-1]), sum(counts)


def _put_rows(kv, pages, first, rows):
    """Rows [n, planes * heads, row] of positions first, first + 1, … into a cache [pages, planes, heads, page, row]."""
    at = torch.arange(first, first + rows.shape[0], device=rows.device)
    ids = torch.tensor(np.asarray(pages), device=rows.device)
    kv.flatten(1, 2)[ids[at // PAGE], :, at % PAGE] = rows.to(kv.dtype)


def _layer(case, seed):
    dtype = torch.float32 if case.get("dtype") == "float32" else torch.bfloat16
    if case["kind"] == "experts":
        s = _sizes(case)
        part = parts.make_feed_forward("moe", prefix="", hidden=s["W"], n_experts=s["E"], top_k=s["top"], intermediate=s["I"], norm_topk=False,
                                       shared_intermediate=s["S"])
    else:
        part = _mixer(case)
    part.run_dtype = dtype
    ensure_built(part.kernels())
    part.bind(WeightStore(_Weights(_shapes(case), seed), part.weight_specs(), DEVICE, dtype))
    ctx, cache = _context(case, dtype), None
    if case["kind"] != "experts":
        need, state = part.cache_need(), part.state_need()
        cache = parts.LayerCache(page_size=PAGE)
        if need is not None:
            pages, total = _pages(case)
            cache.kv = torch.zeros((total, need.planes, need.n_kv_heads, PAGE, need.head_dim), dtype=dtype, device=DEVICE)
            table = np.full((len(pages), max(len(p) for p in pages)), -1, dtype=np.int32)
            for i, (p, n) in enumerate(zip(pages, _lens(case)[1])):
                table[i, :len(p)] = p
                if n:
                    _put_rows(cache.kv, p, 0, _held_rows(case, seed, i, n))
            cache.page_table = torch.tensor(table, device=DEVICE)
        if state is not None:
            cache.state = torch.zeros((ctx.n_seqs,) + tuple(state.shape), dtype=state.dtype, device=DEVICE)
    return {"case": case, "part": part, "x": _inputs(case, seed), "ctx": ctx, "cache": cache}


def _call(st):
    """One layer of one step, as a model runs it."""
    st["ctx"].carry = {}                       # a step starts with nothing carried over
    if st["cache"] is None:
        return st["part"].forward(st["x"], st["ctx"])
    if st["cache"].state is not None:
        st["cache"].state.zero_()              # the sequences begin here
    return st["part"].forward(st["x"], st["ctx"], st["cache"])


def _prepare_model(case, seed):
    model = tq.build_model(MODEL, "bfloat16")
    ensure_built(model.kernels())
    shapes = {s.name: (tuple(s.shape), "one" if s.init == "one_plus_normal" else "normal") for s in model.weight_specs()}
    model.bind(WeightStore(_Weights(shapes, seed), model.weight_specs(), DEVICE, torch.bfloat16))
    _, held = _lens(case)
    engine = tq.Engine(model, max_tokens=sum(-(-(n + 1) // PAGE) * PAGE for n in held), max_slots=len(held))
    rng = np.random.RandomState(seed)
    seqs = []
    for n in held:                             # the prompts that the sequences hold
        seqs.append(engine.open())
        engine.step([tq.StepEntry(seqs[-1], rng.randint(0, VOCAB, n).tolist())])
    tokens = torch.tensor(rng.randint(0, VOCAB, len(held)), dtype=torch.int32, device=DEVICE)
    for _ in range(2):                         # the step of this batch size is captured when it first runs
        engine.step_ahead(seqs, tokens)
        engine.drop_ahead()
    return {"case": case, "engine": engine, "seqs": seqs, "tokens": tokens}


def prepare(case, seed):
    if case["kind"] == "model":
        return _prepare_model(case, seed)
    st = _layer(case, seed)
    if "new" not in case:                      # a decode step's layer: captured, as the engine captures its steps
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            _call(st)
        torch.cuda.current_stream().wait_stream(side)
        st["graph"] = torch.cuda.CUDAGraph()
        with torch.cuda.graph(st["graph"]):
            st["y"] = _call(st)
    return st


def run(st):
    if st["case"]["kind"] == "model":          # the next token's logits; the sequences stay as they are
        logits = st["engine"].step_ahead(st["seqs"], st["tokens"])
        st["engine"].drop_ahead()
        return logits
    if "graph" in st:
        st["graph"].replay()
        return {"y": st["y"], "kv": st["cache"].kv}
    y = _call(st)
    if st["cache"] is None:
        return y
    if st["cache"].state is not None:
        return {"y": y, "state": st["cache"].state}
    return {"y": y, "kv": st["cache"].kv}


# ---- the least a pass has to do ---------------------------------------------------------------------------------------
def work(case):
    s, k = _sizes(case), case["kind"]
    new, held = _lens(case)
    T, W = sum(new), s["W"]
    el = 4 if case.get("dtype") == "float32" else 2
    if k in ("model", "experts"):
        E, top, I, S = s["E"], s["top"], s["I"], s["S"]
        touched = E * (1.0 - (1.0 - top / E) ** T)
        weights = (E + 1) * W + touched * 3 * W * I + 3 * W * S
        flops = 2.0 * T * ((E + 1) * W + top * 3 * W * I + 3 * W * S)
        if k == "experts":
            return {"bytes": 2 * weights + T * W * (2 + 4), "flops": flops}
        L, seen = MODEL["num_hidden_layers"], sum(h + 1 for h in held)
        return {"bytes": L * (2 * weights + 2 * 4 * W * W + 2 * 2 * W * seen) + 2 * VOCAB * W + 4 * T * VOCAB,
                "flops": L * (flops + 2.0 * T * 4 * W * W + 4.0 * W * seen) + 2.0 * T * W * VOCAB}
    weights = sum(math.prod(shape) for shape, _ in _shapes(case).values())
    io = T * W * (el + 4)
    if k in ("delta", "memory"):
        state = s["H"] * s["D"] * s["V"]
        return {"bytes": 2 * weights + io + 4 * state * len(new), "flops": 2.0 * T * weights + (7.0 if k == "delta" else 5.0) * T * state}
    window = s.get("window", 0)
    seen = sum(min(p + 1, window + s.get("keep", 0)) if window else p + 1 for n, h in zip(new, held) for p in range(h, h + n))
    kept = sum(min(h, window) if window else h for h in held)
    if k in ("latent", "latent_q"):
        row, per_pair = s["rank"] + s["R"], min(2 * s["rank"] + s["R"], s["D"] + s["R"] + s["V"]) * 2.0
    elif k == "attention":
        row, per_pair = 2 * s["G"] * s["D"], 4.0 * s["D"]
    else:
        row, per_pair = s["G"] * (s["D"] + s["V"]), 2.0 * (s["D"] + s["V"])
    return {"bytes": el * weights + io + el * row * (kept + T), "flops": 2.0 * T * weights + s["H"] * per_pair * seen}


def tolerance(case):
    return TOLERANCES[case.get("dtype", case["kind"]) if case["kind"] == "attention" else case["kind"]]


# four times what the outputs showed against exact() when the file was written (bfloat16 rows 0.0016 to 0.0042, float32 9e-7);
# a whole model's rounding travels through four layers and their routers
TOLERANCES = {
    "model": {"rel": 0.02, "max": 0.2}, "experts": {"rel": 0.007, "max": 0.1}, "bfloat16": {"rel": 0.009, "max": 0.1},
    "float32": {"rel": 5e-6, "max": 1e-4}, "window": {"rel": 0.013, "max": 0.1}, "rotated": {"rel": 0.017, "max": 0.1},
    "rows": {"rel": 0.01, "max": 0.1}, "latent": {"rel": 0.015, "max": 0.1}, "latent_q": {"rel": 0.012, "max": 0.1},
    "delta": {"rel": 0.007, "max": 0.1}, "memory": {"rel": 0.007, "max": 0.1},
}


# ---- the same in 64 bits, plainly -------------------------------------------------------------------------------------
def _rms(x, w=1.0):
    return x / torch.sqrt(x.square().mean(-1, keepdim=True) + EPS) * w


def _turn(x, pos, freq, mag=1.0, halves=True):
    """x [n, heads, d]: its first 2 len(freq) elements turned by pos * freq, in pairs of halves or of neighbours."""
    n = freq.shape[0]
    a = pos[:, None, None].double() * freq
    c, s = torch.cos(a) * mag, torch.sin(a) * mag
    i = torch.arange(n, device=x.device)
    u, v = (i, i + n) if halves else (2 * i, 2 * i + 1)
    y = x.clone()
    y[..., u], y[..., v] = x[..., u] * c - x[..., v] * s, x[..., v] * c + x[..., u] * s
    return y


def _stretched(dims, s):
    i = torch.arange(dims // 2, dtype=torch.float64, device=DEVICE)
    f = s["base"] ** (-2.0 * i / dims)
    pair = lambda turns: dims * math.log(s["original"] / (2.0 * math.pi * turns)) / (2.0 * math.log(s["base"]))
    lo, hi = max(math.floor(pair(s["fast"])), 0), min(math.ceil(pair(s["slow"])), dims - 1)
    ramp = torch.clamp((i - lo) / max(hi - lo, 0.001), 0.0, 1.0)
    return f / s["factor"] * ramp + f * (1.0 - ramp), 0.1 * math.log(s["factor"]) + 1.0


def _attend(q, k, v, first, scale, window=0, keep=0, bias=None, far=0, cap=0.0, sink=None):
    """q [n, H, dk] at positions first, …; k [m, G, dk], v [m, G, dv] from position 0."""
    n, H, m = q.shape[0], q.shape[1], k.shape[0]
    i, j = torch.arange(first, first + n, device=q.device)[:, None], torch.arange(m, device=q.device)[None]
    see = j <= i
    if window:
        see &= (i - j < window) | (j < keep)
    out = torch.empty((n, H, v.shape[2]), dtype=torch.float64, device=q.device)
    for h in range(H):
        g = h * k.shape[1] // H
        s = q[:, h] @ k[:, g].t() * scale
        if cap:
            s = cap * torch.tanh(s / cap)
        if bias is not None:
            s = s + bias[:, h][torch.clamp(i - j, 0, far)]
        s = s.masked_fill(~see, -math.inf)
        top = s.max(1, keepdim=True).values
        if sink is not None:
            top = torch.clamp(top, min=float(sink[h]))
        p = torch.exp(s - top)
        total = p.sum(1, keepdim=True)
        if sink is not None:
            total = total + torch.exp(sink[h] - top)
        out[:, h] = (p / total) @ v[:, g]
    return out


def _buckets(rows, far):
    half = rows // 2
    return torch.tensor([n if n < half else min(rows - 1, half + int(math.floor(math.log(n / half) / math.log(far / half) * (rows - half))))
                         for n in range(far + 1)], device=DEVICE)


def _exact_experts(case, x, w):
    s = _sizes(case)
    p = torch.softmax(x @ w("gate.weight").t(), dim=1)
    top, ids = torch.topk(p, s["top"], dim=1)
    y = torch.zeros_like(x)
    glu = lambda rows, name: (torch.nn.functional.silu(rows @ w(name + "gate_proj.weight").t()) * (rows @ w(name + "up_proj.weight").t())) @ w(name + "down_proj.weight").t()
    for e in range(s["E"]):
        t, j = torch.nonzero(ids == e, as_tuple=True)
        if t.numel():
            y[t] += top[t, j][:, None] * glu(x[t], f"experts.{e}.")
    return y + torch.sigmoid(x @ w("shared_expert_gate.weight").t()) * glu(x, "shared_expert.")


def _exact_rows(case, seed, x, w):
    """Softmax attentions: what each of them caches per position, and the layer's output."""
    s, k = _sizes(case), case["kind"]
    new, held = _lens(case)
    H, G, D, V, W = s["H"], s["G"], s["D"], s["V"], s["W"]
    pages, total = _pages(case)
    planes, heads, row = (2, G, D) if k == "attention" else (1, 1, s["rank"] + s["R"]) if k in ("latent", "latent_q") else (1, G, D + V)
    kv = torch.zeros((total, planes, heads, PAGE, row), dtype=torch.float64, device=DEVICE)
    out, at = [], 0
    for i, (n, h) in enumerate(zip(new, held)):
        xs, pos = x[at:at + n], torch.arange(h, h + n, device=DEVICE)
        at += n
        old = _held_rows(case, seed, i, h).double()
        if k in ("latent", "latent_q"):
            rank, R = s["rank"], s["R"]
            q = ((_rms(xs @ w("dq").t(), w("dq.norm")) @ w("uq").t()) if s["qr"] else xs @ w("q").t()).view(n, H, D + R)
            d = xs @ w("dkv").t()
            rows = torch.cat([_rms(d[:, :rank], w("dkv.norm")), d[:, rank:]], 1)[:, None]
            if R:
                f, mag = _stretched(R, s)
                q = torch.cat([q[..., :D], _turn(q[..., D:], pos, f, mag, halves=False)], -1)
                rows = torch.cat([rows[..., :rank], _turn(rows[..., rank:], pos, f, mag, halves=False)], -1)
            rows = torch.cat([old, rows])
            c = rows[:, 0, :rank]
            keys = torch.cat([(c @ w("uk").t()).view(-1, H, D), rows[..., rank:].expand(-1, H, -1)], -1)
            o = _attend(q, keys, (c @ w("uv").t()).view(-1, H, V), h, s["scale"], s["window"], sink=w("sink") if k == "latent" else None)
            y = o.reshape(n, -1) @ w("o").t()
        elif k == "attention":
            part = lambda a, hs: (xs @ w(a + "_proj.weight").t() + w(a + "_proj.bias")).view(n, hs, D)
            f = s["theta"] ** (-2.0 * torch.arange(D // 2, dtype=torch.float64, device=DEVICE) / D)
            rows = torch.cat([old, torch.cat([_turn(part("k", G), pos, f), part("v", G)], 1)])
            y = _attend(_turn(part("q", H), pos, f), rows[:, :G], rows[:, G:], h, D ** -0.5).reshape(n, -1) @ w("o_proj.weight").t()
        else:
            q, kk, v = ((xs @ w(a).t()).view(n, hs, -1) for a, hs in (("q", H), ("k", G), ("v", G)))
            more = {}
            if k == "rotated":
                f, mag = _stretched(D, s)
                fv = s["base"] ** (-2.0 * torch.arange(V // 2, dtype=torch.float64, device=DEVICE) / V)
                q, kk, v = _turn(_rms(q, w("q.norm")), pos, f, mag), _turn(_rms(kk, w("k.norm")), pos, f, mag), _turn(v, pos, fv)
                more = dict(cap=s["cap"])
            else:
                more = dict(sink=torch.zeros(H, dtype=torch.float64, device=DEVICE))
                if k == "window":
                    more.update(window=s["window"], keep=s["keep"], bias=w("rel")[_buckets(s["rows"], s["far"])], far=s["far"])
            rows = torch.cat([old, torch.cat([kk, v], -1)])
            o = _attend(q, rows[..., :D], rows[..., D:], h, s["scale"], **more)
            if k == "rotated":
                o = _turn(o, -pos, fv) * torch.sigmoid(xs @ w("g").t())[..., None]
            y = o.reshape(n, -1) @ w("o").t()
        _put_rows(kv, pages[i], 0, rows)
        out.append(y)
    return {"y": torch.cat(out), "kv": kv}


def _exact_recurrence(case, x, w):
    s, k = _sizes(case), case["kind"]
    H, D, V = s["H"], s["D"], s["V"]
    outs, states, at = [], [], 0
    for n in _lens(case)[0]:
        xs = x[at:at + n]
        at += n
        proj = lambda a: xs @ w(a).t()
        S, o = torch.zeros((H, D, V), dtype=torch.float64, device=DEVICE), torch.empty((n, H, V), dtype=torch.float64, device=DEVICE)
        if k == "delta":
            raw = torch.cat([proj("q"), proj("k"), proj("v")], 1)
            taps, kept = torch.cat([w("q.conv"), w("k.conv"), w("v.conv")]), s["taps"] - 1
            pad = torch.cat([raw.new_zeros((kept, raw.shape[1])), raw])
            c = torch.nn.functional.silu(sum(pad[j:j + n] * taps[:, j] for j in range(s["taps"])))
            q, key, v = c[:, :H * D].reshape(n, H, D), c[:, H * D:2 * H * D].reshape(n, H, D), c[:, 2 * H * D:].reshape(n, H, V)
            unit = lambda a: a / torch.sqrt(a.square().sum(-1, keepdim=True) + 1e-6)
            q, key, beta = unit(q) * D ** -0.5, unit(key), torch.sigmoid(proj("b"))
            decay = torch.exp(-torch.exp(w("A_log")) * torch.nn.functional.softplus(proj("a") + w("dt_bias")))
            for t in range(n):
                S = S * decay[t][:, None, None]
                u = beta[t][:, None] * (v[t] - torch.einsum("hdv,hd->hv", S, key[t]))
                S = S + key[t][:, :, None] * u[:, None]
                o[t] = torch.einsum("hdv,hd->hv", S, q[t])
            y = (_rms(o, w("norm")) * torch.nn.functional.silu(proj("g").view(n, H, V))).reshape(n, -1) @ w("o").t()
            states.append(torch.cat([pad[n:n + kept].reshape(-1), S.transpose(1, 2).reshape(-1)]))
        else:
            q, key, v = (proj("q") * D ** -0.5).view(n, H, D), proj("k").view(n, H, D), proj("v").view(n, H, V)
            gi = s["cap"] * torch.tanh((proj("i") + w("i.b")) / s["cap"])
            gf = torch.nn.functional.logsigmoid(s["cap"] * torch.tanh((proj("f") + w("f.b")) / s["cap"]))
            N, m = torch.zeros((H, D), dtype=torch.float64, device=DEVICE), torch.zeros(H, dtype=torch.float64, device=DEVICE)
            for t in range(n):
                top = torch.maximum(gf[t] + m, gi[t])
                a, b = torch.exp(gf[t] + m - top), torch.exp(gi[t] - top)
                S = S * a[:, None, None] + (b[:, None] * key[t])[:, :, None] * v[t][:, None]
                N, m = N * a[:, None] + b[:, None] * key[t], top
                d = torch.maximum((N * q[t]).sum(-1).abs(), torch.exp(-m)) + 1e-6
                o[t] = torch.einsum("hdv,hd->hv", S, q[t]) / d[:, None]
            y = (_rms(o).reshape(n, -1) * w("norm") * torch.sigmoid(proj("g"))) @ w("o").t()
            states.append(torch.cat([torch.cat([S.transpose(1, 2), N[:, None]], 1).reshape(-1), m]))
        outs.append(y)
    return {"y": torch.cat(outs), "state": torch.stack(states)}


def exact(case, seed):
    """None for whole models: a router's near-tie that falls the other way in 64 bits changes all that follows it."""
    if case["kind"] == "model":
        return None
    shapes = _shapes(case)
    source = _Weights(shapes, seed)
    w = lambda name: source.read(name, DEVICE).double()
    x = _inputs(case, seed).double()
    if case["kind"] == "experts":
        return _exact_experts(case, x, w)
    if case["kind"] in ("delta", "memory"):
        return _exact_recurrence(case, x, w)
    return _exact_rows(case, seed, x, w)
