"""What the framework is timed on: calls of its public entry points as programs make them, from one short sequence to full batches.

Four groups. `step`: one decode step of the paged cache per layer (append + attention). `chunk`: prompt chunks through the cache
(append, then causal attention over pages). `operator`: the attention operator over plain tensors. `generate` and `serve`: whole
decoders behind the model API. `delta`: a recurrent mixer over prompts. A pass covers a few layers, each with pages of its own, as a
model's pass does; sizes are those of the benchmark's configurations and of the layers it compares (widths 1536 and 4096, heads 12 / 2 and
32 / 8 of 128), and odd ones between them.
"""
import math

import numpy as np
import torch

import llaisys_b200 as llaisys

D, PAGE = 128, 16
TORCH = {"bf16": torch.bfloat16, "f16": torch.float16, "f32": torch.float32}
NAMES = {"bf16": "BF16", "f16": "F16", "f32": "F32"}
VOCAB, WIDTH, FF, MODEL_LAYERS, THETA, EPS = 32768, 1536, 8960, 4, 1e6, 1e-6
TAPS = 4


def listed():
    return [
        # one user in the middle of a short answer: launches and latency are all there is
        dict(name="step_one", kind="step", seqs=1, low=777, high=777, heads=12, kv_heads=2, layers=4, dtype="bf16"),
        # a small server's step: 32 conversations of very different lengths
        dict(name="step_ragged", kind="step", seqs=32, low=128, high=4096, heads=12, kv_heads=2, layers=4, dtype="bf16"),
        # a full server's step: 64 conversations of 4096 tokens
        dict(name="step_batch", kind="step", seqs=64, low=4096, high=4096, heads=12, kv_heads=2, layers=2, dtype="bf16"),
        # one very long document
        dict(name="step_long", kind="step", seqs=1, low=131072, high=131072, heads=12, kv_heads=2, layers=2, dtype="f16"),
        # chunked prefill of eight conversations
        dict(name="chunk_serving", kind="chunk", seqs=8, low=0, high=8192, short=512, long=512, window=0, heads=12, kv_heads=2, layers=2,
             dtype="bf16"),
        # a whole prompt at once, layers of width 4096
        dict(name="chunk_prompt", kind="chunk", seqs=1, low=0, high=0, short=8192, long=8192, window=0, heads=32, kv_heads=8, layers=1,
             dtype="bf16"),
        # the same in a model whose attention has a sliding window and a gate per head
        dict(name="chunk_window", kind="chunk", seqs=3, low=0, high=2000, short=1500, long=4000, window=1024, heads=32, kv_heads=8, layers=1,
             dtype="bf16"),
        # an iteration of continuous batching: decode rows and small pieces of prompts side by side
        dict(name="chunk_mixed", kind="chunk", seqs=24, low=1, high=3000, short=1, long=96, window=0, heads=12, kv_heads=2, layers=2,
             dtype="f16"),
        # the operator itself in 32 bits, as programs call it that check a model's arithmetic
        dict(name="operator_f32", kind="operator", rows=96, total=777, heads=12, kv_heads=2, dim=128, dtype="f32"),
        # one prompt in, an answer out
        dict(name="generate", kind="generate", prompt=300, new=24),
        # a batch of prompts, then greedy decoding of all of them
        dict(name="serve", kind="serve", seqs=32, low=100, high=700, new=24),
        # a linear-recurrent mixer (gated delta rule, decays per channel) over eight prompts
        dict(name="delta", kind="delta", seqs=8, low=1024, high=1024, heads=16, rank=128),
    ]


def _log(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    heads, kv_heads = rng.choice([(12, 2), (12, 2), (32, 8)])
    kind = rng.choice(["step", "step", "step", "chunk", "chunk", "chunk", "operator", "generate", "serve", "delta"])
    if kind == "step":
        seqs = _log(rng, 1, 64)
        high = _log(rng, 64, min(131072, 262144 * 2 // (kv_heads * seqs)))
        return dict(kind=kind, seqs=seqs, low=max(1, int(high * rng.uniform(0.03, 1.0))), high=high, heads=heads, kv_heads=kv_heads,
                    layers=rng.randint(1, 4), dtype=rng.choice(["bf16", "bf16", "f16"]))
    if kind == "chunk":
        seqs = _log(rng, 1, 24)
        long = max(2, _log(rng, 16, 8192) // seqs)
        high = _log(rng, 16, 8192)
        return dict(kind=kind, seqs=seqs, low=rng.randint(0, high // 2), high=high, short=max(1, int(long * rng.uniform(0.05, 1.0))), long=long,
                    window=rng.choice([0, 0, 1024]), heads=heads, kv_heads=kv_heads, layers=rng.randint(1, 2),
                    dtype=rng.choice(["bf16", "bf16", "f16"]))
    if kind == "operator":
        rows = _log(rng, 1, 400)
        return dict(kind=kind, rows=rows, total=rows + rng.randint(0, 1200), heads=heads, kv_heads=kv_heads, dim=rng.choice([64, 128]),
                    dtype=rng.choice(["f32", "f32", "bf16", "f16"]))
    if kind == "generate":
        return dict(kind=kind, prompt=_log(rng, 10, 2000), new=rng.randint(4, 32))
    if kind == "serve":
        high = _log(rng, 50, 700)
        return dict(kind=kind, seqs=_log(rng, 2, 32), low=rng.randint(10, high), high=high, new=rng.randint(4, 24))
    seqs = _log(rng, 1, 8)
    high = _log(rng, 64, 8192 // seqs)
    return dict(kind=kind, seqs=seqs, low=max(TAPS, int(high * rng.uniform(0.1, 1.0))), high=high, heads=rng.choice([6, 16]),
                rank=rng.choice([0, 16, 128]))


# ---- inputs -------------------------------------------------------------------------------------------------------------


def _generators(seed):
    return torch.Generator(device="cuda").manual_seed(seed), np.random.default_rng(seed)


def _lengths(rng, n, low, high):
    return [int(x) for x in rng.integers(low, high + 1, n)]


def _i32(values):
    return torch.tensor(values, dtype=torch.int32, device="cuda")


def _randn(gen, *shape, dtype=torch.bfloat16, scale=1.0):
    return (torch.randn(*shape, generator=gen, device="cuda") * scale).to(dtype)


def _sizes(case):
    """Tokens before the pass and new tokens, of every sequence, for a case whose sizes do not depend on its seed's values."""
    rng = np.random.default_rng([int(case[k]) for k in ("seqs", "low", "high")])
    if case["kind"] == "step":
        return [(x - 1, 1) for x in _lengths(rng, case["seqs"], case["low"], case["high"])]
    if case["kind"] == "chunk":
        before = _lengths(rng, case["seqs"], case["low"], case["high"])
        return list(zip(before, _lengths(rng, case["seqs"], case["short"], case["long"])))
    return [(0, x) for x in _lengths(rng, case["seqs"], case["low"], case["high"])]


def _paged_inputs(case, seed):
    """Pages of every sequence in a pool's order, the pool's values, queries and new rows of every layer."""
    gen, rng = _generators(seed)
    sizes, dtype = _sizes(case), TORCH[case["dtype"]]
    counts = [-(-(before + new) // PAGE) for before, new in sizes]
    order = rng.permutation(sum(counts))
    ends = np.cumsum(counts)
    pages = [order[end - n:end].tolist() for n, end in zip(counts, ends)]
    rows, layers = sum(new for _, new in sizes), []
    for _ in range(case["layers"]):
        layers.append(dict(pool=_randn(gen, sum(counts), 2, case["kv_heads"], PAGE, D, dtype=dtype),
                           q=_randn(gen, rows, case["heads"], D, dtype=dtype), k=_randn(gen, rows, case["kv_heads"], D, dtype=dtype),
                           v=_randn(gen, rows, case["kv_heads"], D, dtype=dtype)))
    factor = torch.rand(rows, case["heads"], generator=gen, device="cuda") if case.get("window") else None
    return sizes, pages, layers, factor


class _DeviceMemory:
    """Memory of the framework's as torch.as_tensor takes it."""

    def __init__(self, address, shape, kind):
        self.__cuda_array_interface__ = {"data": (address, False), "shape": tuple(shape), "typestr": kind, "version": 3}


def _prepare_paged(case, seed):
    sizes, pages, layers, factor = _paged_inputs(case, seed)
    total = [before + new for before, new in sizes]
    cache = llaisys.PagedKVCache(sum(map(len, pages)), case["kv_heads"], D, page_size=PAGE, nlayer=case["layers"],
                                 dtype=llaisys.DataType[NAMES[case["dtype"]]], device=llaisys.DeviceType.NVIDIA, max_seqs=case["seqs"],
                                 max_pages_per_seq=max(map(len, pages)))
    cache.set_launch_overlap(True)
    ids = [cache.add_seq() for _ in sizes]
    for seq, mine in zip(ids, pages):
        cache.assign_pages(seq, mine)
    cache.flush()
    pool = []
    for i, layer in enumerate(layers):
        values = layer.pop("pool")
        pool.append(torch.as_tensor(_DeviceMemory(cache.pool_ptr(i), values.shape, "<i2"), device="cuda"))
        pool[i].copy_(values.view(torch.int16))
        layer["out"] = torch.empty_like(layer["q"])
    state = dict(kind=case["kind"], cache=cache, layers=layers, pool=pool, factor=factor, window=case.get("window", 0), heads=case["heads"],
                 n=len(ids), rows=sum(new for _, new in sizes), longest=max(total), most=max(new for _, new in sizes), ids=_i32(ids),
                 lens=_i32(total), starts=_i32([0, *np.cumsum([new for _, new in sizes]).tolist()]),
                 row_ids=_i32([s for s, (_, new) in zip(ids, sizes) for _ in range(new)]),
                 positions=_i32([before + t for before, new in sizes for t in range(new)]), stream=llaisys.context_stream())
    torch.cuda.synchronize()
    return state


def _wrap(tensor):
    """A torch tensor's values in a tensor of the framework's."""
    kind = {torch.float32: "F32", torch.bfloat16: "BF16", torch.float16: "F16"}[tensor.dtype]
    mine = llaisys.Tensor(tuple(tensor.shape), llaisys.DataType[kind], llaisys.DeviceType.NVIDIA)
    host = tensor.cpu()  # (load() takes an address)
    mine.load(host)
    return mine


def _operator_inputs(case, seed):
    gen, dtype = _generators(seed)[0], TORCH[case["dtype"]]
    return (_randn(gen, case["rows"], case["heads"], case["dim"], dtype=dtype),
            *(_randn(gen, case["total"], case["kv_heads"], case["dim"], dtype=dtype) for _ in range(2)))


def _config():
    return {"hidden_size": WIDTH, "num_attention_heads": 12, "num_key_value_heads": 2, "head_dim": D, "intermediate_size": FF,
            "num_hidden_layers": MODEL_LAYERS, "vocab_size": VOCAB, "rms_norm_eps": EPS, "rope_theta": THETA}


def _model_weights(gen, rng):
    """Random layers between an embedding and a vocabulary projection that agree on what follows a token, so that the greedy choice is as
    clear as a trained model's."""
    following = torch.from_numpy(rng.permutation(VOCAB)).to("cuda")
    embed = _randn(gen, VOCAB, WIDTH)
    head = torch.empty_like(embed)
    head[following] = (embed.float() * 0.02).bfloat16()
    yield "model.embed_tokens.weight", embed
    yield "lm_head.weight", head
    yield "model.norm.weight", 1 + _randn(gen, WIDTH, scale=0.1)
    for i in range(MODEL_LAYERS):
        p = f"model.layers.{i}."
        yield p + "input_layernorm.weight", 1 + _randn(gen, WIDTH, scale=0.1)
        yield p + "post_attention_layernorm.weight", 1 + _randn(gen, WIDTH, scale=0.1)
        for name, rows in (("q", 12 * D), ("k", 2 * D), ("v", 2 * D)):
            yield p + f"self_attn.{name}_proj.weight", _randn(gen, rows, WIDTH, scale=0.02)
            yield p + f"self_attn.{name}_proj.bias", _randn(gen, rows, scale=0.02)
        yield p + "self_attn.o_proj.weight", _randn(gen, WIDTH, 12 * D, scale=0.02)
        yield p + "mlp.gate_proj.weight", _randn(gen, FF, WIDTH, scale=0.02)
        yield p + "mlp.up_proj.weight", _randn(gen, FF, WIDTH, scale=0.02)
        yield p + "mlp.down_proj.weight", _randn(gen, WIDTH, FF, scale=0.02)


def _prompts(case, rng):
    lens = [case["prompt"]] if case["kind"] == "generate" else [new for _, new in _sizes(case)]
    return [rng.integers(0, VOCAB, n).tolist() for n in lens]


def _prepare_model(case, seed):
    gen, rng = _generators(seed)
    prompts = _prompts(case, rng)
    longest = max(map(len, prompts)) + case["new"] + PAGE
    model = llaisys.models.Qwen2(config=_config(), device=llaisys.DeviceType.NVIDIA, dtype=llaisys.DataType.BF16, max_seq_len=longest)
    for name, value in _model_weights(gen, rng):
        model.load_tensor(name, value)
    model.configure_cache(len(prompts), longest)
    torch.cuda.synchronize()
    return dict(kind=case["kind"], model=model, prompts=prompts, new=case["new"])


def _delta_inputs(case, seed):
    gen = _generators(seed)[0]
    lens, heads, rank = [new for _, new in _sizes(case)], case["heads"], case["rank"]
    at, width = {}, 0
    for name, n in (("q", heads * D), ("k", heads * D), ("v", heads * D), ("b", heads), ("a", rank or heads), ("g", heads * D)):
        at[name], width = width, width + (n + 7) // 8 * 8
    t = dict(proj=_randn(gen, sum(lens), width, scale=0.7), conv_q=_randn(gen, heads * D, TAPS, scale=0.5),
             conv_k=_randn(gen, heads * D, TAPS, scale=0.5), conv_v=_randn(gen, heads * D, TAPS, scale=0.5),
             decay_w=_randn(gen, heads * D, rank, scale=0.3 / math.sqrt(max(rank, 1) / 16)) if rank else None, a_log=_randn(gen, heads, scale=0.1),
             dt_bias=_randn(gen, heads * D if rank else heads) - 5, norm_w=1 + _randn(gen, D, scale=0.1))
    return lens, at, width, t


def _prepare_delta(case, seed):
    lens, at, width, t = _delta_inputs(case, seed)
    heads, rank, rows, kind = case["heads"], case["rank"], sum(lens), llaisys.DataType.BF16
    floats, n_scratch, n_segments = llaisys.gated_delta_sizes(kind, rows, heads, heads, D, D, TAPS)
    state = torch.zeros(len(lens), floats, device="cuda")
    out = torch.empty(rows, heads * D, dtype=torch.bfloat16, device="cuda")
    keep = [_i32(list(range(len(lens)))), _i32([0, *np.cumsum(lens).tolist()]), _i32(lens), torch.empty(n_scratch, device="cuda"),
            torch.empty(max(n_segments, 1), device="cuda")]
    call = dict(row_stride=width, **{name + "_at": at[name] for name in "qkvba"}, **t, decay_ld=rank, gate=t["proj"].data_ptr() + at["g"] * 2,
                gate_stride=width, gate_silu=1, q_scale=D ** -0.5, eps=EPS, unit_eps=1e-6, taps=TAPS, heads=heads, kv_heads=heads, dk=D, dv=D,
                rank=rank, state=state, slot_stride=floats, seq_ids_dev=keep[0], q_starts_dev=keep[1], kv_lens_dev=keep[2], n_seqs=len(lens),
                n_rows=rows, max_q_len=max(lens), out=out, out_stride=heads * D, scratch=keep[3], scratch_floats=n_scratch,
                scratch_segments=keep[4], scratch_segment_floats=n_segments)
    torch.cuda.synchronize()
    return dict(kind="delta", call=call, out=out, state=state, stream=llaisys.context_stream())


def prepare(case, seed):
    llaisys.set_context_runtime(llaisys.DeviceType.NVIDIA, 0)
    if case["kind"] in ("step", "chunk"):
        return _prepare_paged(case, seed)
    if case["kind"] == "operator":
        q, k, v = (_wrap(x) for x in _operator_inputs(case, seed))
        out = _wrap(torch.zeros(case["rows"], case["heads"], case["dim"], dtype=TORCH[case["dtype"]]))
        seen = _DeviceMemory(out.data_ptr(), out.shape(), "<f4" if case["dtype"] == "f32" else "<i2")
        view = torch.as_tensor(seen, device="cuda")
        torch.cuda.synchronize()
        return dict(kind="operator", q=q, k=k, v=v, out=out, view=view if case["dtype"] == "f32" else view.view(TORCH[case["dtype"]]),
                    scale=case["dim"] ** -0.5)
    return _prepare_delta(case, seed) if case["kind"] == "delta" else _prepare_model(case, seed)


# ---- passes -------------------------------------------------------------------------------------------------------------


def run(state):
    kind = state["kind"]
    if kind == "step":
        for i, t in enumerate(state["layers"]):
            state["cache"].decode_step_dev(i, t["out"], t["q"], t["k"], t["v"], state["ids"], state["lens"], state["n"], state["longest"],
                                           state["heads"], D ** -0.5, state["stream"])
        return {"out": [t["out"] for t in state["layers"]], "pool": state["pool"]}
    if kind == "chunk":
        cache = state["cache"]
        for i, t in enumerate(state["layers"]):
            cache.append_dev(i, t["k"], t["v"], state["row_ids"], state["positions"], state["rows"], state["stream"])
            if state["window"]:
                cache.attention_dev(i, t["out"], t["q"], state["ids"], state["starts"], state["lens"], n_seqs=state["n"], total_q=state["rows"],
                                    max_q_len=state["most"], max_kv_len=state["longest"], nh=state["heads"], scale=D ** -0.5,
                                    stream=state["stream"], window=state["window"], row_scale=state["factor"])
            else:
                cache.prefill_dev(i, t["out"], t["q"], state["ids"], state["starts"], state["lens"], state["n"], state["rows"], state["most"],
                                  state["longest"], state["heads"], D ** -0.5, state["stream"])
        return {"out": [t["out"] for t in state["layers"]], "pool": state["pool"]}
    if kind == "operator":
        llaisys.Ops.self_attention(state["out"], state["q"], state["k"], state["v"], state["scale"])
        return state["view"]
    if kind == "generate":
        tokens = state["model"].generate(state["prompts"][0], max_new_tokens=state["new"])
        return {"tokens": np.array(tokens), "logits": state["model"].last_logits()}
    if kind == "serve":
        model = state["model"]
        seqs = [model.add_seq() for _ in state["prompts"]]
        first = model.step(seqs, state["prompts"])
        tokens = model.decode_loop(seqs, first, state["new"])
        logits = model.last_logits(len(seqs))
        for seq in seqs:
            model.free_seq(seq)
        return {"first": np.array(first), "tokens": tokens, "logits": logits}
    llaisys.gated_delta_dev(llaisys.DataType.BF16, decode=False, stream=state["stream"], **state["call"])
    return {"out": state["out"], "state": state["state"]}


# ---- what a pass cannot do without ----------------------------------------------------------------------------------------


def _seen(before, new, window):
    """(query, key) pairs of `new` tokens behind `before` others."""
    return sum(min(p + 1, window) if window else p + 1 for p in range(before, before + new))


def work(case):
    kind = case["kind"]
    if kind in ("step", "chunk"):
        sizes, size = _sizes(case), 2
        window = case.get("window", 0)
        rows = sum(new for _, new in sizes)
        cached = sum(before if not window else min(before, window - 1) for before, _ in sizes)
        per_layer = cached * case["kv_heads"] * 2 * D * size + rows * (2 * case["heads"] + 4 * case["kv_heads"]) * D * size
        pairs = sum(_seen(before, new, window) for before, new in sizes)
        return {"bytes": case["layers"] * per_layer, "flops": case["layers"] * 4.0 * D * case["heads"] * pairs}
    if kind == "operator":
        size = 4 if case["dtype"] == "f32" else 2
        pairs = _seen(case["total"] - case["rows"], case["rows"], 0)
        return {"bytes": size * case["dim"] * (2 * case["rows"] * case["heads"] + 2 * case["total"] * case["kv_heads"]),
                "flops": 4.0 * case["dim"] * case["heads"] * pairs}
    if kind == "delta":
        rows, heads = sum(new for _, new in _sizes(case)), case["heads"]
        width = 4 * heads * D + heads + (case["rank"] or heads)
        return {"bytes": rows * (width + heads * D) * 2 + case["seqs"] * (heads * D * D + TAPS * 3 * heads * D) * 4,
                "flops": rows * heads * (6.0 * D * D + 2.0 * D * case["rank"])}
    lens = [case["prompt"]] if kind == "generate" else [new for _, new in _sizes(case)]
    new = case["new"] if kind == "serve" else case["new"] - 1  # steps behind the prompt's
    per_token = MODEL_LAYERS * (WIDTH * 16 * D + WIDTH * 12 * D + 3 * WIDTH * FF)
    head, kv = VOCAB * WIDTH, MODEL_LAYERS * 2 * 2 * D
    tokens = sum(lens) + new * len(lens)
    pairs = sum(_seen(0, n + new, 0) for n in lens)
    cached = sum(n + t for n in lens for t in range(new))
    return {"bytes": (1 + new) * (per_token + head) * 2 + (tokens + cached) * kv * 2 + len(lens) * VOCAB * 4,
            "flops": 2.0 * tokens * per_token + 2.0 * (1 + new) * len(lens) * head + 4.0 * D * 12 * MODEL_LAYERS * pairs}


def tolerance(case):
    # about four times what each path is off from 64 bits: the rounding of its results and, in bf16, of its weights
    if case["kind"] in ("generate", "serve"):
        return {"rel": 0.03}
    if case["kind"] == "delta":
        return {"rel": 0.012}
    return {"rel": {"bf16": 1e-2, "f16": 1.2e-3, "f32": 2e-6}[case["dtype"]]}


# ---- the same in 64 bits ----------------------------------------------------------------------------------------------------


def _attend(q, k, v, window=0):
    """q [n, H, d] are the newest of k, v [total, G, d]: causal attention, head h of q with head h // (H / G) of k and v."""
    n, heads, d = q.shape
    total, share = k.shape[0], heads // k.shape[1]
    out = torch.empty(n, heads, v.shape[2], dtype=torch.float64, device=q.device)
    keys = torch.arange(total, device=q.device)
    for at in range(0, n, 2048):
        rows = torch.arange(at, min(n, at + 2048), device=q.device) + total - n
        hidden = keys[None, :] > rows[:, None]
        if window:
            hidden |= keys[None, :] <= rows[:, None] - window
        for h in range(heads):
            scores = q[at:at + 2048, h].double() @ k[:, h // share].double().T / math.sqrt(d)
            out[at:at + 2048, h] = torch.softmax(scores.masked_fill_(hidden, -math.inf), dim=1) @ v[:, h // share].double()
    return out


def _exact_paged(case, seed):
    sizes, pages, layers, factor = _paged_inputs(case, seed)
    outs = []
    for layer in layers:
        parts, row = [], 0
        for (before, new), mine in zip(sizes, pages):
            held = layer["pool"][torch.tensor(mine, device="cuda")]  # [pages, K|V, head, slot, d]
            k, v = (held[:, i].permute(0, 2, 1, 3).reshape(-1, case["kv_heads"], D)[:before + new].clone() for i in range(2))
            k[before:], v[before:] = layer["k"][row:row + new], layer["v"][row:row + new]
            parts.append(_attend(layer["q"][row:row + new], k, v, case.get("window", 0)))
            row += new
        outs.append(torch.cat(parts))
        if factor is not None:
            outs[-1] *= factor.double().unsqueeze(2)
    return {"out": outs, "pool": [None] * len(layers)}


def _rms(x, eps=EPS):
    return x / torch.sqrt(x.square().mean(-1, keepdim=True) + eps)


def _rotate(x):
    """x [T, H, d] at positions 0, 1, ..: dims i and i + d / 2 turned by position / theta^(2 i / d)."""
    half = x.shape[2] // 2
    freq = THETA ** (-torch.arange(half, dtype=torch.float64, device=x.device) / half)
    angle = torch.arange(x.shape[0], dtype=torch.float64, device=x.device)[:, None] * freq
    cos, sin = angle.cos()[:, None], angle.sin()[:, None]
    a, b = x[..., :half], x[..., half:]
    return torch.cat([a * cos - b * sin, b * cos + a * sin], dim=2)


def _exact_model(case, seed):
    gen, rng = _generators(seed)
    prompts = _prompts(case, rng)
    w = dict(_model_weights(gen, rng))
    follow = np.empty(VOCAB, dtype=np.int64)  # the weights were made to agree on this choice; the argmax below says whether they do
    rng = _generators(seed)[1]
    _prompts(case, rng)
    follow[:] = rng.permutation(VOCAB)
    fed, new = [], case["new"] if case["kind"] == "serve" else case["new"] - 1
    for prompt in prompts:
        fed.append(list(prompt))
        for _ in range(new):
            fed[-1].append(int(follow[fed[-1][-1]]))
    ends = np.cumsum([len(f) for f in fed]).tolist()
    x = w["model.embed_tokens.weight"][torch.tensor([t for f in fed for t in f], device="cuda")].double()
    for i in range(MODEL_LAYERS):
        p = f"model.layers.{i}."

        def linear(y, name):
            return y @ w[p + name + ".weight"].double().T

        h = _rms(x) * w[p + "input_layernorm.weight"].double()
        q, k, v = ((linear(h, f"self_attn.{n}_proj") + w[p + f"self_attn.{n}_proj.bias"].double()).view(x.shape[0], -1, D) for n in "qkv")
        parts = [_attend(_rotate(q[e - len(f):e]), _rotate(k[e - len(f):e]), v[e - len(f):e]) for f, e in zip(fed, ends)]
        x = x + linear(torch.cat(parts).reshape(x.shape[0], -1), "self_attn.o_proj")
        h = _rms(x) * w[p + "post_attention_layernorm.weight"].double()
        x = x + linear(torch.nn.functional.silu(linear(h, "mlp.gate_proj")) * linear(h, "mlp.up_proj"), "mlp.down_proj")
    x = _rms(x) * w["model.norm.weight"].double()
    head = w["lm_head.weight"].double()
    rows = [x[e - 1 - new:e] for e in ends]  # the last token of the prompt, then every token decoded
    chosen = [(r @ head.T).argmax(1).cpu().numpy() for r in rows]
    logits = torch.stack([r[-1] for r in rows]) @ head.T
    if case["kind"] == "generate":
        return {"tokens": np.concatenate([np.array(prompts[0]), chosen[0]]), "logits": logits}
    return {"first": np.array([c[0] for c in chosen]), "tokens": np.stack([c[1:] for c in chosen], axis=1), "logits": logits}


def _exact_delta(case, seed):
    lens, at, _, t = _delta_inputs(case, seed)
    heads, rank, most = case["heads"], case["rank"], max(lens)
    t = {name: None if x is None else x.double() for name, x in t.items()}
    proj = torch.zeros(len(lens), most, t["proj"].shape[1], dtype=torch.float64, device="cuda")
    live = torch.arange(most, device="cuda")[None, :] < torch.tensor(lens, device="cuda")[:, None]
    proj[live] = t["proj"]

    def part(name, n):
        return proj[..., at[name]:at[name] + n]

    def conv(name):
        x, y = part(name, heads * D), 0
        for back in range(TAPS):
            y = y + torch.nn.functional.pad(x, (0, 0, back, 0))[:, :most] * t["conv_" + name][:, TAPS - 1 - back]
        return torch.nn.functional.silu(y).view(len(lens), most, heads, D)

    def unit(x):
        return x / torch.sqrt(x.square().sum(-1, keepdim=True) + 1e-6)

    q, k, v = unit(conv("q")) * D ** -0.5, unit(conv("k")), conv("v")
    beta = torch.sigmoid(part("b", heads))
    if rank:
        inner = (part("a", rank) @ t["decay_w"].T + t["dt_bias"]).view(len(lens), most, heads, D)
    else:
        inner = (part("a", heads) + t["dt_bias"]).unsqueeze(-1).expand(len(lens), most, heads, D)
    decay = torch.exp(-torch.exp(t["a_log"])[:, None] * torch.nn.functional.softplus(inner))
    S = torch.zeros(len(lens), heads, D, D, dtype=torch.float64, device="cuda")
    y = torch.empty(len(lens), most, heads, D, dtype=torch.float64, device="cuda")
    for i in range(most):
        now = S * decay[:, i].unsqueeze(-1)
        u = beta[:, i].unsqueeze(-1) * (v[:, i] - torch.einsum("nhdv,nhd->nhv", now, k[:, i]))
        now = now + k[:, i].unsqueeze(-1) * u.unsqueeze(-2)
        y[:, i] = torch.einsum("nhdv,nhd->nhv", now, q[:, i])
        S = torch.where(live[:, i, None, None, None], now, S)
    y = (_rms(y) * t["norm_w"]).flatten(2) * torch.nn.functional.silu(part("g", heads * D))
    ring = torch.zeros(len(lens), TAPS, 3 * heads * D, dtype=torch.float64, device="cuda")
    raw = torch.cat([part(n, heads * D) for n in "qkv"], dim=2)
    for s, n in enumerate(lens):
        for p in range(n - TAPS, n):
            ring[s, p % TAPS] = raw[s, p]
    return {"out": y[live], "state": torch.cat([S.flatten(1), ring.flatten(1)], dim=1)}


def exact(case, seed):
    with torch.no_grad():
        if case["kind"] in ("step", "chunk"):
            return _exact_paged(case, seed)
        if case["kind"] == "operator":
            return _attend(*_operator_inputs(case, seed))
        return _exact_delta(case, seed) if case["kind"] == "delta" else _exact_model(case, seed)
