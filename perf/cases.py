"""Cases that stand for the work of this framework in use: one step of a model, through the models' own entry points.

A decode step is a replay of the program's CUDA graph over ``forward`` and ``logits``, a prompt step an eager call of the two, the
vision tower one ``encode_vision``; inputs, weights and paged caches are random and lie on the GPU.  The layer sizes are those of
the repository's layer benchmarks: four layers at width 4096 (the widths of Qwen3-VL-8B's decoder) or 2048, a vocabulary of
32768, and the 8B model's whole vision tower.  What is left out of a whole model is only more of the same layers.

Sequence lengths of a batch run from a quarter of ``tokens`` to all of it, no two alike, unless ``even`` is set.
"""

import math

import torch

from prism_infer_b200 import ops
from prism_infer_b200.models import architecture as A
from prism_infer_b200.models.common import AttnMeta
from prism_infer_b200.models.model_registry import load_model_class, resolve_model_family
from prism_infer_b200.models.weights import iter_random_weights
from prism_infer_b200.ops.recurrent import StateCache

LAYERS, VOCAB, PAGE, WINDOW, KEEP, SIDE, STATE, RANK = 4, 32_768, 256, 1024, 16, 256, 64, 64
# width -> heads, key heads, head width, feed-forward, latent, experts, chosen, expert feed-forward
SIZES = {2048: (16, 4, 128, 6144, 256, 32, 4, 768), 4096: (32, 8, 128, 12288, 512, 32, 4, 1536)}
KV_MODES = {"bf16": ops.KV_BF16, "fp8": ops.KV_FP8, "scaled_fp8": ops.KV_FP8_SCALED}
DEV = "cuda"


def listed():
    def text(name, family, step, batch, tokens, *, width=4096, history=0, kv="bf16", even=True):
        return dict(name=name, family=family, step=step, width=width, batch=batch, tokens=tokens, history=history, kv=kv, even=even)

    return [
        # the smallest call: one user of a small model, a short conversation; launches and latency
        text("decode 1, width 2048", "grouped", "decode", 1, 333, width=2048),
        # the headline workload's decode step: one request of eight images, batch 1, scaled 8-bit cache
        text("decode 1", "grouped", "decode", 1, 1650, kv="scaled_fp8"),
        # a server under load: a few dozen conversations of different lengths
        text("decode 32", "grouped", "decode", 32, 2048, kv="scaled_fp8", even=False),
        # throughput serving: a full batch of shorter requests, 16-bit cache
        text("decode 128", "grouped", "decode", 128, 1024, even=False),
        # first token of a question about one image
        text("prompt 230", "grouped", "prompt", 1, 230, kv="scaled_fp8"),
        # first token of the headline request
        text("prompt 1616", "grouped", "prompt", 1, 1616, kv="scaled_fp8"),
        # a prompt step that batches several requests
        text("prompts 8 up to 1500", "grouped", "prompt", 8, 1500, even=False),
        # the last chunk of a long prompt, over the cached ones before it
        text("chunk 2048 after 14336", "grouped", "prompt", 1, 2048, history=14336, kv="scaled_fp8"),
        # the images of the headline request
        dict(name="vision 8 x 448", family="vision", step="encode", images=8, rows=28, cols=28),
        # the other families: latent attention, experts behind windowed attention, recurrence in front of experts
        text("latent decode 32", "latent", "decode", 32, 2048, even=False),
        text("experts prompt 2048", "experts", "prompt", 1, 2048),
        text("recurrent decode 32", "recurrent", "decode", 32, 2048, even=False),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["decode"] * 4 + ["prompt"] * 3 + ["chunk", "vision", "other", "other", "other"])
    width, kv = rng.choice([2048, 4096, 4096]), rng.choice(sorted(KV_MODES))
    if kind == "vision":
        return dict(family="vision", step="encode", images=log(1, 8), rows=2 * rng.randint(6, 14), cols=2 * rng.randint(6, 14))
    case = dict(family="grouped", step="decode", width=width, batch=1, tokens=0, history=0, kv=kv, even=bool(rng.randint(0, 1)))
    if kind == "other":
        case.update(family=rng.choice(["latent", "experts", "recurrent"]), kv="bf16")
        kind = rng.choice(["decode", "prompt"])
    if kind == "decode":
        case["batch"] = log(1, 128)
        case["tokens"] = log(16, min(4096, 131072 // case["batch"]))
    elif kind == "prompt":
        case.update(step="prompt", batch=rng.choice([1, 1, 2, 3, 5, 8]))
        case["tokens"] = log(16, (2048 if case["family"] != "grouped" else 8192) // case["batch"])
    else:
        case.update(step="prompt", tokens=log(64, 2048), history=log(256, 14336))
    return case


# ------------------------------------------------------------------------------------------------ inputs
def _generator(seed, salt):
    return torch.Generator(DEV).manual_seed(seed * 7919 + salt)


def _arch(case):
    if case["family"] == "vision":
        return A.Qwen3VLArch(text=A.TextArch(vocab_size=1024, num_layers=1), image_token_id=1023, video_token_id=1022, vision_start_token_id=1021,
                             vision_end_token_id=1020, eos_token_id=1019)
    width = case["width"]
    heads, groups, dim, ff, rank, experts, top, expert_ff = SIZES[width]
    if case["family"] == "grouped":
        tower = A.VisionArch(hidden_size=128, depth=1, num_heads=4, intermediate_size=256, num_position_embeddings=256, out_hidden_size=width,
                             deepstack_visual_indexes=(0,))
        return A.Qwen3VLArch(text=A.TextArch(vocab_size=VOCAB, hidden_size=width, num_layers=LAYERS, num_heads=heads, num_kv_heads=groups,
                                             head_dim=dim, intermediate_size=ff), vision=tower, image_token_id=VOCAB - 1,
                             video_token_id=VOCAB - 2, vision_start_token_id=VOCAB - 3, vision_end_token_id=VOCAB - 4, eos_token_id=VOCAB - 5)
    if case["family"] == "latent":
        return A.PoralornArch.like_8b(LAYERS, width=width, heads=heads, dim=dim, kv_rank=rank, ff=ff, vocab_size=VOCAB)
    if case["family"] == "experts":
        mixer = A.WindowAttentionArch(heads=heads, kv_heads=groups, dim=dim, vdim=dim, scale=dim ** -0.5, rot=A.RotaryArch(1e6, dim),
                                      window=WINDOW, keep_first=KEEP, qk_norm=True, gate=True)
        layer = A.DolidraLayer(mixer, moe=A.MixtureArch(experts, top, expert_ff, expert_ff))
        return A.DolidraArch(vocab_size=VOCAB, width=width, layers=(layer,) * LAYERS, side_dim=SIDE)
    moe = A.MixtureArch(experts, top, expert_ff, expert_ff, scored=True, groups=4, groups_kept=2, scale=2.5, shared_gate=True)
    return A.BokoraxArch(vocab_size=VOCAB, width=width, layers=(A.BokoraxLayer(A.TimeMixArch(width // STATE, STATE, RANK), moe),) * LAYERS)


def _weights(case, seed):
    """Random weights by their checkpoint names.  A trained router is decisive and its experts are used alike: every token's embedding
    leans towards the router rows of experts drawn for it, so that no choice hangs on a rounding error."""
    arch = _arch(case)
    w = dict(iter_random_weights(arch, dtype=torch.bfloat16, device=DEV, seed=seed))
    if case["family"] in ("experts", "recurrent"):
        g, moe, width = _generator(seed, 4), arch.layers[0].moe, case["width"]
        embed = torch.randn(VOCAB, width, generator=g, device=DEV)
        for i in range(LAYERS):
            open_ = torch.rand(VOCAB, moe.groups, 1, generator=g, device=DEV).topk(moe.groups_kept, 1).indices
            order = torch.rand(VOCAB, moe.groups, moe.experts // moe.groups, generator=g, device=DEV)
            chosen = torch.zeros_like(order).scatter_(2, order.topk(moe.top // moe.groups_kept, 2).indices, 1.0)
            chosen *= torch.zeros_like(order[:, :, :1]).scatter_(1, open_, 1.0)
            embed += 0.15 * math.sqrt(width) * chosen.flatten(1) @ torch.nn.functional.normalize(w[f"l{i}.mlp.router"].float(), dim=1)
        w["embed"] = (3.0 * embed).to(torch.bfloat16)
    return w


def _lengths(case):
    """(new tokens, tokens up to the last of them) of every sequence."""
    def share(i):
        return 1.0 if case["even"] else 0.25 + 0.75 * (((i + 1) * 0.6180339887) % 1.0)

    sizes = [max(1, round(case["tokens"] * share(i))) for i in range(case["batch"])]
    return [(1, n) for n in sizes] if case["step"] == "decode" else [(n, case["history"] + n) for n in sizes]


def _positions(first, count):
    """Three-axis positions of a prompt's tokens: images of 14 x 14 merged patches with four words between them."""
    i = torch.arange(first, first + count)
    base, r = i // 200 * 18, i % 200
    cell = (r - 4).clamp_min(0)
    word = torch.where(r < 4, r, torch.full_like(r, 4))
    return torch.stack([base + word, base + word + cell // 14, base + word + cell % 14])


def _inputs(case, seed):
    """Token ids, positions, pages and slots of a step."""
    lens, g = _lengths(case), _generator(seed, 1)
    pages = [-(-total // PAGE) for _, total in lens]
    order = torch.randperm(sum(pages), generator=g, device=DEV).to(torch.int32)
    table = torch.full((len(lens), max(pages)), -1, dtype=torch.int32, device=DEV)
    slots, positions, at = [], [], 0
    for s, (new, total) in enumerate(lens):
        table[s, :pages[s]] = order[at:at + pages[s]]
        at += pages[s]
        i = torch.arange(total - new, total, device=DEV)
        slots.append(table[s, i // PAGE].long() * PAGE + i % PAGE)
        plain = case["family"] != "grouped" or case["step"] == "decode"
        positions.append(torch.arange(total - new, total).expand(3, -1) if plain else _positions(total - new, new))
    ids = torch.randint(0, VOCAB - 8, (sum(n for n, _ in lens),), generator=g, device=DEV)
    return dict(lens=lens, pages=sum(pages), table=table, slots=torch.cat(slots), ids=ids,
                positions=torch.cat(positions, 1).to(DEV, torch.int32).contiguous())


def _fill(case, seed, cache, state):
    """What earlier steps left behind: normal keys, values and latents (their norms make them so), a recurrent state of order one."""
    if case["step"] == "prompt" and not case["history"]:
        return
    g = _generator(seed, 2)
    flat = cache.payload.view(-1, cache.payload.shape[-1] if not cache.rows else cache.rows[0])
    for lo in range(0, flat.shape[0], 1 << 20):
        x = torch.randn(flat[lo:lo + (1 << 20)].shape, generator=g, device=DEV, dtype=torch.bfloat16)
        if cache.mode == ops.KV_BF16:
            flat[lo:lo + (1 << 20)] = x
        else:
            q, scale = ops.quantize_fp8_rows(x, cache.mode == ops.KV_FP8_SCALED)
            flat[lo:lo + (1 << 20)] = q
            if scale is not None:
                cache.scales.view(-1)[lo:lo + (1 << 20)] = scale
    for i in range(len(state.sizes) if state is not None else 0):
        state.layer(i).normal_(generator=g)


def _containers(case, arch, pages):
    g = arch.kv_geometry()
    cache = ops.KVCache(g.layers, pages, g.heads, PAGE, g.row, KV_MODES[case["kv"]], DEV, planes=g.planes, rows=g.rows)
    return cache, (StateCache(arch.state_sizes(), case["batch"], DEV) if arch.state_sizes() else None)


def _model(case, seed):
    arch = _arch(case)
    ops.set_pdl(True)
    ops.apply_tuning()
    model = load_model_class(resolve_model_family(arch.model_type))(arch, device=DEV, dtype=torch.bfloat16)
    model.load(_weights(case, seed).items())
    return arch, model


def _pixels(case, seed):
    grid = [(1, case["rows"], case["cols"])] * case["images"]
    n = case["images"] * case["rows"] * case["cols"]
    return torch.rand((n, 3 * 2 * 16 * 16), generator=_generator(seed, 3), device=DEV).mul(2).sub(1).to(torch.bfloat16), grid


def prepare(case, seed):
    arch, model = _model(case, seed)
    if case["family"] == "vision":
        pixels, grid = _pixels(case, seed)
        return dict(model=model, pixels=pixels, grid=grid)
    x = _inputs(case, seed)
    lens = x["lens"]
    cache, state = _containers(case, arch, x["pages"])
    _fill(case, seed, cache, state)
    new, total = ([l[k] for l in lens] for k in (0, 1))
    i32 = dict(dtype=torch.int32, device=DEV)
    extra = dict(state=state, state_slots=torch.arange(len(lens), **i32)) if state is not None else {}
    st = dict(model=model, cache=cache, state=state, ids=x["ids"], positions=x["positions"])
    if case["step"] == "prompt":
        cu = [0]
        for n in new:
            cu.append(cu[-1] + n)
        st["meta"] = AttnMeta(is_prefill=True, block_tables=x["table"], slots=x["slots"], cu_seqlens_q=torch.tensor(cu, **i32),
                              kv_lens=torch.tensor(total, **i32), max_q_len=max(new), no_history=new == total, total_kv=sum(total),
                              max_kv_len=max(total), host_lens=lens, attended_pairs=sum(a * b for a, b in lens), **extra)
        if new != total:
            st["meta"].cu_seqlens_kv = torch.tensor([0] + torch.tensor(total).cumsum(0).tolist(), **i32)
        st["last"] = torch.tensor(cu[1:], device=DEV) - 1
        return st
    st["meta"] = AttnMeta(is_prefill=False, block_tables=x["table"], slots=x["slots"], context_lens=torch.tensor(total, **i32), **extra)
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        _forward(st)
        stream.synchronize()
        st["graph"] = torch.cuda.CUDAGraph()
        with torch.cuda.graph(st["graph"], stream=stream):
            st["out"] = _forward(st)
    torch.cuda.current_stream().wait_stream(stream)
    return st


def _forward(st):
    hidden = st["model"].forward(st["ids"], st["positions"], st["meta"], st["cache"])
    rows = hidden[st["last"]] if "last" in st else hidden
    return hidden, st["model"].logits(rows)


def run(state):
    if "pixels" in state:
        return list(_flat(state["model"].encode_vision(state["pixels"], state["grid"])))
    if "graph" in state:
        state["graph"].replay()
        hidden, logits = state["out"]
    else:
        hidden, logits = _forward(state)
    out = dict(hidden=hidden, logits=logits.reshape(-1, VOCAB), cache=state["cache"].payload)
    if state["cache"].scales is not None:
        out["scales"] = state["cache"].scales
    if state["state"] is not None:
        out["state"] = [state["state"].layer(i) for i in range(LAYERS)]
    return out


def _flat(pair):
    main, deep = pair
    yield main
    yield from deep


# --------------------------------------------------------------------------------------------------- work
def work(case):
    if case["family"] == "vision":
        v = A.VisionArch()
        n, h, f = case["images"] * case["rows"] * case["cols"], v.hidden_size, v.intermediate_size
        mergers = 1 + len(v.deepstack_visual_indexes)
        block, merger, patch = 4 * h * h + 2 * h * f, v.merged_dim * (v.merged_dim + v.out_hidden_size), v.patch_input_dim * h
        attention = 4 * n * case["rows"] * case["cols"] * h * v.depth
        return dict(bytes=2 * (v.depth * block + mergers * merger + patch) + 2 * n * v.patch_input_dim + 2 * mergers * (n // 4) * v.out_hidden_size,
                    flops=2 * n * (v.depth * block + patch) + 2 * (n // 4) * mergers * merger + attention)
    width = case["width"]
    heads, groups, dim, ff, rank, experts, top, expert_ff = SIZES[width]
    lens = _lengths(case)
    tokens, last = sum(n for n, _ in lens), len(lens)
    used = experts * (1.0 - (1.0 - top / experts) ** tokens) + 1
    moe_bytes, moe_flops = used * 3 * width * expert_ff, (top + 1) * 3 * width * expert_ff
    window = WINDOW + KEEP if case["family"] == "experts" else 1 << 30
    pairs = sum(sum(min(window, total - new + i + 1) for i in range(new)) for new, total in lens)
    seen = sum(min(total, new + window) for new, total in lens)   # cached rows that a step reads or writes
    if case["family"] == "grouped":
        weights = active = (2 * heads + 2 * groups) * dim * width + 3 * width * ff
        row, pair = 2 * groups * dim * (2 if case["kv"] == "bf16" else 1) + (8 * groups if case["kv"] == "scaled_fp8" else 0), 4 * heads * dim
    elif case["family"] == "latent":
        weights = active = (3 * heads * dim + rank + 2 * width) * width + 2 * heads * dim * rank + 2 * width * ff
        row, pair = 2 * rank, 4 * heads * (rank if case["step"] == "decode" else dim)
    elif case["family"] == "experts":
        weights = active = (2 * heads + 2 * groups) * dim * width + (heads + experts + 2 * SIDE) * width
        row, pair = 4 * groups * dim, 4 * heads * dim
    else:
        weights = active = 5 * width * width + (2 * RANK + experts + 1) * width
        row, pair, seen, pairs = 2 * 4 * (STATE + 1) * width, 8 * STATE * width, last, tokens
    if case["family"] in ("experts", "recurrent"):
        weights, active = weights + moe_bytes, active + moe_flops
    return dict(bytes=LAYERS * (2 * weights + seen * row) + 2 * VOCAB * width + tokens * width * 4 + last * VOCAB * 4,
                flops=LAYERS * (2 * tokens * active + pairs * pair) + 2 * last * VOCAB * width)


def tolerance(case):
    """Measured against ``exact``: 0.013 - 0.024 where the residual stream is bf16 (Qwen3-VL), 0.005 and 0.0035 where it is fp32; the
    largest single difference is about five times that."""
    rel = {"latent": 0.02, "experts": 0.015, "recurrent": 0.015}.get(case["family"], 0.03)
    return {"rel": rel, "max": 0.4 if rel == 0.03 else 0.2}


# -------------------------------------------------------------------------------- the same in 64 bits
def exact(case, seed):
    w = _weights(case, seed)
    if case["family"] == "vision":
        return _exact_vision(case, w, *_pixels(case, seed))
    x = _inputs(case, seed)
    arch = _arch(case)
    cache, state = _containers(case, arch, x["pages"])
    _fill(case, seed, cache, state)
    hidden = {"grouped": _exact_grouped, "latent": _exact_latent, "experts": _exact_experts, "recurrent": _exact_recurrent}[case["family"]](
        case, arch, w, x, cache, state)
    ends = torch.tensor([n for n, _ in x["lens"]]).cumsum(0) - 1
    name = "lm_head.weight" if case["family"] == "grouped" else "head"
    gain, cap = (float(w["final.norm"]), arch.logit_softcap) if case["family"] == "latent" else (1.0, 0.0)
    logits = gain * hidden[ends.to(DEV)] @ w[name].double().T
    out = dict(hidden=hidden, logits=cap * torch.tanh(logits / cap) if cap else logits, cache=None)
    if cache.scales is not None:
        out["scales"] = None
    if state is not None:
        out["state"] = None
    return out


def _rms(x, eps, weight=1.0):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * weight


def _half_turn(x, angle):
    """Pairs (i, i + n / 2) of the last dimension by ``angle [T, n / 2]``; x ``[T, heads, n]``."""
    c, s = angle.cos()[:, None], angle.sin()[:, None]
    u, v = x.chunk(2, -1)
    return torch.cat([u * c - v * s, v * c + u * s], -1)


def _attend(q, k, v, scale, window=1 << 30, keep=0):
    """The last queries of a sequence over all its keys: q ``[t, H, d]``, k, v ``[n, G, d]``."""
    (t, heads, d), (n, groups, _) = q.shape, k.shape
    out, at = torch.empty(t, heads, v.shape[2], dtype=q.dtype, device=q.device), torch.arange(n, device=q.device)
    step = max(1, (1 << 27) // (n * heads))
    for lo in range(0, t, step):
        hi = min(t, lo + step)
        pos = torch.arange(n - t + lo, n - t + hi, device=q.device)[:, None]
        open_ = (at <= pos) & ((pos - at < window) | (at < keep))
        s = torch.einsum("tgsd,ngd->gstn", q[lo:hi].view(hi - lo, groups, -1, d), k) * scale
        p = torch.softmax(s.masked_fill(~open_, -math.inf), -1)
        out[lo:hi] = torch.einsum("gstn,ngd->tgsd", p, v).reshape(hi - lo, heads, -1)
    return out


def _sequences(x):
    """(rows of the step, page numbers and offsets of what is cached before them) of every sequence."""
    at = 0
    for s, (new, total) in enumerate(x["lens"]):
        i = torch.arange(total - new, device=DEV)
        yield slice(at, at + new), x["table"][s, i // PAGE].long(), i % PAGE
        at += new


def _exact_grouped(case, arch, w, x, cache, state):
    t, p = arch.text, "model.language_model."
    heads, groups, dim, eps = t.num_heads, t.num_kv_heads, t.head_dim, t.rms_norm_eps
    axis = torch.tensor([1 if i % 3 == 1 and i < 60 else 2 if i % 3 == 2 and i < 60 else 0 for i in range(dim // 2)], device=DEV)
    rate = t.rope_theta ** (-torch.arange(0, dim, 2, dtype=torch.float64, device=DEV) / dim)
    angle = x["positions"].double()[axis].T * rate
    h = w[p + "embed_tokens.weight"][x["ids"]].double()
    for i in range(LAYERS):
        def m(name):
            return w[f"{p}layers.{i}.{name}.weight"].double()

        n = _rms(h, eps, m("input_layernorm"))
        q, k, v = ((n @ m(f"self_attn.{s}_proj").T).view(-1, c, dim) for s, c in (("q", heads), ("k", groups), ("v", groups)))
        q, k = _half_turn(_rms(q, eps, m("self_attn.q_norm")), angle), _half_turn(_rms(k, eps, m("self_attn.k_norm")), angle)
        a = torch.empty_like(q)
        for rows, page, off in _sequences(x):
            past = [cache.payload[j, i][page, :, off].double() * (1.0 if cache.scales is None else cache.scales[j, i][page, :, off].double()[..., None])
                    for j in (0, 1)]
            a[rows] = _attend(q[rows], torch.cat([past[0], k[rows]]), torch.cat([past[1], v[rows]]), dim ** -0.5)
        h = h + a.flatten(1) @ m("self_attn.o_proj").T
        n = _rms(h, eps, m("post_attention_layernorm"))
        h = h + (torch.nn.functional.silu(n @ m("mlp.gate_proj").T) * (n @ m("mlp.up_proj").T)) @ m("mlp.down_proj").T
    return _rms(h, eps, w[p + "norm.weight"].double())


def _exact_latent(case, arch, w, x, cache, state):
    eps = arch.norm_eps
    h = w["embed"][x["ids"]].double()
    for i, layer in enumerate(arch.layers):
        z = layer.mixer

        def m(name):
            return w[f"l{i}.{name}"].double()

        n1, n2 = _rms(h, eps, m("norm1")), _rms(h, eps, m("norm2"))
        q, c = (n1 @ m("mix.q").T).view(-1, z.heads, z.dim), _rms(n1 @ m("mix.dkv").T, eps, m("mix.dkv.norm"))
        a = torch.empty(len(h), z.heads, z.vdim, dtype=h.dtype, device=DEV)
        for rows, page, off in _sequences(x):
            seen = torch.cat([cache.latent(i)[page, off, :z.kv_rank].double(), c[rows]])
            a[rows] = _attend(q[rows], (seen @ m("mix.uk").T).view(-1, z.heads, z.dim), (seen @ m("mix.uv").T).view(-1, z.heads, z.vdim), z.scale)
        y = (a.flatten(1) * torch.sigmoid(n1 @ m("mix.g").T)) @ m("mix.o").T * torch.sigmoid(n1 @ m("rg1").T + m("rg1.b"))
        f = torch.nn.functional.gelu(n2 @ m("mlp.up").T) @ m("mlp.down").T * torch.sigmoid(n2 @ m("rg2").T + m("rg2.b"))
        h = h + arch.residual_mult * (y + f)
    return _rms(h, eps)


def _experts(n, m, count, chosen, weight):
    """Sum over the chosen experts of every row, times their weights."""
    def unit(rows, p):
        return (torch.nn.functional.silu(rows @ m(p + ".gate").T) * (rows @ m(p + ".up").T)) @ m(p + ".down").T

    y = unit(n, "mlp.shared")
    if weight.shape[1] > chosen.shape[1]:   # the last weight is the shared expert's
        y = y * weight[:, -1:]
    for e in range(count):
        row, slot = (chosen == e).nonzero(as_tuple=True)
        if len(row):
            y[row] += weight[row, slot, None] * unit(n[row], f"mlp.e{e}")
    return y


def _exact_experts(case, arch, w, x, cache, state):
    eps, pos = arch.norm_eps, x["positions"][0].double()
    h = w["embed"][x["ids"]].double()
    for i, layer in enumerate(arch.layers):
        z, moe = layer.mixer, layer.moe

        def m(name):
            return w[f"l{i}.{name}"].double()

        angle = pos[:, None] * z.rot.base ** (-torch.arange(0, z.dim, 2, dtype=torch.float64, device=DEV) / z.dim)
        n = _rms(h, eps, m("norm1"))
        q = _half_turn(_rms(n @ m("mix.q").T, eps, m("mix.q.norm")).view(-1, z.heads, z.dim), angle)
        k = _half_turn(_rms(n @ m("mix.k").T, eps, m("mix.k.norm")).view(-1, z.kv_heads, z.dim), angle)
        v, a = (n @ m("mix.v").T).view(-1, z.kv_heads, z.vdim), torch.empty_like(q)
        for rows, page, off in _sequences(x):
            past = cache.token_rows(i)[page, off].double().view(-1, 2, z.kv_heads, z.dim)
            a[rows] = _attend(q[rows], torch.cat([past[:, 0], k[rows]]), torch.cat([past[:, 1], v[rows]]), z.scale, z.window, z.keep_first)
        a = a * torch.sigmoid(n @ m("mix.g").T)[:, :, None]
        h = h + _rms(a.flatten(1) @ m("mix.o").T, eps, m("norm1b"))
        n = _rms(h, eps, m("norm2"))
        best = (n @ m("mlp.router").T).topk(moe.top, 1)
        h = h + _rms(_experts(n, m, moe.experts, best.indices, torch.softmax(best.values, 1)), eps, m("norm2b"))
        side = torch.nn.functional.gelu(h @ m("side.gate").T, approximate="tanh") * w["side.embed"][x["ids"], i * SIDE:(i + 1) * SIDE].double()
        h = h + _rms(side @ m("side.proj").T, eps, m("side.norm"))
    return _rms(h, eps, w["final.norm"].double())


def _exact_recurrent(case, arch, w, x, cache, state):
    eps, H, width = arch.norm_eps, case["width"] // STATE, case["width"]
    h = w["embed"][x["ids"]].double()
    for i, layer in enumerate(arch.layers):
        moe = layer.moe

        def m(name):
            return w[f"l{i}.{name}"].double()

        o, mixed = torch.empty(len(h), H, STATE, dtype=h.dtype, device=DEV), {}
        old, before = [], h.clone()
        for s, (rows, page, _) in enumerate(_sequences(x)):
            old.append(state.layer(i)[s, len(page) & 1].double() * (len(page) > 0))
            before[rows] = torch.cat([old[-1][None, H * STATE * STATE:], h[rows][:-1]])
        for s in "rkvgw":
            mixed[s] = h + (before - h) * m("mix.mu." + s)
        r, k, v = ((mixed[s] @ m("mix." + s).T).view(-1, H, STATE) for s in "rkv")
        d = torch.exp(-torch.exp(torch.tanh(mixed["w"] @ m("mix.w1").T) @ m("mix.w2").T + m("mix.w0"))).view(-1, H, STATE)
        u = m("mix.u")
        for s, (rows, _, _) in enumerate(_sequences(x)):
            S = old[s][:H * STATE * STATE].view(H, STATE, STATE)
            for t in range(rows.start, rows.stop):
                kv = k[t][:, :, None] * v[t][:, None, :]
                o[t] = torch.bmm(r[t][:, None], S + u[:, :, None] * kv)[:, 0]
                S = d[t][:, :, None] * S + kv
        y = _rms(o, eps).flatten(1) * m("mix.norm") * torch.nn.functional.silu(mixed["g"] @ m("mix.g").T)
        h = h + _rms(y @ m("mix.o").T, eps, 1.0 + m("norm1"))
        score = torch.softmax(h @ m("mlp.router").T, 1)
        choice = score + m("mlp.correction")
        size = moe.outputs // moe.groups
        kept = choice.view(-1, moe.groups, size).amax(2).topk(moe.groups_kept, 1).indices
        open_ = torch.zeros(len(h), moe.groups, dtype=torch.bool, device=DEV).scatter_(1, kept, True).repeat_interleave(size, 1)
        chosen = choice.masked_fill(~open_, -math.inf).topk(moe.top, 1).indices
        weight = score.gather(1, chosen)
        weight = torch.cat([weight / weight.sum(1, keepdim=True) * moe.scale, torch.sigmoid(h @ m("mlp.shared.sg").T)], 1)
        h = h + _rms(_experts(h, m, moe.experts, chosen, weight), eps, 1.0 + m("norm2"))
    return _rms(h, eps, 1.0 + w["final.norm"].double()) * arch.logit_scale


def _exact_vision(case, w, pixels, grid):
    v, p = A.VisionArch(), "model.visual."
    n_side, heads, dim, eps = v.grid_per_side, v.num_heads, v.head_dim, v.layer_norm_eps
    rows, cols, images = case["rows"], case["cols"], case["images"]

    def lin(x, name):
        m = w[p + name + ".weight"].double()
        return x @ m.reshape(m.shape[0], -1).T + w[p + name + ".bias"].double()

    def norm(x, name):
        return torch.nn.functional.layer_norm(x, x.shape[-1:], w[p + name + ".weight"].double(), w[p + name + ".bias"].double(), eps)

    # patches come in 2 x 2 blocks
    grid_rc = torch.stack(torch.meshgrid(torch.arange(rows), torch.arange(cols), indexing="ij"), -1)
    rc = grid_rc.view(rows // 2, 2, cols // 2, 2, 2).permute(0, 2, 1, 3, 4).reshape(-1, 2).to(DEV)
    r, c = (rc[:, j].double() * (n_side - 1) / (k - 1) for j, k in ((0, rows), (1, cols)))
    table = w[p + "pos_embed.weight"].double().view(n_side, n_side, -1)
    r0, c0 = r.floor().long().clamp_max(n_side - 1), c.floor().long().clamp_max(n_side - 1)
    r1, c1, fr, fc = (r0 + 1).clamp_max(n_side - 1), (c0 + 1).clamp_max(n_side - 1), (r - r0)[:, None], (c - c0)[:, None]
    place = (1 - fr) * ((1 - fc) * table[r0, c0] + fc * table[r0, c1]) + fr * ((1 - fc) * table[r1, c0] + fc * table[r1, c1])
    rate = v.rope_theta ** (-torch.arange(0, dim // 2, 2, dtype=torch.float64, device=DEV) / (dim // 2))
    angle = torch.cat([rc[:, :1] * rate, rc[:, 1:] * rate], 1).repeat(images, 1)
    x = lin(pixels.double(), "patch_embed.proj") + place.repeat(images, 1)
    deep = []

    def merge(x, name, late):
        y = norm(x.reshape(-1, v.merged_dim) if late else x, name + ".norm").reshape(-1, v.merged_dim)
        return lin(torch.nn.functional.gelu(lin(y, name + ".linear_fc1")), name + ".linear_fc2")

    for i in range(v.depth):
        b = f"blocks.{i}."
        q, k, val = lin(norm(x, b + "norm1"), b + "attn.qkv").view(-1, 3, heads, dim).unbind(1)
        q, k = _half_turn(q, angle), _half_turn(k, angle)
        q, k, val = (t.reshape(images, -1, heads, dim).transpose(1, 2) for t in (q, k, val))
        a = torch.softmax(q @ k.transpose(2, 3) * dim ** -0.5, -1) @ val
        x = x + lin(a.transpose(1, 2).reshape(len(x), -1), b + "attn.proj")
        x = x + lin(torch.nn.functional.gelu(lin(norm(x, b + "norm2"), b + "mlp.linear_fc1"), approximate="tanh"), b + "mlp.linear_fc2")
        if i in v.deepstack_visual_indexes:
            deep.append(merge(x, f"deepstack_merger_list.{len(deep)}", True))
    return [merge(x, "merger", False), *deep]
