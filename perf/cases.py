"""What this engine is timed on: decode steps, first tokens, whole layers and single mixers and feed-forwards.

A case is a dict of plain values; `prepare` makes what a serving program has in hand (a model with random weights on the
GPU, requests whose earlier tokens are in the cache), `run` does one pass through the package's own entry points, `exact`
gives the same results in 64-bit from plain torch operations.  Sizes are those of the OPT family and of the other
decoders' benchmark configurations (heads of 128 on a quarter as many key/value heads, sixteen experts of half the
width, recurrent states of 128 x 128 a head).

Kinds of cases:
  decode      a whole decode step of OPT through StepRunner.step (a captured graph, as the engine runs it): logits
  prompt      the first token of a short prompt through StepRunner.step (a request comes, runs and goes): logits
  block       one OPT layer over a portion of a prompt, alone or beside other requests' decode tokens: the stream
  attention   an attention mixer with shared key/value heads over decode tokens: what it adds to the stream
  experts     a feed-forward of routed experts
  retention   a retention mixer (fixed decay per head) over portions of prompts: its output and the state it leaves
  delta       a delta-rule mixer over portions of prompts: its output and the state it leaves
"""
import math

import torch

DEV = "cuda:0"
PAGE, LIMIT = 16, 2048                # tokens of a page; the longest context of the family
VOCAB = 50272
STD = 0.02                            # of every random matrix, as the family is initialised
# hidden, heads, inner width of the feed-forward, layers that a case keeps of the model
OPT = {"125m": (768, 12, 3072, 12), "1.3b": (2048, 32, 8192, 6), "2.7b": (2560, 32, 10240, 6),
       "6.7b": (4096, 32, 16384, 4), "13b": (5120, 40, 20480, 2)}
TORCH = {"float16": torch.float16, "bfloat16": torch.bfloat16, "float32": torch.float32}


def listed():
    return [
        # one user's chat on the smallest model: the step is launches and latency
        dict(name="decode_125m_b1", kind="decode", size="125m", dtype="float16", batch=1, context=180),
        # one user on a large model: the weights are streamed for a single token
        dict(name="decode_6.7b_b1", kind="decode", size="6.7b", dtype="float16", batch=1, context=1500),
        # a small serving batch with heads of 80 dims
        dict(name="decode_2.7b_b8", kind="decode", size="2.7b", dtype="bfloat16", batch=8, context=1400),
        # a full serving batch with short, ragged contexts
        dict(name="decode_13b_b64", kind="decode", size="13b", dtype="float16", batch=64, context=400),
        # time to the first token of a chat message
        dict(name="prompt_1.3b_45", kind="prompt", size="1.3b", dtype="bfloat16", tokens=45),
        # a layer of a long prompt
        dict(name="block_6.7b_2048", kind="block", size="6.7b", dtype="float16", portion=2048, past=0, rows=0, context=1),
        # a layer of a served step: a portion of one prompt beside the decode tokens of others
        dict(name="block_13b_mixed", kind="block", size="13b", dtype="float16", portion=481, past=512, rows=31, context=900),
        # the 32-bit engine, on a checkpoint stored in 16 bits
        dict(name="block_1.3b_fp32", kind="block", size="1.3b", dtype="float32", portion=499, past=256, rows=3, context=700),
        # a served batch of decode tokens, four query heads a key/value head
        dict(name="attention_gqa_b48", kind="attention", dtype="bfloat16", width=4096, heads=32, kv_heads=8, batch=48, context=1900),
        # a prompt through routed experts
        dict(name="experts_2048", kind="experts", dtype="bfloat16", width=4096, ff=2048, experts=16, top=4, tokens=2048),
        # a prompt through the recurrent mixers
        dict(name="retention_2048", kind="retention", dtype="bfloat16", width=2048, heads=16, tokens=2048, requests=1),
        dict(name="delta_1536_r3", kind="delta", dtype="bfloat16", width=2048, heads=16, kv_heads=4, tokens=1536, requests=3),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["decode", "decode", "prompt", "block", "block", "attention", "attention", "experts", "retention", "delta"])
    dtype = rng.choice(["float16", "bfloat16"])
    if kind == "decode":
        size = rng.choice(list(OPT))
        return dict(kind=kind, size=size, dtype=dtype, batch=_log(rng, 1, 64), context=rng.choice([1, 2, 4]) * rng.randint(140, 400))
    if kind == "prompt":
        return dict(kind=kind, size=rng.choice(["125m", "1.3b", "2.7b"]), dtype=dtype, tokens=_log(rng, 2, 700))
    if kind == "block":
        if rng.random() < 0.25:
            return dict(kind=kind, size=rng.choice(["125m", "1.3b"]), dtype="float32", portion=_log(rng, 2, 500),
                        past=rng.randint(0, 256), rows=rng.randint(0, 4), context=rng.randint(20, 700))
        size = rng.choice(["1.3b", "2.7b", "6.7b", "13b"])
        portion = _log(rng, 100, 2048 if size != "13b" else 1024)
        return dict(kind=kind, size=size, dtype=dtype, portion=portion, past=rng.choice([0, rng.randint(1, LIMIT - portion)]) if portion < LIMIT else 0,
                    rows=rng.choice([0, rng.randint(1, 32)]), context=rng.randint(20, 900))
    if kind == "attention":
        heads = rng.choice([16, 32])
        return dict(kind=kind, dtype=dtype, width=128 * heads, heads=heads, kv_heads=heads // rng.choice([2, 4, 4, 8, heads]),
                    batch=_log(rng, 2, 64), context=_log(rng, 100, 1900))
    if kind == "experts":
        width = rng.choice([2048, 4096])
        experts, top = rng.choice([(8, 2), (16, 4)])
        return dict(kind=kind, dtype=dtype, width=width, ff=width // 2 + rng.choice([0, 0, 96]), experts=experts, top=top, tokens=_log(rng, 1, 2048))
    requests = rng.randint(1, 4)
    tokens = _log(rng, 64, 2048)
    if kind == "retention":
        return dict(kind=kind, dtype=dtype, width=2048, heads=16, tokens=tokens, requests=min(requests, tokens // 32))
    return dict(kind=kind, dtype=dtype, width=2048, heads=16, kv_heads=rng.choice([4, 8, 16]), tokens=tokens, requests=min(requests, tokens // 32))


# ---- inputs, made from the seed alone --------------------------------------------------------------------
def _generator(seed, stream=0):
    return torch.Generator(device=DEV).manual_seed(1000003 * int(seed) + stream)


def _normal(g, *shape, dtype=torch.float32, std=1.0, mean=0.0):
    return (torch.randn(shape, generator=g, device=DEV) * std + mean).to(dtype)


def _lengths(case, seed, n, most):
    """n ragged lengths between half of `most` and `most`; the first is `most` itself."""
    g = torch.Generator().manual_seed(int(seed) + 77)
    return [most] + torch.randint(max(1, most // 2), most + 1, (n,), generator=g).tolist()[1:] if n else []


def _stored(case):
    return torch.float16 if case["dtype"] == "float32" else TORCH[case["dtype"]]


def _opt_weights(case, seed, layers, vocab):
    H, _, F, _ = OPT[case["size"]]
    g, t = _generator(seed, 1), _stored(case)
    d = "model.decoder."
    w = {d + "embed_tokens.weight": _normal(g, vocab, H, dtype=t, std=STD), d + "embed_positions.weight": _normal(g, LIMIT + 2, H, dtype=t, std=STD)}

    def norm(p):
        w[p + ".weight"], w[p + ".bias"] = _normal(g, H, dtype=t, std=STD, mean=1.0), _normal(g, H, dtype=t, std=STD)

    for i in range(layers):
        p = f"{d}layers.{i}."
        for name, o, n in (("self_attn.q_proj", H, H), ("self_attn.k_proj", H, H), ("self_attn.v_proj", H, H), ("self_attn.out_proj", H, H),
                           ("fc1", F, H), ("fc2", H, F)):
            w[p + name + ".weight"], w[p + name + ".bias"] = _normal(g, o, n, dtype=t, std=STD), _normal(g, o, dtype=t, std=STD)
        norm(p + "self_attn_layer_norm")
        norm(p + "final_layer_norm")
    norm(d + "final_layer_norm")
    w["lm_head.weight"] = w[d + "embed_tokens.weight"]
    return w


def _opt_model(case, weights, layers, vocab):
    from transformers_neuronx_b200.config import OPTConfig
    from transformers_neuronx_b200.engine import build_model
    from transformers_neuronx_b200.models import opt
    H, heads, F, _ = OPT[case["size"]]
    cfg = OPTConfig.from_dict(dict(vocab_size=vocab, hidden_size=H, num_hidden_layers=layers, num_attention_heads=heads, ffn_dim=F,
                                   max_position_embeddings=LIMIT, word_embed_proj_dim=H, do_layer_norm_before=True, enable_bias=True,
                                   layer_norm_elementwise_affine=True, activation_function="relu", init_std=STD,
                                   architectures=["OPTForCausalLM"], model_type="opt"))
    return build_model(opt.build_spec(cfg), weights, case["dtype"], DEV, verbose=False)


def _part_model(width, weights, dtype, mixer, feed_forward=None):
    """A model of one layer around the part that is timed, with a small embedding; the part is called by itself."""
    from transformers_neuronx_b200.engine import build_model
    from transformers_neuronx_b200.parts.spec import EmbeddingSpec, HeadSpec, LayerSpec, ModelSpec, NormSpec, ScheduleEntry
    weights["embed"] = torch.zeros(64, width, dtype=TORCH[dtype], device=DEV)
    layer = LayerSpec(block="post_norm_scaled", norm1=NormSpec("rms_norm", width, 1e-5), mixer=mixer,
                      norm2=NormSpec("rms_norm", width, 1e-5) if feed_forward is not None else None, feed_forward=feed_forward)
    spec = ModelSpec(hidden_size=width, vocab_size=64, max_positions=LIMIT, embedding=EmbeddingSpec("embed", 64, width), layers=(layer,),
                     schedule=(ScheduleEntry(0, 0),), head=HeadSpec(weight="embed", vocab=64, dim=width))
    return build_model(spec, weights, dtype, DEV, verbose=False)


def _pages(lengths):
    return sum(-(-n // PAGE) + 1 for n in lengths)


class _State:
    pass


# ---- decode, prompt --------------------------------------------------------------------------------------
WARM = 2                              # decode steps before the timed ones: the second is where the graph is captured


def _decode_tokens(case, seed):
    lengths = _lengths(case, seed, case["batch"], case["context"])
    g = torch.Generator().manual_seed(int(seed))
    return [torch.randint(3, VOCAB, (n + WARM + 1,), generator=g).tolist() for n in lengths]


def _prepare_decode(case, seed):
    from transformers_neuronx_b200.engine import StepEntry, StepRunner
    s = _State()
    layers = OPT[case["size"]][3]
    model = _opt_model(case, _opt_weights(case, seed, layers, VOCAB), layers, VOCAB)
    toks = _decode_tokens(case, seed)
    s.starts = [len(t) - 1 for t in toks]
    top = 256                         # contexts stay in the range of one captured graph; at its end other requests take over
    while top < max(s.starts) + 1:
        top *= 2
    s.steps_left = s.steps = min(top, LIMIT) - max(s.starts)
    s.runner = StepRunner(model, PAGE, _pages([n + s.steps for n in s.starts]), case["batch"], LIMIT, use_cuda_graphs=True)
    for b, t in enumerate(toks):
        s.runner.add_request(b)
        s.runner.step([StepEntry(b, t[:-WARM - 1], [])])
    for i in range(WARM):
        s.runner.step([StepEntry(b, [t[i - WARM - 1]], [0]) for b, t in enumerate(toks)])
    s.entries = [StepEntry(b, [t[-1]], [0]) for b, t in enumerate(toks)]
    return s


def _run_decode(s):
    if s.steps_left == 0:             # these requests have ended; others of the same lengths go on in their pages
        for b in range(len(s.starts)):
            s.runner.finish(b)
        for b, n in enumerate(s.starts):
            s.runner.add_request(b)
            s.runner.cache.append(b, n)
        s.steps_left = s.steps
    s.steps_left -= 1
    return s.runner.step(s.entries)


def _prepare_prompt(case, seed):
    from transformers_neuronx_b200.engine import StepEntry, StepRunner
    s = _State()
    layers = OPT[case["size"]][3]
    model = _opt_model(case, _opt_weights(case, seed, layers, VOCAB), layers, VOCAB)
    s.runner = StepRunner(model, PAGE, _pages([case["tokens"]]), 1, LIMIT, use_cuda_graphs=True)
    s.entry = StepEntry("p", _prompt_tokens(case, seed), [case["tokens"] - 1])
    for _ in range(WARM):
        _run_prompt(s)
    return s


def _prompt_tokens(case, seed):
    return torch.randint(3, VOCAB, (case["tokens"],), generator=torch.Generator().manual_seed(int(seed))).tolist()


def _run_prompt(s):
    s.runner.add_request("p")
    logits = s.runner.step([s.entry])
    s.runner.finish("p")
    return logits


# ---- plain 64-bit OPT ------------------------------------------------------------------------------------
def _layer_norm(x, w, p):
    x = x - x.mean(-1, keepdim=True)
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + 1e-5) * w[p + ".weight"] + w[p + ".bias"]


def _linear(x, w, p):
    return x @ w[p + ".weight"].T + w[p + ".bias"]


def _causal_attention(q, k, v, scale):
    """q [heads, T, d] is the last T of the S tokens of k, v [heads, S, d]."""
    T, S = q.shape[1], k.shape[1]
    ok = torch.arange(S, device=DEV)[None, :] <= torch.arange(S - T, S, device=DEV)[:, None]
    return torch.cat([torch.softmax((q[h] @ k[h].T * scale).masked_fill(~ok, -math.inf), -1)[None] @ v[h] for h in range(q.shape[0])])


def _heads(x, n):
    return x.reshape(x.shape[0], n, -1).transpose(0, 1)


def _opt_layer(x, last, w, p, heads):
    """The last `last` rows of a layer over the rows x of one request."""
    h = _layer_norm(x, w, p + "self_attn_layer_norm")
    q = _heads(_linear(h[-last:], w, p + "self_attn.q_proj"), heads)
    k, v = _heads(_linear(h, w, p + "self_attn.k_proj"), heads), _heads(_linear(h, w, p + "self_attn.v_proj"), heads)
    a = _causal_attention(q, k, v, q.shape[2] ** -0.5).transpose(0, 1).reshape(last, -1)
    x = x[-last:] + _linear(a, w, p + "self_attn.out_proj")
    h = torch.relu(_linear(_layer_norm(x, w, p + "final_layer_norm"), w, p + "fc1"))
    return x + _linear(h, w, p + "fc2")


def _exact_logits(case, seed, sequences):
    _, heads, _, layers = OPT[case["size"]]
    w = {k: v.double() for k, v in _opt_weights(case, seed, layers, VOCAB).items()}
    d, rows = "model.decoder.", []
    for ids in sequences:
        n = len(ids)
        x = w[d + "embed_tokens.weight"][torch.tensor(ids, device=DEV)] + w[d + "embed_positions.weight"][2:n + 2]
        for i in range(layers):
            x = _opt_layer(x, n if i + 1 < layers else 1, w, f"{d}layers.{i}.", heads)
        rows.append(_layer_norm(x, w, d + "final_layer_norm") @ w["lm_head.weight"].T)
    return torch.cat(rows)


# ---- block -----------------------------------------------------------------------------------------------
def _block_streams(case, seed):
    """Per request (rows of the 32-bit stream so far, how many of them are this step's)."""
    H = OPT[case["size"]][0]
    g = _generator(seed, 2)
    out = [(_normal(g, case["past"] + case["portion"], H), case["portion"])]
    return out + [(_normal(g, n, H), 1) for n in _lengths(case, seed, case["rows"], case["context"])]


def _prepare_block(case, seed):
    from transformers_neuronx_b200.engine import StepEntry, StepRunner
    s = _State()
    model = _opt_model(case, _opt_weights(case, seed, 1, 512), 1, 512)
    s.block = model.blocks[0]
    streams = _block_streams(case, seed)
    runner = StepRunner(model, PAGE, _pages([x.shape[0] for x, _ in streams]), len(streams), LIMIT)
    for r, (x, last) in enumerate(streams):
        runner.add_request(r)
        if x.shape[0] > last:         # the earlier tokens' keys and values, as an earlier step leaves them
            past = x[:-last]
            ctx = runner.prepare([StepEntry(r, [3] * past.shape[0], [])])
            ctx.cache_id = 0
            h = ctx.empty(*past.shape)
            s.block.norm1.forward(ctx, past.contiguous(), out_act=h)
            s.block.mixer.forward(ctx, h, torch.zeros_like(past))
    s.x0 = torch.cat([x[-last:] for x, last in streams])
    s.x = torch.empty_like(s.x0)
    s.ctx = runner.prepare([StepEntry(r, [3] * last, []) for r, (x, last) in enumerate(streams)])
    s.ctx.cache_id = s.ctx.entry_index = 0
    s.runner = runner
    return s


def _run_block(s):
    s.x.copy_(s.x0)                   # a layer changes the stream in place
    s.ctx.begin_entry()
    s.block.forward(s.ctx, s.x, None)
    return s.x


def _exact_block(case, seed):
    w = {k: v.double() for k, v in _opt_weights(case, seed, 1, 512).items()}
    return torch.cat([_opt_layer(x.double(), last, w, "model.decoder.layers.0.", OPT[case["size"]][1]) for x, last in _block_streams(case, seed)])


# ---- mixers and feed-forwards alone ----------------------------------------------------------------------
def _matrices(case, seed, shapes):
    g = _generator(seed, 3)
    return {k: _normal(g, *shape, dtype=TORCH[case["dtype"]], std=STD) for k, shape in shapes.items()}


def _attention_weights(case, seed):
    W, G = case["width"], case["kv_heads"]
    return _matrices(case, seed, {"q": (W, W), "k": (G * 128, W), "v": (G * 128, W), "o": (W, W)})


def _attention_inputs(case, seed):
    """The normalised rows of every request, its decode token's last."""
    g = _generator(seed, 4)
    return [_normal(g, n, case["width"], dtype=TORCH[case["dtype"]]) for n in _lengths(case, seed, case["batch"], case["context"])]


def _prepare_attention(case, seed):
    from transformers_neuronx_b200.engine import StepEntry, StepRunner
    from transformers_neuronx_b200.parts.spec import AttentionSpec, LinearSpec
    s = _State()
    W, G = case["width"], case["kv_heads"]
    spec = AttentionSpec(kind="attention", hidden=W, n_heads=case["heads"], n_kv_heads=G, head_dim=128, scale=128 ** -0.5, q=LinearSpec(W, W, "q"),
                         k=LinearSpec(W, G * 128, "k"), v=LinearSpec(W, G * 128, "v"), out=LinearSpec(W, W, "o"))
    model = _part_model(W, _attention_weights(case, seed), case["dtype"], spec)
    s.part = model.blocks[0].mixer
    rows = _attention_inputs(case, seed)
    s.runner = StepRunner(model, PAGE, _pages([len(h) for h in rows]), len(rows), LIMIT)
    for r, h in enumerate(rows):
        s.runner.add_request(r)
        if len(h) > 1:
            ctx = s.runner.prepare([StepEntry(r, [3] * (len(h) - 1), [])])
            ctx.cache_id = 0
            s.part.forward(ctx, h[:-1], torch.zeros(len(h) - 1, W, device=DEV))
    return _ready(s, torch.stack([h[-1] for h in rows]), [StepEntry(r, [3], []) for r in range(len(rows))], seed)


def _stream(seed, shape):
    """What the part adds its result to, of about the result's size."""
    return _normal(_generator(seed, 5), *shape, std=0.1)


def _ready(s, h, entries, seed):
    s.h = h
    s.stream = _stream(seed, h.shape)
    s.out = torch.empty_like(s.stream)
    s.ctx = s.runner.prepare(entries)
    s.ctx.cache_id = s.ctx.entry_index = 0
    return s


def _run_part(s):
    s.out.copy_(s.stream)             # the part adds to the stream in place
    s.ctx.begin_entry()
    s.part.forward(s.ctx, s.h, s.out)
    return s.out


def _exact_attention(case, seed):
    w = {k: v.double() for k, v in _attention_weights(case, seed).items()}
    rows = []
    for h in _attention_inputs(case, seed):
        h = h.double()
        q, k, v = _heads(h[-1:] @ w["q"].T, case["heads"]), _heads(h @ w["k"].T, case["kv_heads"]), _heads(h @ w["v"].T, case["kv_heads"])
        k, v = (t.repeat_interleave(case["heads"] // case["kv_heads"], 0) for t in (k, v))
        rows.append(_causal_attention(q, k, v, 128 ** -0.5).reshape(1, -1) @ w["o"].T)
    return torch.cat(rows) + _stream(seed, (case["batch"], case["width"])).double()


def _expert_weights(case, seed):
    W, F = case["width"], case["ff"]
    shapes = {"router": (case["experts"], W), "q": (16, W), "k": (16, W), "v": (16, W), "o": (W, 16)}
    for e in range(case["experts"]):
        shapes.update({f"{e}.gate": (F, W), f"{e}.up": (F, W), f"{e}.down": (W, F)})
    return _matrices(case, seed, shapes)


def _inputs(case, seed):
    return _normal(_generator(seed, 4), case["tokens"], case["width"], dtype=TORCH[case["dtype"]])


def _prepare_experts(case, seed):
    from transformers_neuronx_b200.engine import StepEntry, StepRunner
    from transformers_neuronx_b200.parts.spec import AttentionSpec, ExpertSpec, LinearSpec, RoutedFeedForwardSpec
    s = _State()
    W, F, N = case["width"], case["ff"], case["tokens"]
    small = AttentionSpec(kind="attention", hidden=W, n_heads=1, n_kv_heads=1, head_dim=16, scale=0.25, q=LinearSpec(W, 16, "q"),
                          k=LinearSpec(W, 16, "k"), v=LinearSpec(W, 16, "v"), out=LinearSpec(16, W, "o"))
    spec = RoutedFeedForwardSpec(kind="routed_experts", hidden=W, ff=F, n_experts=case["experts"], top=case["top"], router="router",
                                 experts=tuple(ExpertSpec(f"{e}.gate", f"{e}.up", f"{e}.down") for e in range(case["experts"])),
                                 scores="softmax", weight_on_input=False, act_alpha=1.0, up_shift=0.0)
    model = _part_model(W, _expert_weights(case, seed), case["dtype"], small, spec)
    s.part = model.blocks[0].feed_forward
    few = N <= 32                     # few tokens: a decode step; many: a prompt
    lengths = [1] * N if few else [N]
    s.runner = StepRunner(model, PAGE, _pages(lengths), len(lengths), LIMIT)
    for r in range(len(lengths)):
        s.runner.add_request(r)
    return _ready(s, _inputs(case, seed), [StepEntry(r, [3] * n, []) for r, n in enumerate(lengths)], seed)


def _exact_experts(case, seed):
    w = {k: v.double() for k, v in _expert_weights(case, seed).items()}
    h = _inputs(case, seed).double()
    p = torch.softmax(h @ w["router"].T, -1)
    weight, chosen = p.topk(case["top"], -1)
    y = _stream(seed, h.shape).double()
    for e in range(case["experts"]):
        token, place = (chosen == e).nonzero(as_tuple=True)
        g = h[token] @ w[f"{e}.gate"].T
        z = (g * torch.sigmoid(g) * (h[token] @ w[f"{e}.up"].T)) @ w[f"{e}.down"].T
        y.index_add_(0, token, z * weight[token, place][:, None])
    return y


def _portions(case):
    """The tokens of the requests: ragged, together case["tokens"]."""
    R, N = case["requests"], case["tokens"]
    cut = [N * i // R + (7 * i if i < R else 0) for i in range(R + 1)]
    return [b - a for a, b in zip(cut, cut[1:])]


def _prepare_recurrent(case, seed, spec, weights):
    from transformers_neuronx_b200.engine import StepEntry, StepRunner
    s = _State()
    model = _part_model(case["width"], weights, case["dtype"], spec)
    s.part = model.blocks[0].mixer
    lengths = _portions(case)
    s.runner = StepRunner(model, PAGE, 1, len(lengths), LIMIT)
    s.slots = [s.runner.add_request(r) for r in range(len(lengths))]
    _ready(s, _inputs(case, seed), [StepEntry(r, [3] * n, []) for r, n in enumerate(lengths)], seed)
    s.state = s.ctx.cache(0 if case["kind"] == "delta" else None)
    return s


def _run_recurrent(s):
    for slot in s.slots:              # what admitting a request does: its state starts at zero
        s.runner.storage.clear_slot(slot)
    return _run_part(s), s.state


def _decays(case):
    return tuple(1.0 - 2.0 ** (-5 - 7 * h / case["heads"]) for h in range(case["heads"]))


def _retention_weights(case, seed):
    W = case["width"]
    return _matrices(case, seed, {k: (W, W) for k in ("q", "k", "v", "gate", "o")})


def _prepare_retention(case, seed):
    from transformers_neuronx_b200.parts.spec import LinearSpec, RetentionSpec, RotarySpec
    W = case["width"]
    lin = {k: LinearSpec(W, W, "o" if k == "out" else k) for k in ("q", "k", "v", "gate", "out")}
    spec = RetentionSpec(kind="retention", hidden=W, n_heads=case["heads"], k_dim=128, v_dim=128, decay=_decays(case),
                         rotary=RotarySpec(128, 10000.0), k_scale=128 ** -0.5, **lin)
    return _prepare_recurrent(case, seed, spec, _retention_weights(case, seed))


def _turn(x):
    """x [T, heads, 128]: dim i turns with dim i + 64 by position * 10000^(-i / 64); frequency and angle are 32-bit numbers."""
    freq = (10000.0 ** (-torch.arange(64, dtype=torch.float64, device=DEV) / 64)).float()
    angle = (torch.arange(x.shape[0], device=DEV).float()[:, None] * freq).double()[:, None, :]
    a, b = x[..., :64], x[..., 64:]
    return torch.cat([a * angle.cos() - b * angle.sin(), b * angle.cos() + a * angle.sin()], -1)


def _rms(x, eps=1e-6):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _exact_retention(case, seed):
    w = {k: v.double() for k, v in _retention_weights(case, seed).items()}
    H, rows, states = case["heads"], [], []
    log_decay = torch.tensor(_decays(case), dtype=torch.float64).float().double().log().to(DEV)
    for h in _inputs(case, seed).double().split(_portions(case)):
        T = h.shape[0]
        q, k = (_turn((h @ w[n].T).reshape(T, H, 128)).transpose(0, 1) for n in ("q", "k"))
        k, v = k * 128 ** -0.5, _heads(h @ w["v"].T, H)
        ago = torch.arange(T, device=DEV)[:, None] - torch.arange(T, device=DEV)[None, :]
        o = torch.cat([((q[i] @ k[i].T) * torch.where(ago >= 0, torch.exp(ago.clamp(min=0) * log_decay[i]), 0.0))[None] @ v[i] for i in range(H)])
        left = torch.exp(log_decay[:, None] * torch.arange(T - 1, -1, -1, device=DEV))
        states.append((v * left[..., None]).transpose(1, 2) @ k)                     # [heads, v_dim, k_dim]
        gate = h @ w["gate"].T
        rows.append((_rms(o).transpose(0, 1).reshape(T, -1) * gate * torch.sigmoid(gate)) @ w["o"].T)
    y = torch.cat(rows)
    return y + _stream(seed, y.shape).double(), torch.stack(states)


RANK, TAPS = 64, 4                    # of the delta rule's low-rank decays and gates; of its convolution


def _delta_weights(case, seed):
    W, H, G = case["width"], case["heads"], case["kv_heads"]
    w = _matrices(case, seed, {"q": (G * 128, W), "k": (G * 128, W), "v": (H * 128, W), "b": (H, W), "a1": (RANK, W), "a2": (H * 128, RANK),
                               "g1": (RANK, W), "g2": (H * 128, RANK), "o": (W, H * 128), "norm": (128,)})
    g = _generator(seed, 6)
    t = TORCH[case["dtype"]]
    for n, ch in (("q", G), ("k", G), ("v", H)):
        w[n + ".conv"] = _normal(g, ch * 128, TAPS, dtype=t, std=0.5)
    w["norm"] = w["norm"] + 1.0
    w["A_log"] = _normal(g, H, dtype=t, std=0.5, mean=-3.0)         # decays around 0.97 a token
    w["dt_bias"] = _normal(g, H * 128, dtype=t, std=0.5)
    return w


def _prepare_delta(case, seed):
    from transformers_neuronx_b200.parts.spec import DeltaRuleSpec, LinearSpec
    W, H, G = case["width"], case["heads"], case["kv_heads"]
    lin = lambda n_in, n_out, name: LinearSpec(n_in, n_out, name)
    spec = DeltaRuleSpec(kind="delta_rule", hidden=W, n_heads=H, n_kv_heads=G, k_dim=128, v_dim=128, conv_taps=TAPS, q=lin(W, G * 128, "q"),
                         k=lin(W, G * 128, "k"), v=lin(W, H * 128, "v"), beta=lin(W, H, "b"), a1=lin(W, RANK, "a1"), a2=lin(RANK, H * 128, "a2"),
                         g1=lin(W, RANK, "g1"), g2=lin(RANK, H * 128, "g2"), out=lin(H * 128, W, "o"), q_conv="q.conv", k_conv="k.conv",
                         v_conv="v.conv", a_log="A_log", dt_bias="dt_bias", out_norm="norm", norm_eps=1e-5, q_scale=128 ** -0.5)
    return _prepare_recurrent(case, seed, spec, _delta_weights(case, seed))


def _exact_delta(case, seed):
    w = {k: v.double() for k, v in _delta_weights(case, seed).items()}
    H, G, rows, states = case["heads"], case["kv_heads"], [], []

    def conv(u, c):
        past = torch.cat([torch.zeros(TAPS - 1, u.shape[1], dtype=u.dtype, device=DEV), u])
        y = sum(c[:, j] * past[j:j + u.shape[0]] for j in range(TAPS))
        return y * torch.sigmoid(y)

    for h in _inputs(case, seed).double().split(_portions(case)):
        T = h.shape[0]
        q, k, v = (conv(h @ w[n].T, w[n + ".conv"]).reshape(T, -1, 128) for n in ("q", "k", "v"))
        q, k = (t / torch.sqrt((t * t).sum(-1, keepdim=True) + 1e-6) for t in (q, k))
        q, k = (t.repeat_interleave(H // G, 1) for t in (q * 128 ** -0.5, k))
        beta = torch.sigmoid(h @ w["b"].T)
        step = torch.nn.functional.softplus((h @ w["a1"].T) @ w["a2"].T + w["dt_bias"]).reshape(T, H, 128)
        decay = torch.exp(-torch.exp(w["A_log"])[None, :, None] * step)
        S, o = torch.zeros(H, 128, 128, dtype=torch.float64, device=DEV), []         # [heads, v_dim, k_dim]
        for i in range(T):
            S = S * decay[i][:, None, :]
            u = beta[i][:, None] * (v[i] - (S @ k[i][..., None])[..., 0])
            S = S + u[..., None] * k[i][:, None, :]
            o.append((S @ q[i][..., None])[..., 0])
        gate = torch.sigmoid((h @ w["g1"].T) @ w["g2"].T).reshape(T, H, 128)
        rows.append((_rms(torch.stack(o), 1e-5) * w["norm"] * gate).reshape(T, -1) @ w["o"].T)
        states.append(S)
    y = torch.cat(rows)
    return y + _stream(seed, y.shape).double(), torch.stack(states)


# ---- the interface ---------------------------------------------------------------------------------------
_PREPARE = {"decode": _prepare_decode, "prompt": _prepare_prompt, "block": _prepare_block, "attention": _prepare_attention,
            "experts": _prepare_experts, "retention": _prepare_retention, "delta": _prepare_delta}
_RUN = {"decode": _run_decode, "prompt": _run_prompt, "block": _run_block, "attention": _run_part, "experts": _run_part,
        "retention": _run_recurrent, "delta": _run_recurrent}


def prepare(case, seed):
    state = _PREPARE[case["kind"]](case, seed)
    state.kind = case["kind"]
    return state


def run(state):
    return _RUN[state.kind](state)


def exact(case, seed):
    kind = case["kind"]
    if kind == "decode":
        return _exact_logits(case, seed, _decode_tokens(case, seed))
    if kind == "prompt":
        return _exact_logits(case, seed, [_prompt_tokens(case, seed)])
    return {"block": _exact_block, "attention": _exact_attention, "experts": _exact_experts, "retention": _exact_retention,
            "delta": _exact_delta}[kind](case, seed)


def work(case):
    """Every weight once (of experts those that are expected to be chosen), the live keys and values once, inputs and
    outputs once; two operations a multiply-add."""
    kind, e = case["kind"], 4 if case["dtype"] == "float32" else 2
    if kind in ("decode", "prompt", "block"):
        H, _, F, L = OPT[case["size"]]
        L = 1 if kind == "block" else L
        per_layer = 4 * H * H + 2 * H * F
        if kind == "decode":
            N, mean = case["batch"], int(0.75 * case["context"]) + 1
            keys, pairs = N * mean, N * mean
        else:
            T, past = (case["tokens"], 0) if kind == "prompt" else (case["portion"], case["past"])
            n = 0 if kind == "prompt" else case["rows"]
            others = int(0.75 * n * case["context"]) if n else 0
            N, keys = T + n, T + past + others
            pairs = T * past + T * (T + 1) // 2 + others
        weights = per_layer * L * 2                                                 # stored in 16 bits also in the 32-bit engine
        flops = 2 * N * per_layer * L + 4 * pairs * H * L
        nbytes = weights + keys * 2 * H * e * L
        if kind == "block":
            return {"bytes": nbytes + N * H * 8, "flops": flops}
        out = case["batch"] if kind == "decode" else 1
        return {"bytes": nbytes + VOCAB * H * 2 + out * VOCAB * 4 + N * H * 4, "flops": flops + 2 * out * VOCAB * H}
    W = case["width"]
    if kind == "attention":
        N, G = case["batch"], case["kv_heads"] * 128
        keys = int(0.75 * case["context"] * N)
        mats = 2 * W * W + 2 * W * G
        return {"bytes": mats * 2 + keys * 2 * G * 2 + N * W * 10, "flops": 2 * N * mats + 4 * keys * W}
    N = case["tokens"]
    if kind == "experts":
        used = case["experts"] * (1.0 - (1.0 - case["top"] / case["experts"]) ** N)
        per = 3 * W * case["ff"]
        return {"bytes": used * per * 2 + N * W * 10, "flops": 2.0 * N * case["top"] * per + 2 * N * W * case["experts"]}
    H = case["heads"]
    state = case["requests"] * H * 128 * 128
    G = H if kind == "retention" else case["kv_heads"]
    mats = W * 128 * (2 * G + (2 if kind == "retention" else 1) * H) + 128 * H * W
    per_token = (4 if kind == "retention" else 6) * 128 * 128 * H                  # the state's update and its product with q
    if kind == "delta":
        mats += W * (2 * RANK + H) + 2 * RANK * 128 * H
    return {"bytes": mats * 2 + state * 4 + N * W * 10, "flops": 2.0 * N * mats + N * per_token}


def tolerance(case):
    """About four times the error against `exact` that was measured (a few roundings to the activation type per result;
    whole models pass a layer's rounding on to the next), and for single values twenty times that."""
    if case["dtype"] == "float32":
        return {"rel": 5e-6, "max": 1e-4}
    rel = (3e-3 if case["kind"] in ("decode", "prompt") else 1.6e-3) * (1.0 if case["dtype"] == "float16" else 7.0)
    return {"rel": rel, "max": 20 * rel}
