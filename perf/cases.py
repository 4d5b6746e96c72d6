"""What this framework is used for, as cases whose speed and results can be measured.

Seven kinds of work, each through the call that a program makes:

``token``     one new token of every sequence against a bf16 cache, with the summed attention weights that
              score-based caches keep (``ops.decode_attention``)
``chunk``     a chunk of new tokens against a cache, with the summed weights (``ops.sdpa_fwd``): a step of a chunked
              prompt or of the forward half of training
``gradient``  the backward half of such a chunk, added to the gradients of the cache (``ops.sdpa_bwd``)
``lora``      loss and LoRA gradients of a long sequence through an H2O cache (``LongContextGradientModel``)
``prompt``    a batch of long prompts through a quantized H2O cache to the logits of their last tokens
              (``LongContextInferenceModel``)
``next``      one captured decode step of a batch whose quantized H2O caches are full (``Decoder``)
``layered``   prompts of a model that is described layer by layer (``LongContextInferenceModel``)

Whole models are cut to a few of their layers: every layer does the same work. Weights are random, tokens uniform over the
vocabulary, queries, keys and values normal, as in ``bench.py`` and ``keys_values_b200/tools``. Slots of a cache that evicts
hold its tokens in no order, and a chunk's own tokens lie scattered among them.
"""
import math

import torch

D = 128  # head size of the models below


def listed():
    return [
        # A short conversation with one user: launches and latency count.
        dict(name="token_1x4096", kind="token", batch=1, heads=32, groups=8, slots=4096),
        # Four long contexts: the cache's bytes count.
        dict(name="token_4x32768", kind="token", batch=4, heads=32, groups=8, slots=32768),
        # A short chunk against a short cache, the least that chunked prompt processing does at a time.
        dict(name="chunk_256x4096", kind="chunk", batch=1, heads=32, groups=8, new=256, slots=4096, scattered=False),
        # One layer and chunk of the flagship fine-tuning run (Qwen3-4B heads, evicting cache of 16384 slots).
        dict(name="chunk_1024x16384", kind="chunk", batch=1, heads=32, groups=8, new=1024, slots=16384, scattered=True),
        # The largest cell of the attention benchmark: a batch of prompts at a long context.
        dict(name="chunk_4x2048x32768", kind="chunk", batch=4, heads=32, groups=8, new=2048, slots=32768, scattered=False),
        # The last, shorter chunk of prompts of any length, with Qwen3-14B heads (five to a group).
        dict(name="chunk_ragged_g5", kind="chunk", batch=2, heads=40, groups=8, new=499, slots=7919, scattered=True),
        # Backward half of the flagship's layer and chunk.
        dict(name="gradient_1024x16384", kind="gradient", batch=1, heads=32, groups=8, new=1024, slots=16384, scattered=True),
        # The last chunk of a fine-tuning sequence, Qwen3-14B heads and chunk size, smaller cache.
        dict(name="gradient_ragged_g5", kind="gradient", batch=1, heads=40, groups=8, new=421, slots=8192, scattered=True),
        # The flagship step on two of its layers and a quarter of its sequence.
        dict(name="lora_32768", kind="lora", model="Qwen3-4B", layers=2, batch=1, tokens=32768, targets=1024, slots=16384, chunk=1024, bits=8),
        # Prompts of the inference benchmark, four layers and a quarter of the length.
        dict(name="prompt_4x16384", kind="prompt", model="Llama-3-8B", layers=4, batch=4, tokens=16384, slots=8192, chunk=2048, bits=4),
        # Its decode step, eight layers.
        dict(name="next_4x8192", kind="next", model="Llama-3-8B", layers=8, batch=4, slots=8192, chunk=2048, bits=4),
        # Prompts of a layered model: state-space and attention layers.
        dict(name="layered_2x8192", kind="layered", model="Pazenex-2k", batch=2, tokens=8192),
    ]


# (query heads, key / value heads) of Qwen3-4B and Llama-3-8B, Qwen3-14B, Qwen3-1.7B, Qwen2.5-7B
HEADS = ((32, 8), (40, 8), (16, 8), (28, 4))


def _size(rng, low, high):
    """A size between the two, spread over its logarithm; two of three are odd, one is a multiple of 128 where there is one."""
    n = int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))
    if rng.random() < 1 / 3:
        return min(max(n // 128 * 128, -(-low // 128) * 128), high)
    return min(n | 1, high)


def draw(rng):
    kind = rng.choice(("token", "token", "chunk", "chunk", "chunk", "gradient", "gradient", "lora", "prompt", "next", "layered"))
    heads, groups = rng.choice(HEADS)
    if kind == "token":
        # the longest contexts of a batch of one, fewer slots for larger batches
        batch = rng.choice((1, 1, 2, 4, 8))
        return dict(kind=kind, batch=batch, heads=heads, groups=groups, slots=_size(rng, 1024, 131072 // max(batch, 4)))
    if kind in ("chunk", "gradient"):
        batch = rng.choice((1, 1, 2, 4))
        new, slots = _size(rng, 128, 2048), _size(rng, 4096, 32768 if kind == "chunk" else 16384)
        return dict(kind=kind, batch=batch, heads=heads, groups=groups, new=new, slots=slots, scattered=rng.random() < 0.6)
    if kind == "lora":
        slots = rng.choice((4096, 8192, 16384))
        return dict(kind=kind, model="Qwen3-4B", layers=2, batch=1, tokens=_size(rng, slots + 1024, 32768), targets=1024, slots=slots,
                    chunk=rng.choice((512, 1024)), bits=rng.choice((4, 8)))
    if kind == "prompt":
        slots = rng.choice((4096, 8192))
        return dict(kind=kind, model="Llama-3-8B", layers=4, batch=rng.choice((1, 2, 4)), tokens=_size(rng, slots + 512, 16384), slots=slots,
                    chunk=rng.choice((1024, 2048)), bits=rng.choice((4, 8)))
    if kind == "next":
        return dict(kind=kind, model="Llama-3-8B", layers=8, batch=rng.choice((1, 2, 4, 8)), slots=_size(rng, 2048, 16384) // 64 * 64, chunk=1024,
                    bits=rng.choice((4, 8)))
    return dict(kind=kind, model=rng.choice(("Pazenex-2k", "Ladadra-2k", "Dotorax-2k")), batch=rng.choice((1, 2)), tokens=_size(rng, 1024, 8192))


# ------------------------------------------------------------------------------------------------ inputs
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _normal(shape, g, dtype=torch.bfloat16):
    return torch.randn(shape, generator=g, device="cuda", dtype=torch.float32).to(dtype)


def _ids(shape, vocab, g):
    return torch.randint(0, vocab, shape, generator=g, device="cuda")


def _positions(case, g):
    """``(token_pos, input_pos)``: ``None`` for a cache that holds its tokens in order with the chunk at the end, else a position
    for every slot: older tokens in random order, the chunk's own (the newest) in random slots."""
    B, G, T, L = case["batch"], case["groups"], case["new"], case["slots"]
    if not case["scattered"] or T >= L:
        return None, max(L - T, 0)
    order = torch.rand((B, G, L), generator=g, device="cuda").argsort(dim=-1)  # slots of the tokens from the oldest on
    pos = torch.cat((2 * torch.arange(L - T, device="cuda"), 2 * L + torch.arange(T, device="cuda"))).to(torch.int32)
    return torch.zeros((B, G, L), dtype=torch.int32, device="cuda").scatter_(2, order, pos.expand(B, G, L)), 2 * L


def _chunk_inputs(case, seed):
    g = _generator(seed)
    B, H, G, L = case["batch"], case["heads"], case["groups"], case["slots"]
    T = min(case.get("new", 1), L)
    q = _normal((B, H, T, D), g)
    k, v = _normal((B, G, L, D), g), _normal((B, G, L, D), g)
    return g, q, k, v


def _model(case, seed):
    """Random weights of a LitGPT-shaped model, cut to some of its layers, for inference."""
    from keys_values_b200.config import Config
    from keys_values_b200.models.model import GPT

    torch.manual_seed(seed)
    config = Config.from_name(case["model"], n_layer=case["layers"])
    with torch.device("cuda"):
        model = GPT(config).to(torch.bfloat16).eval()
    return config, model


def prepare(case, seed):
    kind = case["kind"]
    if kind == "token":
        _, q, k, v = _chunk_inputs(case, seed)
        return dict(case=case, q=q, k=k, v=v)
    if kind == "chunk":
        g, q, k, v = _chunk_inputs(case, seed)
        token_pos, input_pos = _positions(case, g)
        return dict(case=case, q=q, k=k, v=v, token_pos=token_pos, input_pos=input_pos)
    if kind == "gradient":
        from keys_values_b200 import ops

        g, q, k, v = _chunk_inputs(case, seed)
        token_pos, input_pos = _positions(case, g)
        out, _, lse = ops.sdpa_fwd(q, k, v, D**-0.5, input_pos, token_pos, False)  # kept by the forward half
        return dict(case=case, q=q, k=k, v=v, token_pos=token_pos, input_pos=input_pos, out=out, lse=lse, grad=_normal(out.shape, g),
                    dk=torch.zeros(k.shape, device="cuda"), dv=torch.zeros(v.shape, device="cuda"))
    g = _generator(seed)
    if kind == "lora":
        from keys_values_b200.finetune.engine import build_lora_training_setup

        setup = build_lora_training_setup(
            case["model"], torch.device("cuda"), torch.bfloat16, cache_name=f"h2o-torch-quantized{case['bits']}", cache_length=case["slots"],
            chunk_size=case["chunk"], lora_r=8, lora_alpha=16, micro_batch_size=case["batch"], n_layer=case["layers"], seed=seed,
        )
        for name, p in setup.gpt_model.named_parameters():
            if "lora_B" in name:  # a run that is under way: the second factor has left zero
                p.data.copy_(_normal(p.shape, g, torch.float32) * 0.02)
        vocab = setup.config.vocab_size
        return dict(case=case, model=setup.model, weights=[(n, p) for n, p in setup.gpt_model.named_parameters() if p.requires_grad],
                    ids=_ids((case["batch"], case["tokens"]), vocab, g), targets=_ids((case["batch"], case["targets"]), vocab, g))
    from keys_values_b200.kvcache.factory import KVCacheFactory
    from keys_values_b200.long_context import LongContextInferenceModel
    from keys_values_b200.models.head_model import CrossEntropyOnLogits

    if kind == "layered":
        from keys_values_b200.config import Config
        from keys_values_b200.models.registry import create_model, default_cache_name

        torch.manual_seed(seed)
        config = Config.from_name(case["model"])
        with torch.device("cuda"):
            model = create_model(config).to(torch.bfloat16).eval()
        name, slots, chunk, more = default_cache_name(config), case["tokens"] + 64, 2048, None
    else:
        config, model = _model(case, seed)
        name, slots, chunk, more = f"h2o-torch-quantized{case['bits']}", case["slots"], case["chunk"], dict(max_chunk_size=case["chunk"])
    model.assign_kv_caches(KVCacheFactory.create(model, name, case["batch"], slots, device=torch.device("cuda"), dtype=torch.bfloat16, cache_kwargs=more))
    through = LongContextInferenceModel(model, CrossEntropyOnLogits(config), chunk_size=chunk)
    if kind != "next":
        return dict(case=case, model=through, ids=_ids((case["batch"], case["tokens"]), config.vocab_size, g))
    from keys_values_b200.generate.decode_graph import Decoder

    # a generation under way: the prompts have filled the caches and the step has been captured
    through.fixed_max_seq_length = 1 << 17
    tokens = _ids((64, case["batch"], 1), config.vocab_size, g)
    with torch.inference_mode():
        through(_ids((case["batch"], case["slots"] + case["chunk"]), config.vocab_size, g))
        decoder = Decoder(model, case["batch"])
        for i in range(4):
            decoder(tokens[i])
    return dict(case=case, decoder=decoder, tokens=tokens, at=4)


# ------------------------------------------------------------------------------------------------ the work
def run(state):
    kind = state["case"]["kind"]
    if kind in ("token", "chunk", "gradient"):
        from keys_values_b200 import ops

        q, k, v = state["q"], state["k"], state["v"]
        if kind == "token":
            out, weights = ops.decode_attention(q, k, v, D**-0.5, k.shape[2] - 1, None, True)
            return dict(out=out, weights=weights)
        if kind == "chunk":
            out, weights, lse = ops.sdpa_fwd(q, k, v, D**-0.5, state["input_pos"], state["token_pos"], True)
            return dict(out=out, weights=weights, lse=lse)
        dq, _, _ = ops.sdpa_bwd(state["grad"], q, k, v, state["out"], state["lse"], D**-0.5, state["input_pos"], state["token_pos"],
                                dk_accum=state["dk"], dv_accum=state["dv"])
        return dict(dq=dq, dk=state["dk"], dv=state["dv"])
    if kind == "lora":
        for _, p in state["weights"]:
            p.grad = None
        loss = state["model"](state["ids"], state["targets"])
        loss.backward()
        return dict(loss=loss.detach(), **{n: p.grad for n, p in state["weights"]})
    with torch.inference_mode():
        if kind == "next":
            logits = state["decoder"](state["tokens"][state["at"]])
            state["at"] = (state["at"] + 1) % len(state["tokens"])
            return logits
        return state["model"](state["ids"])


# ------------------------------------------------------------------------------------------------ what it takes
def _pairs(new, slots):
    """Pairs of a chunk's query with a token that it may see."""
    new = min(new, slots)
    return new * (slots - new) + new * (new + 1) // 2


def _gpt_sizes(case):
    """(weights of a layer, width of an output row, heads x head size, keys' width, vocabulary) of the LitGPT-shaped models."""
    from keys_values_b200.config import Config

    c = Config.from_name(case["model"])
    hd, gd = c.n_head * c.head_size, c.n_query_groups * c.head_size
    return c.n_embd * (2 * hd + 2 * gd + 3 * c.intermediate_size), c.n_embd, hd, gd, c.padded_vocab_size


def work(case):
    kind = case["kind"]
    if kind in ("token", "chunk", "gradient"):
        B, H, G, L = case["batch"], case["heads"], case["groups"], case["slots"]
        T = min(case.get("new", 1), L)
        rows, cache = 2 * B * H * T * D, 2 * B * G * L * D  # bytes of queries or outputs, of keys or values
        if kind == "gradient":  # q, out, grad, dq; keys and values; their fp32 gradients read and written; lse
            return dict(flops=10 * B * H * D * _pairs(T, L), bytes=4 * rows + 2 * cache + 8 * cache + 4 * B * H * T)
        return dict(flops=4 * B * H * D * _pairs(T, L), bytes=2 * rows + 2 * cache + 4 * B * G * L + (4 * B * H * T if kind == "chunk" else 0))
    if kind == "layered":
        from keys_values_b200.config import Config
        from keys_values_b200.models.registry import create_model

        with torch.device("meta"):
            weights = sum(p.numel() for b in create_model(Config.from_name(case["model"])).transformer.h for p in b.parameters())
        return dict(flops=2 * weights * case["batch"] * case["tokens"], bytes=2 * weights)
    per_layer, width, hd, gd, vocab = _gpt_sizes(case)
    B, layers, L = case["batch"], case["layers"], case["slots"]
    if kind == "next":
        stored = 2 * B * gd * L * case["bits"] // 8 + 2 * 8 * B * (gd // D) * L  # codes, scales and zero points
        return dict(flops=B * (2 * (layers * per_layer + vocab * width) + layers * 4 * hd * L),
                    bytes=2 * (layers * per_layer + vocab * width) + layers * (stored + 8 * B * (gd // D) * L) + 2 * B * vocab)
    T = case["tokens"]
    pairs = _pairs(min(T, L), min(T, L)) + max(T - L, 0) * L
    forward = B * layers * (2 * per_layer * T + 4 * hd * pairs)
    if kind == "prompt":
        return dict(flops=forward + 2 * B * vocab * width, bytes=2 * (layers * per_layer + vocab * width))
    # forward, gradients of the activations (weights are frozen), attention backward, the head on the targets
    back = B * layers * (2 * per_layer * T + 10 * hd * pairs)
    return dict(flops=forward + back + 4 * B * case["targets"] * vocab * width, bytes=2 * 2 * (layers * per_layer + vocab * width))


def tolerance(case):
    # About four times the distance to the plain PyTorch restatement of attention on the same inputs (0.0026 for attention, 0.0049
    # for logits). LoRA gradients are 0.012 from it: the restatement's scores evict other slots here and there.
    if case["kind"] == "lora":
        return {"rel": 0.03}
    return {"rel": 0.01} if case["kind"] in ("token", "chunk", "gradient") else {"rel": 0.02}


# ------------------------------------------------------------------------------------------------ in 64 bits
def exact(case, seed):
    """Attention in 64 bits, one (sequence, group) after the other; whole models have no such value."""
    kind = case["kind"]
    if kind not in ("token", "chunk", "gradient"):
        return None
    g, q, k, v = _chunk_inputs(case, seed)
    B, H, T, _ = q.shape
    G, L = k.shape[1], k.shape[2]
    gs = H // G
    token_pos, input_pos = _positions(case, g) if kind != "token" else (None, L - 1)
    o = torch.empty((B, T, H, D), dtype=torch.float64, device="cuda")
    lse = torch.empty((B, H, T), dtype=torch.float64, device="cuda")
    weights = torch.empty((B, G, L), dtype=torch.float64, device="cuda")
    if kind == "gradient":
        grad = _normal((B, T, H * D), g).view(B, T, H, D)
        dq = torch.empty((B, H, T, D), dtype=torch.float64, device="cuda")
        dk, dv = torch.empty((B, G, L, D), dtype=torch.float64, device="cuda"), torch.empty((B, G, L, D), dtype=torch.float64, device="cuda")
    at = torch.arange(T, device="cuda").repeat(gs) + input_pos
    for b in range(B):
        for n in range(G):
            heads = slice(n * gs, (n + 1) * gs)
            qq, kk, vv = q[b, heads].reshape(gs * T, D).double(), k[b, n].double(), v[b, n].double()
            pos = torch.arange(L, device="cuda") if token_pos is None else token_pos[b, n]
            s = (qq @ kk.T).mul_(D**-0.5).masked_fill_(pos[None, :] > at[:, None], -math.inf)
            z = torch.logsumexp(s, dim=-1)
            p = s.sub_(z[:, None]).exp_()
            lse[b, heads] = z.view(gs, T)
            weights[b, n] = p.sum(0) / gs
            res = p @ vv
            o[b, :, heads] = res.view(gs, T, D).transpose(0, 1)
            if kind == "gradient":
                go = grad[b, :, heads].transpose(0, 1).reshape(gs * T, D).double()
                dv[b, n] = p.T @ go
                ds = (go @ vv.T).sub_((go * res).sum(-1, keepdim=True)).mul_(p).mul_(D**-0.5)
                dq[b, heads] = (ds @ kk).view(gs, T, D)
                dk[b, n] = ds.T @ qq
    if kind == "gradient":
        return dict(dq=dq, dk=dk, dv=dv)
    out = o.view(B, T, H * D)
    return dict(out=out, weights=weights) if kind == "token" else dict(out=out, weights=weights, lse=lse)
