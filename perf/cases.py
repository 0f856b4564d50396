"""What a program does with this framework on one GPU, as a list of measurable cases.

Five kinds of work, each through the calls that a user's program makes:

* ``step``: one token per sequence on a filled ``StaticKVCache``, replayed from a CUDA graph (what ``GraphedGreedyDecoder`` does for
  every token); returns the logits and the cache.
* ``prompt``: a whole prompt through a fused model without gradients, filling the cache; returns the last token's logits and the cache.
* ``layers``: the same for a model whose layers are recurrences, scans and grouped-query attention (Begovik).
* ``train``: one micro-batch, forward and backward, of a fused model whose gradients live in ``FusedAdamW``'s flat buffer; returns the
  loss and every gradient.
* ``experts``: a mixture of experts with a shared expert, added to the residual stream.

Weights and inputs come from the seed. ``exact`` states the same in 64-bit PyTorch.
"""
from __future__ import annotations

import math

import torch

VOCAB = {"gpt2": 50257, "gpt_neo": 50257, "gptj": 50400}
POSITIONS = 2048
WINDOW = 256                 # GPT-Neo's local layers
ROTARY = 64                  # GPT-J's rotated dimensions per head
EPS = 1e-5
TYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}
LOSS_SCALE = {"bf16": 1.0, "fp16": 4096.0}
TRAINED = {"gpt2": 4, "gpt_neo": 4, "gptj": 2}       # most layers of a training case (their gradients are all returned)


# ------------------------------------------------------------------------------------------------------------------ the cases
def listed():
    return [
        # a chat with a small model: launches and latency are everything
        dict(name="gpt2_step_1", kind="step", family="gpt2", width=768, heads=12, layers=12, rows=1, cached=173, dtype="bf16"),
        # one user of a large model: weights stream once per token
        dict(name="gptj_step_1", kind="step", family="gptj", width=4096, heads=16, layers=4, rows=1, cached=640, dtype="bf16"),
        # a few users with long contexts: weights and cache weigh alike
        dict(name="gptj_step_8", kind="step", family="gptj", width=2048, heads=16, layers=6, rows=8, cached=2047, dtype="bf16"),
        # a server's full batch, 16-bit floats as GPT-J is published
        dict(name="gptj_step_32", kind="step", family="gptj", width=4096, heads=16, layers=4, rows=32, cached=1100, dtype="fp16"),
        # scoring two documents of odd length: global and windowed layers
        dict(name="neo_prompt_2x1531", kind="prompt", family="gpt_neo", width=2048, heads=16, layers=4, rows=2, tokens=1531, dtype="fp16"),
        # the prompts of a batch at full context
        dict(name="gptj_prompt_4x2048", kind="prompt", family="gptj", width=4096, heads=16, layers=4, rows=4, tokens=2048, dtype="bf16"),
        # prompts of the model with recurrent layers, one group of its three kinds
        dict(name="begovik_prompt_4x2048", kind="layers", width=2048, heads=16, layers=3, rows=4, tokens=2048, dtype="bf16"),
        # fine-tuning a small model on padded sequences, 16-bit floats with a loss scale
        dict(name="gpt2_train_8x1000", kind="train", family="gpt2", width=768, heads=12, layers=4, rows=8, tokens=1000, dtype="fp16", padded=True),
        # training with windowed layers and an odd length
        dict(name="neo_train_4x1777", kind="train", family="gpt_neo", width=2048, heads=16, layers=2, rows=4, tokens=1777, dtype="bf16", padded=False),
        # a micro-batch of the headline training run (two of its layers, the whole vocabulary)
        dict(name="gptj_train_4x2048", kind="train", family="gptj", width=4096, heads=16, layers=2, rows=4, tokens=2048, dtype="bf16", padded=False),
        # experts of a decode step and of a prompt
        dict(name="experts_64", kind="experts", width=2048, ff=1344, experts=16, top=3, rows=64, dtype="bf16"),
        dict(name="experts_6000", kind="experts", width=2048, ff=1344, experts=16, top=3, rows=6000, dtype="bf16"),
    ]


def _log(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    dtype = rng.choice(["bf16", "fp16"])
    kind = rng.choice(["step", "step", "prompt", "train", "train", "layers", "experts"])
    family, width, heads = rng.choice([("gpt2", 768, 12), ("gpt_neo", 2048, 16), ("gptj", 2048, 16), ("gptj", 4096, 16)])
    if kind == "step":
        rows = _log(rng, 1, 64)
        limit = 1023 if family == "gpt2" else 2047
        return dict(kind=kind, family=family, width=width, heads=heads, layers=rng.randint(2, 4), rows=rows,
                    cached=min(_log(rng, 16, limit), 40000 // rows), dtype=dtype)
    if kind == "prompt":
        rows = _log(rng, 1, 8)
        return dict(kind=kind, family=family, width=width, heads=heads, layers=rng.randint(2, 4), rows=rows,
                    tokens=min(_log(rng, 17, 1024 if family == "gpt2" else 2048), 8192 // rows), dtype=dtype)
    if kind == "train":
        rows = _log(rng, 1, 8)
        layers = 1 if width == 4096 else 2
        return dict(kind=kind, family=family, width=width, heads=heads, layers=layers, rows=rows,
                    tokens=min(_log(rng, 65, 1024 if family == "gpt2" else 2048), 7000 // rows), dtype=dtype, padded=rng.random() < 0.3)
    if kind == "layers":
        rows = _log(rng, 1, 8)
        width = rng.choice([1024, 2048])
        return dict(kind=kind, width=width, heads=width // 128, layers=3, rows=rows, tokens=min(_log(rng, 17, 2048), 8192 // rows), dtype=dtype)
    return dict(kind=kind, width=rng.choice([1024, 2048]), ff=rng.choice([640, 1344]), experts=rng.choice([8, 16, 32]), top=rng.randint(2, 4),
                rows=_log(rng, 1, 8192), dtype=dtype)


# ------------------------------------------------------------------------------------------------------------------ weights and inputs
def _begovik(case):
    """Configuration of the layered model: recurrence with a bonus, selective scan, attention beside constant decays."""
    w, h = case["width"], case["heads"]
    dim = w // h
    mlp = {"kind": "dense", "ff": 8 * w // 3 // 64 * 64, "limit": 7.0}
    left = {"heads": h, "kv_heads": h // 4, "dim": dim, "vdim": dim, "scale": dim ** -0.5, "softcap": 50.0, "rot": {"base": 500000.0, "dims": dim // 2}}
    right = {"heads": h, "dim": dim, "vdim": dim, "decay": [1.0 - 2.0 ** (-1 - 9 * i / h) for i in range(h)]}
    kinds = [("wkv", {"heads": w // 64, "dim": 64, "decay_rank": 64}),
             ("mamba1", {"inner": 2 * w, "state": 16, "dt_rank": w // 16, "conv": 4}), ("parallel", {"left": left, "right": right})]
    return dict(vocab=VOCAB["gptj"], width=w, norm={"eps": EPS}, embedding={"scale": w ** 0.5}, residual_mult=0.5,
                layers=[{"type": kinds[i % 3][0], "mixer": kinds[i % 3][1], "mlp": mlp} for i in range(case["layers"])])


def _shapes(case):
    """``{name: (shape, mean, spread)}`` of the model's parameters. A spread of ``None``: values of their own (``_special``)."""
    w, n = case["width"], case["layers"] if "layers" in case else 0
    one, bias = (1.0, 0.1), (0.0, 0.02)
    out = {}
    if case["kind"] == "experts":
        e, ff = case["experts"], case["ff"]
        return {"router.weight": ((e, w), 0.0, 0.05), "up": ((e, 2 * ff, w), 0.0, 0.02), "down": ((e, w, ff), 0.0, 0.02),
                "shared.in_proj.weight": ((2 * ff, w), 0.0, 0.02), "shared.down.weight": ((w, ff), 0.0, 0.02)}
    if case["kind"] == "layers":
        cfg = _begovik(case)
        out["embed"], out["final.norm"], out["head"] = ((cfg["vocab"], w), 0.0, 0.02), ((w,), *one), ((cfg["vocab"], w), 0.0, 0.02)
        for i, layer in enumerate(cfg["layers"]):
            m, mx, ff = layer["mixer"], f"l{i}.mix.", layer["mlp"]["ff"]
            for name in ("norm1", "norm2"):
                out[f"l{i}.{name}"] = ((w,), *one)
            mats = {}
            if layer["type"] == "wkv":
                inner = m["heads"] * m["dim"]
                mats = {**{c: (inner, w) for c in "rkvg"}, "w1": (m["decay_rank"], w), "w2": (inner, m["decay_rank"]), "o": (w, inner)}
                for c in "rkvgw":
                    out[f"{mx}mu.{c}"] = ((w,), 0.5, 0.1)
                out.update({mx + "w0": ((inner,), 0.0, None), mx + "u": ((m["heads"], m["dim"]), 0.0, 0.3), mx + "norm": ((inner,), *one)})
            elif layer["type"] == "mamba1":
                inner, rank, state = m["inner"], m["dt_rank"], m["state"]
                mats = {"in": (2 * inner, w), "x": (rank + 2 * state, inner), "dt": (inner, rank), "o": (w, inner)}
                out.update({mx + "conv": ((inner, m["conv"]), 0.0, 0.5), mx + "conv.b": ((inner,), *bias), mx + "dt.b": ((inner,), 0.0, None),
                            mx + "A_log": ((inner, state), 0.0, None), mx + "D": ((inner,), *one)})
            else:
                a, b = m["left"], m["right"]
                kv = a["kv_heads"] * a["dim"]
                mats = {"left.q": (w, w), "left.k": (kv, w), "left.v": (kv, w), "left.o": (w, w), **{f"right.{c}": (w, w) for c in "qkvgo"}}
                out.update({mx + "left.q.norm": ((a["dim"],), *one), mx + "left.k.norm": ((a["dim"],), *one), mx + "right.norm": ((w,), *one),
                            mx + "left.out": ((w,), *one), mx + "right.out": ((w,), *one)})
            mats = {mx + k: v for k, v in mats.items()}
            mats.update({f"l{i}.mlp.gate": (ff, w), f"l{i}.mlp.up": (ff, w), f"l{i}.mlp.down": (w, ff)})
            out.update({k: (v, 0.0, 0.02) for k, v in mats.items()})
        return out
    family = case["family"]
    t = "transformer."
    spread = 0.01 if family == "gpt_neo" else 0.02          # GPT-Neo's scores are not scaled
    out[t + "wte.weight"] = ((VOCAB[family], w), 0.0, 0.02)
    if family != "gptj":
        out[t + "wpe.weight"] = ((POSITIONS, w), 0.0, 0.02)
    for i in range(n):
        h = f"{t}h.{i}."
        for name in ("ln_1",) if family == "gptj" else ("ln_1", "ln_2"):
            out[f"{h}{name}.weight"], out[f"{h}{name}.bias"] = ((w,), *one), ((w,), *bias)
        if family == "gpt2":                                 # weights [in, out]
            mats = {"attn.c_attn": (w, 3 * w, 3 * w), "attn.c_proj": (w, w, w), "mlp.c_fc": (w, 4 * w, 4 * w), "mlp.c_proj": (4 * w, w, w)}
        else:                                                # weights [out, in]; the last entry: size of the bias, 0 for none
            at, up, down = ("attn.", "mlp.fc_in", "mlp.fc_out") if family == "gptj" else ("attn.attention.", "mlp.c_fc", "mlp.c_proj")
            mats = {**{f"{at}{c}_proj": (w, w, 0) for c in "qkv"}, f"{at}out_proj": (w, w, 0 if family == "gptj" else w), up: (4 * w, w, 4 * w),
                    down: (w, 4 * w, w)}
        for name, (a, b, c) in mats.items():
            out[f"{h}{name}.weight"] = ((a, b), 0.0, spread)
            if c:
                out[f"{h}{name}.bias"] = ((c,), *bias)
    out[t + "ln_f.weight"], out[t + "ln_f.bias"] = ((w,), *one), ((w,), *bias)
    if family == "gptj":
        out["lm_head.weight"], out["lm_head.bias"] = ((VOCAB[family], w), 0.0, 0.02), ((VOCAB[family],), *bias)
    return out


def _special(name, shape, device):
    """Decays and step sizes as such models are initialised."""
    if name.endswith("w0"):
        return torch.linspace(-6.0, -1.0, shape[0], device=device)
    if name.endswith("dt.b"):
        return torch.linspace(math.log(math.expm1(1e-3)), math.log(math.expm1(0.1)), shape[0], device=device)
    return torch.log(torch.arange(1.0, shape[1] + 1.0, device=device)).repeat(shape[0], 1)


def _weights(case, gen):
    dtype = TYPES[case["dtype"]]
    out = {}
    for name, (shape, mean, spread) in _shapes(case).items():
        if spread is None:
            out[name] = _special(name, shape, gen.device).to(dtype)
        else:
            out[name] = torch.empty(shape, dtype=dtype, device=gen.device).normal_(mean, spread, generator=gen)
    return out


def _inputs(case, gen):
    """Token ids, the next token, the padding mask (or ``None``) and labels; or the rows that the experts read."""
    if case["kind"] == "experts":
        x = torch.randn(case["rows"], case["width"], device=gen.device, generator=gen)
        h = x * torch.rsqrt(x.square().mean(-1, keepdim=True) + EPS)
        return dict(x=x * 3.0, h=h.to(TYPES[case["dtype"]]))
    vocab = VOCAB[case.get("family", "gptj")]
    n = case["cached"] if case["kind"] == "step" else case["tokens"]
    ids = torch.randint(0, vocab, (case["rows"], n), device=gen.device, generator=gen)
    out = dict(ids=ids, cur=torch.randint(0, vocab, (case["rows"], 1), device=gen.device, generator=gen), mask=None, labels=ids)
    if case.get("padded"):
        length = torch.randint(n // 2, n + 1, (case["rows"], 1), device=gen.device, generator=gen)
        out["mask"] = (torch.arange(n, device=gen.device) < length).long()
        out["labels"] = ids.masked_fill(out["mask"] == 0, -100)
    return out


def _made(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    return _weights(case, gen), _inputs(case, gen)


# ------------------------------------------------------------------------------------------------------------------ the framework's side
def _model(case, weights):
    import oslo_b200 as ob
    dtype = TYPES[case["dtype"]]
    w, n, heads = case["width"], case["layers"], case["heads"]
    if case["kind"] == "layers":
        cls, cfg = ob.BegovikForCausalLM, ob.BegovikConfig(**_begovik(case), torch_dtype=dtype)
    elif case["family"] == "gpt2":
        cls, cfg = ob.GPT2LMHeadModel, ob.GPT2Config(vocab_size=VOCAB["gpt2"], n_positions=POSITIONS, n_embd=w, n_layer=n, n_head=heads,
                                                     resid_pdrop=0.0, embd_pdrop=0.0, attn_pdrop=0.0, torch_dtype=dtype)
    elif case["family"] == "gpt_neo":
        cls, cfg = ob.GPTNeoForCausalLM, ob.GPTNeoConfig(
            vocab_size=VOCAB["gpt_neo"], max_position_embeddings=POSITIONS, hidden_size=w, num_layers=n, num_heads=heads, window_size=WINDOW,
            attention_types=[[[["global", "local"][i % 2]], 1] for i in range(n)], torch_dtype=dtype)
    else:
        cls, cfg = ob.GPTJForCausalLM, ob.GPTJConfig(vocab_size=VOCAB["gptj"], n_positions=POSITIONS, n_embd=w, n_layer=n, n_head=heads,
                                                     rotary_dim=ROTARY, torch_dtype=dtype)
    with torch.device("cuda"):
        model = cls._from_config(cfg, torch_dtype=dtype)
    model.load_checkpoint_state(weights)
    model.tie_weights()
    return model.fuse()


def prepare(case, seed):
    weights, inputs = _made(case, seed)
    state = dict(case=case, **inputs)
    if case["kind"] == "experts":
        from oslo_b200.models.mixers import MixtureOfExperts
        dtype = TYPES[case["dtype"]]
        moe = MixtureOfExperts(case["width"], case["ff"], case["experts"], case["top"], unit="clamped", scored="sigmoid", limit=7.0,
                               scale_input=True, shared=case["ff"], shared_gate=False, shared_limit=7.0).to("cuda", dtype)
        moe.load_state_dict(weights)
        for m in moe.modules():
            m.oslo_fused = True
        state["moe"] = moe.requires_grad_(False)
        return state
    from oslo_b200.models.common import StaticKVCache
    model = state["model"] = _model(case, weights)
    if case["kind"] == "train":
        from oslo_b200.optim import FusedAdamW
        model.train()
        state["optimizer"] = FusedAdamW(model.parameters(), lr=1e-4)
        state["parameters"] = dict(model.named_parameters())
        return state
    model.eval().requires_grad_(False)
    if case["kind"] != "step":
        state["cache"] = StaticKVCache(case["tokens"])
        return state
    # prompt, then the step as a graph whose positions live on the device
    n = case["cached"]
    cache = state["cache"] = StaticKVCache(n + 1)
    with torch.no_grad():
        model(input_ids=state["ids"], past_key_values=cache, use_cache=True, last_token_logits=True)

        def step():
            return model(input_ids=state["cur"], past_key_values=cache, position_ids=cache.lengths_dev.long().unsqueeze(1), use_cache=True,
                         last_token_logits=True).logits

        def rewind():
            cache.length = n
            cache.use_device_positions(True)

        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            for _ in range(2):
                rewind()
                step()
            rewind()
        torch.cuda.current_stream().wait_stream(side)
        state["graph"] = torch.cuda.CUDAGraph()
        with torch.cuda.graph(state["graph"]):
            state["logits"] = step()
        cache.length = n
    return state


def _kept(case, cache):
    """What the cache holds, layer by layer."""
    out = []
    for i in range(case["layers"]):
        if i in cache.k:
            out += [cache.k[i], cache.v[i]]
        out += [cache.state[key] for key in (i, (i, "shift"), (i, "conv")) if key in cache.state]
    return out


def run(state):
    case = state["case"]
    if case["kind"] == "train":
        model = state["model"]
        state["optimizer"].zero_grad()
        loss = model(input_ids=state["ids"], labels=state["labels"], attention_mask=state["mask"], output_logits=False, use_cache=False).loss
        (loss * LOSS_SCALE[case["dtype"]]).backward()
        return [loss.detach(), {k: p.grad for k, p in state["parameters"].items()}]
    with torch.no_grad():
        if case["kind"] == "experts":
            from oslo_b200 import ops
            from oslo_b200.ops.reference import Branch
            out = state["moe"](state["h"])
            x, copies = ops.branch_join(state["x"], [Branch(out.y, slots=out.slots, top=case["top"]), Branch(out.shared)], 1.0, EPS, [],
                                        TYPES[case["dtype"]])
            return [x, copies[0]]
        cache = state["cache"]
        if case["kind"] == "step":
            cache.use_device_positions(True)         # the same token again
            state["graph"].replay()
            return [state["logits"], *_kept(case, cache)]
        cache.reset()
        logits = state["model"](input_ids=state["ids"], past_key_values=cache, use_cache=True, last_token_logits=True).logits
        return [logits, *_kept(case, cache)]


# ------------------------------------------------------------------------------------------------------------------ what a pass cannot do without
def work(case):
    w, size = case["width"], 2
    if case["kind"] == "experts":
        n, ff = case["rows"], case["ff"]
        flops = 6.0 * n * (case["top"] + 1) * w * ff
        used = min(case["experts"], n * case["top"])
        return {"bytes": size * 3.0 * (used + 1) * w * ff + n * w * (size + 4 + 4 + size), "flops": flops}
    n = case["rows"] * (1 if case["kind"] == "step" else case["tokens"])
    vocab = VOCAB[case.get("family", "gptj")]
    params = sum(math.prod(shape) for name, (shape, _, _) in _shapes(case).items() if "wte" not in name and "wpe" not in name and name != "embed"
                 and "head" not in name)
    head, layers = vocab * w, case["layers"]
    if case["kind"] == "step":
        cache = 2.0 * case["rows"] * case["cached"] * w
        if case["family"] == "gpt_neo":
            cache = cache * sum(min(1.0, WINDOW / case["cached"]) if i % 2 else 1.0 for i in range(layers)) / layers
        return {"bytes": size * (params + head + layers * cache), "flops": 2.0 * n * (params + head) + 2.0 * layers * cache}
    t = case["tokens"]
    if case["kind"] == "layers":
        m = w // 128
        pairs = case["rows"] * t * t / 2 * 4 * w                                  # grouped-query attention
        rest = n * w * (4.0 * 128 + 6.0 * 64 + 2 * 6.0 * 16)                      # constant decays, bonus recurrence, scan: per state element
        states = case["rows"] * (128 * w + 64 * w + 2 * w * 16) * 4.0
        return {"bytes": size * (params + head + 2.0 * n * (m // 4) * 128) + states, "flops": 2.0 * n * params + 2.0 * case["rows"] * head + pairs + rest}
    reach = [t * t / 2 if case["family"] != "gpt_neo" or i % 2 == 0 or t <= WINDOW else WINDOW * t - WINDOW * WINDOW / 2 for i in range(layers)]
    pairs = case["rows"] * 4.0 * w * sum(reach)
    if case["kind"] == "prompt":
        return {"bytes": size * (params + head + 2.0 * n * w * layers), "flops": 2.0 * n * params + 2.0 * case["rows"] * head + pairs}
    # every weight read and every gradient written, the embeddings' among them (tied to the head except in GPT-J)
    gradients = sum(math.prod(shape) for shape, _, _ in _shapes(case).values())
    return {"bytes": size * (params + head + gradients), "flops": 3.0 * (2.0 * n * (params + head) + pairs)}


def tolerance(case):
    """About four times the error of the 16-bit path against ``exact``: activations, probabilities and gradients are rounded to 8
    (bf16) or 11 (fp16) bits once per kernel."""
    wide = case["dtype"] == "bf16"
    return {"rel": 0.03 if wide else 0.006, "max": 0.6 if wide else 0.15}


# ------------------------------------------------------------------------------------------------------------------ 64 bits
def _norm(x, w, b):
    mean = x.mean(-1, keepdim=True)
    return (x - mean) * torch.rsqrt((x - mean).square().mean(-1, keepdim=True) + EPS) * w + b


def _rms(x, w=1.0):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + EPS) * w


def _turn(x, dims, base):
    """``x`` ``[..., tokens, dim]``: pairs ``(2i, 2i + 1)`` of the first ``dims`` turn by ``position * base^(-2i / dims)``."""
    at = torch.arange(x.shape[-2], dtype=x.dtype, device=x.device)[:, None] * base ** (-torch.arange(0, dims, 2, dtype=x.dtype, device=x.device) / dims)
    c, s = at.cos(), at.sin()
    u, v = x[..., 0:dims:2], x[..., 1:dims:2]
    turned = torch.stack([u * c - v * s, v * c + u * s], -1).flatten(-2)
    return torch.cat([turned, x[..., dims:]], -1)


def _gelu(x):
    return 0.5 * x * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (x + 0.044715 * x ** 3)))


def _heads(x, heads):
    return x.unflatten(-1, (heads, -1)).transpose(1, 2)


def _attend(q, k, v, scale, mask=None, window=None, cap=0.0, sink=False):
    t = q.size(2)
    i = torch.arange(t, device=q.device)
    seen = i[None, :] <= i[:, None]
    if window is not None:
        seen = seen & (i[None, :] > i[:, None] - window)
    seen = seen[None, None]
    if mask is not None:
        seen = seen & (mask != 0)[:, None, None, :]
    s = torch.matmul(q, k.transpose(-1, -2)) * scale
    if cap:
        s = cap * torch.tanh(s / cap)
    s = s.masked_fill(~seen, -math.inf)
    if sink:
        s = torch.cat([s, s.new_zeros(*s.shape[:-1], 1)], -1)
    p = torch.softmax(s, -1)
    return torch.matmul(p[..., :t], v).transpose(1, 2).flatten(2)


def _gpt(case, p, ids, mask=None):
    """Hidden states after the last norm, and the keys and values of every layer."""
    family, heads = case["family"], case["heads"]
    dim = case["width"] // heads
    x = p["transformer.wte.weight"][ids]
    if family != "gptj":
        x = x + p["transformer.wpe.weight"][:ids.size(1)]
    kept = []
    for i in range(case["layers"]):
        h = f"transformer.h.{i}."
        norm = lambda n, x: _norm(x, p[f"{h}{n}.weight"], p[f"{h}{n}.bias"])                                    # noqa: E731

        def linear(n, x):
            weight = p[f"{h}{n}.weight"]
            return torch.matmul(x, weight if family == "gpt2" else weight.t()) + p.get(f"{h}{n}.bias", 0.0)

        a = norm("ln_1", x)
        if family == "gpt2":
            q, k, v = linear("attn.c_attn", a).chunk(3, -1)
        else:
            at = "attn." if family == "gptj" else "attn.attention."
            q, k, v = (linear(f"{at}{c}_proj", a) for c in "qkv")
        q, k, v = _heads(q, heads), _heads(k, heads), _heads(v, heads)
        if family == "gptj":
            q, k = _turn(q, ROTARY, 10000.0), _turn(k, ROTARY, 10000.0)
        kept += [k, v]
        o = _attend(q, k, v, 1.0 if family == "gpt_neo" else dim ** -0.5, mask, WINDOW if family == "gpt_neo" and i % 2 else None)
        if family == "gptj":
            x = x + linear("attn.out_proj", o) + linear("mlp.fc_out", _gelu(linear("mlp.fc_in", a)))
            continue
        x = x + linear("attn.c_proj" if family == "gpt2" else "attn.attention.out_proj", o)
        x = x + linear("mlp.c_proj", _gelu(linear("mlp.c_fc", norm("ln_2", x))))
    return _norm(x, p["transformer.ln_f.weight"], p["transformer.ln_f.bias"]), kept


def _logits(p, hidden):
    return torch.matmul(hidden, p.get("lm_head.weight", p["transformer.wte.weight"]).t()) + p.get("lm_head.bias", 0.0)


def _clamped(g, u):
    g, u = g.clamp(max=7.0), u.clamp(-7.0, 7.0)
    return g * torch.sigmoid(1.702 * g) * (u + 1.0)


def _wkv(h, get, m):
    """Recurrence with a bonus: outputs, state, last input."""
    b, t, _ = h.shape
    before = torch.cat([h.new_zeros(b, 1, h.size(2)), h[:, :-1]], 1)
    mix = {c: h + (before - h) * get("mu." + c) for c in "rkvgw"}
    r, k, v = ((mix[c] @ get(c).t()).view(b, t, m["heads"], m["dim"]) for c in "rkv")
    gate = torch.nn.functional.silu(mix["g"] @ get("g").t())
    decay = torch.exp(-torch.exp(torch.tanh(mix["w"] @ get("w1").t()) @ get("w2").t() + get("w0"))).view_as(r)
    u, s, out = get("u").view(m["heads"], m["dim"], 1), h.new_zeros(b, m["heads"], m["dim"], m["dim"]), []
    for i in range(t):
        kv = k[:, i, :, :, None] * v[:, i, :, None, :]
        out.append(((s + u * kv) * r[:, i, :, :, None]).sum(2))
        s = decay[:, i, :, :, None] * s + kv
    o = _rms(torch.stack(out, 1)).flatten(2) * get("norm") * gate
    return o @ get("o").t(), [s, h[:, -1]]


def _mamba(h, get, m):
    """Selective scan: outputs, state, last inputs of the convolution."""
    b, t, _ = h.shape
    x, z = (h @ get("in").t()).chunk(2, -1)
    taps = m["conv"]
    padded = torch.cat([x.new_zeros(b, taps - 1, x.size(2)), x], 1)
    last = padded[:, -(taps - 1):]
    x = torch.nn.functional.silu(sum(padded[:, j:j + t] * get("conv")[:, j] for j in range(taps)) + get("conv.b"))
    dt, bb, cc = (x @ get("x").t()).split([m["dt_rank"], m["state"], m["state"]], -1)
    dt = torch.nn.functional.softplus(dt @ get("dt").t() + get("dt.b"))
    a, s, out = -torch.exp(get("A_log")), h.new_zeros(b, m["inner"], m["state"]), []
    for i in range(t):
        s = torch.exp(dt[:, i, :, None] * a) * s + (dt[:, i] * x[:, i])[..., None] * bb[:, i, None, :]
        out.append((s * cc[:, i, None, :]).sum(-1))
    y = (torch.stack(out, 1) + get("D") * x) * torch.nn.functional.silu(z)
    return y @ get("o").t(), [s, last]


def _parallel(h, get, m):
    """Grouped-query attention beside constant decays: outputs, keys, values, state."""
    a, c = m["left"], m["right"]
    q = _rms(_heads(h @ get("left.q").t(), a["heads"]), get("left.q.norm"))
    k = _rms(_heads(h @ get("left.k").t(), a["kv_heads"]), get("left.k.norm"))
    v = _heads(h @ get("left.v").t(), a["kv_heads"])
    q, k = (_turn(t, a["rot"]["dims"], a["rot"]["base"]) for t in (q, k))
    group = a["heads"] // a["kv_heads"]
    o = _attend(q, k.repeat_interleave(group, 1), v.repeat_interleave(group, 1), a["scale"], cap=a["softcap"], sink=True)
    left = _rms(o @ get("left.o").t(), get("left.out"))
    q2, k2, v2 = (_heads(h @ get("right." + n).t(), c["heads"]) for n in "qkv")
    q2, k2, v2 = (torch.nn.functional.silu(t) for t in (q2, k2, v2))
    decay = torch.tensor(c["decay"], dtype=h.dtype, device=h.device)[:, None, None]
    s, out = h.new_zeros(h.size(0), c["heads"], c["dim"], c["vdim"]), []
    for i in range(h.size(1)):
        s = decay * s + k2[:, :, i, :, None] * v2[:, :, i, None, :]
        out.append(torch.matmul(q2[:, :, i, None, :], s)[:, :, 0])
    o = _rms(torch.stack(out, 1).flatten(2), get("right.norm")) * torch.sigmoid(h @ get("right.g").t())
    right = _rms(o @ get("right.o").t(), get("right.out"))
    return 0.5 * (left + right), [k, v, s]


def _layered(case, p, ids):
    cfg, kept = _begovik(case), []
    x = p["embed"][ids] * cfg["embedding"]["scale"]
    for i, layer in enumerate(cfg["layers"]):
        mixer = {"wkv": _wkv, "mamba1": _mamba, "parallel": _parallel}[layer["type"]]
        y, keep = mixer(_rms(x, p[f"l{i}.norm1"]), lambda n, i=i: p[f"l{i}.mix.{n}"], layer["mixer"])
        h = _rms(x, p[f"l{i}.norm2"])
        y = y + _clamped(h @ p[f"l{i}.mlp.gate"].t(), h @ p[f"l{i}.mlp.up"].t()) @ p[f"l{i}.mlp.down"].t()
        x, kept = x + cfg["residual_mult"] * y, kept + keep
    return [_rms(x[:, -1:], p["final.norm"]) @ p["head"].t(), *kept]


def _experts(case, p, inputs):
    h, x = inputs["h"].double(), inputs["x"].double()
    z, idx = torch.topk(h @ p["router.weight"].t(), case["top"], -1)
    weight = torch.sigmoid(z)
    half = case["ff"]
    shared = h @ p["shared.in_proj.weight"].t()
    total = _clamped(shared[:, :half], shared[:, half:]) @ p["shared.down.weight"].t()
    for e in range(case["experts"]):
        row, choice = (idx == e).nonzero(as_tuple=True)
        a = (h[row] * weight[row, choice][:, None]) @ p["up"][e].t()
        total.index_add_(0, row, _clamped(a[:, 0::2], a[:, 1::2]) @ p["down"][e].t())
    return [x + total, x + total]


def exact(case, seed):
    weights, inputs = _made(case, seed)
    train = case["kind"] == "train"
    p = {k: v.double().requires_grad_(train) for k, v in weights.items()}
    with torch.set_grad_enabled(train):
        if case["kind"] == "experts":
            return _experts(case, p, inputs)
        if case["kind"] == "layers":
            return _layered(case, p, inputs["ids"])
        if not train:
            ids = inputs["ids"] if case["kind"] == "prompt" else torch.cat([inputs["ids"], inputs["cur"]], 1)
            hidden, kept = _gpt(case, p, ids)
            return [_logits(p, hidden[:, -1:]), *kept]
        hidden, _ = _gpt(case, p, inputs["ids"], inputs["mask"])
        labels = inputs["labels"][:, 1:]
        loss = torch.nn.functional.cross_entropy(_logits(p, hidden[:, :-1]).flatten(0, 1), labels.flatten(), ignore_index=-100)
        grads = torch.autograd.grad(loss * LOSS_SCALE[case["dtype"]], list(p.values()))
        # no value for the loss: rounding errors of either sign cancel in the mean over all tokens, so how far a 16-bit model's loss is
        # from this one is chance (1e-7 to 1e-5 from seed to seed)
        return [None, dict(zip(p, grads))]
