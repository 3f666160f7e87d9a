"""The work that a user of this package has it do, as cases that can be timed and compared.

Five kinds, each through the public entry points:

  generate   FlashSTU.generate(): prefill of a prompt, then new tokens one by one
  score      FlashSTU.forward(): the logits of every position, in one call or in consecutive cached calls
  block      FlashSTUBlock: prefill of a prompt and, with `steps`, teacher-forced single-token calls on the cache
  mini       MiniSTU, spectral back-end
  lds        MiniSTU, distilled-LDS back-end: prefill and recurrent single-token calls

Weights are random with the scales of a trained model: every sub-layer adds a branch that is small against the
residual stream, so a model's next-token distributions are peaked and rounding does not decide the continuation.
"""
import math
import os

import torch

import flash_stu_2_b200 as F

VOCAB = 50257
FILTERS_8192 = os.path.join(os.path.dirname(os.path.abspath(F.__file__)), "data", "phi_8192_24.pt")
DTYPES = {"bf16": torch.bfloat16, "fp32": torch.float32}
SIZE = {"bf16": 2, "fp32": 4}


# ---------------------------------------------------------------------------------------------------- the cases
def _generate(name, d, layers, heads, L, window, mlp, dtype, batch, prompt, new, sampling, logits=False):
    return dict(name=name, kind="generate", d=d, layers=layers, heads=heads, L=L, window=window, mlp=mlp, dtype=dtype,
                batch=batch, prompt=prompt, new=new, sampling=sampling, logits=logits)


def _score(name, d, layers, heads, L, window, mlp, dtype, batch, length, calls):
    return dict(name=name, kind="score", d=d, layers=layers, heads=heads, L=L, window=window, mlp=mlp, dtype=dtype,
                batch=batch, length=length, calls=calls)


def _block(name, op, d, heads, L, window, dtype, batch, prompt, steps):
    """op: approx or full (the STU layer's two variants), attention."""
    return dict(name=name, kind="block", op=op, d=d, heads=heads, L=L, window=window, mlp=4, dtype=dtype, batch=batch,
                prompt=prompt, steps=steps)


def listed():
    return [
        # the small fp32 model: two short prompts continued greedily, with the logits (token-exact decoding)
        _generate("generate_small_fp32", 512, 12, 8, 2048, 512, 12, "fp32", 2, 128, 128, "greedy", True),
        # one interactive conversation on the 24-layer bf16 model: a token's latency is all that counts
        _generate("generate_one_bf16", 1536, 24, 12, 8192, 1024, 4, "bf16", 1, 333, 64, "top_p"),
        # serving: a full batch of 32 sequences on the same model
        _generate("generate_batch_bf16", 1536, 24, 12, 8192, 1024, 4, "bf16", 32, 2048, 128, "top_k"),
        # evaluation: logits of every position of texts of an odd length (perplexity, ranking)
        _score("score_ragged_bf16", 1024, 12, 16, 4096, 512, 4, "bf16", 4, 1999, 1),
        # a conversation read in three cached calls of uneven phase: chunked prefill
        _score("score_turns_bf16", 768, 12, 12, 4096, 512, 4, "bf16", 2, 2500, 3),
        # the standalone STU layer over its whole context: prefill throughput
        _block("stu_prefill_bf16", "approx", 1024, 16, 8192, 1024, "bf16", 8, 8192, 0),
        # the same layer streaming tokens near the end of its context: decode throughput
        _block("stu_stream_bf16", "approx", 1024, 16, 8192, 1024, "bf16", 8, 7680, 512),
        # the K-filter (einsum) variant of the layer, prefill and steps
        _block("stu_full_stream_bf16", "full", 1024, 16, 8192, 1024, "bf16", 8, 3000, 64),
        # the attention layer of the largest configuration over a long context
        _block("attention_prefill_bf16", "attention", 3072, 24, 8192, 2048, "bf16", 4, 8192, 0),
        # the smallest use: one sequence through a narrow fp32 layer, a short prompt and a few steps
        _block("stu_small_fp32", "approx", 256, 4, 512, 128, "fp32", 1, 50, 14),
        # MiniSTU as its default arguments make it: fp32, different input and output widths
        dict(name="mini_fp32", kind="mini", L=1024, K=24, d_in=64, d_out=96, dtype="fp32", batch=8, length=1000),
        # the distilled recurrent form: a long prefill, then steps at constant cost
        dict(name="lds_stream_bf16", kind="lds", L=16384, d_in=1024, d_out=1024, dtype="bf16", batch=16, length=6000,
             steps=64),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the same ranges.  No drawn case does more work than the batch generation above."""
    kind = rng.choice(["generate", "generate", "score", "block", "block", "block", "mini", "lds"])
    if kind == "generate":
        fp32 = rng.random() < 0.3
        d = rng.choice([256, 512, 768]) if fp32 else rng.choice([512, 768, 1024, 1536])
        head = rng.choice([64, 128])
        L = rng.choice([2048, 4096])
        batch = _log(rng, 1, 4 if fp32 else 32)
        new = rng.randint(16, 100)
        prompt = _log(rng, 16, 256 if fp32 else 1900)
        if fp32:
            how = "greedy"
        elif prompt * (2 if batch > 4 else 1) < 200:
            how = "greedy"
        else:
            how = rng.choice(["greedy", "top_k", "top_p"])
        c = _generate("", d, rng.randint(2, 12) if fp32 else rng.randint(4, 24), d // head, L, rng.choice([256, 500, 1024]),
                      rng.choice([4, 8]) if fp32 else 4, "fp32" if fp32 else "bf16", batch, prompt, new, how, fp32)
    elif kind == "score":
        fp32 = rng.random() < 0.2
        d = rng.choice([256, 384, 512]) if fp32 else rng.choice([512, 768, 1024, 1536])
        c = _score("", d, rng.randint(2, 4) if fp32 else rng.randint(4, 16), d // rng.choice([64, 128]), 4096,
                   rng.choice([256, 500, 1024]), 4, "fp32" if fp32 else "bf16", rng.randint(1, 2 if fp32 else 4),
                   _log(rng, 30, 500 if fp32 else 2500), rng.choice([1, 1, 2, 3]))
    elif kind == "block":
        op = rng.choice(["approx", "approx", "full", "attention"])
        fp32 = rng.random() < 0.25
        L = rng.choice([1024, 2048, 3000]) if (fp32 or op == "full") else rng.choice([2048, 4096, 8192])
        d = rng.choice([128, 256, 512]) if fp32 else rng.choice([512, 768, 1024] if op == "full" else [512, 1024, 1536, 2048])
        steps = rng.choice([0, rng.randint(1, 200)])
        prompt = _log(rng, 16, (600 if fp32 else L) - steps)
        batch = _log(rng, 1, 4 if fp32 else (4 if d > 1024 else 16))
        c = _block("", op, d, d // rng.choice([64, 128]), L, rng.choice([200, 512, 1024]), "fp32" if fp32 else "bf16",
                   batch, prompt, steps)
    elif kind == "mini":
        fp32 = rng.random() < 0.6
        L = rng.choice([256, 700, 1024, 2048])
        wide = [16, 32, 64, 96] if fp32 else [64, 128, 256, 512]
        c = dict(kind="mini", L=L, K=rng.choice([16, 24]), d_in=rng.choice(wide), d_out=rng.choice(wide),
                 dtype="fp32" if fp32 else "bf16", batch=_log(rng, 1, 8), length=rng.randint(L // 2, L))
    else:
        fp32 = rng.random() < 0.25
        wide = [64, 128, 256] if fp32 else [256, 512, 1024]
        c = dict(kind="lds", L=16384, d_in=rng.choice(wide), d_out=rng.choice(wide), dtype="fp32" if fp32 else "bf16",
                 batch=_log(rng, 1, 2 if fp32 else 16), length=_log(rng, 100, 1500 if fp32 else 8000),
                 steps=rng.choice([0, rng.randint(1, 128)]))
    c.pop("name", None)
    return c


# ---------------------------------------------------------------------------------------------------- state
_PHI = {}


def _filters(L, K, device):
    """The spectral filters of a length: input data that depends on no seed, kept as a program would keep them."""
    if (L, K) not in _PHI:
        if (L, K) == (8192, 24):
            phi = F.load_spectral_filters(FILTERS_8192, device=device, dtype=torch.float32)
        else:
            phi = F.get_spectral_filters(L, K, device=device, dtype=torch.float32)
        _PHI[(L, K)] = phi
    return _PHI[(L, K)]


def _fill(module, gen, stream, layers):
    """Random parameters: unit-gain inner matrices; embeddings of width `stream`; every matrix that writes to the
    residual stream scaled so that 2 * layers branches together stay below it."""
    branch = 0.7 * stream / math.sqrt(2 * layers)
    with torch.no_grad():
        for name, p in module.named_parameters():
            if name.endswith("norm.weight"):
                p.normal_(1.0, 0.1, generator=gen)
            elif name.endswith(("tok_emb.weight", "lm_head.weight")):
                p.normal_(0.0, stream, generator=gen)
            elif name.endswith("M_filters"):
                p.normal_(0.0, branch, generator=gen)
            elif "M_phi" in name:
                p.normal_(0.0, branch / math.sqrt(p.shape[1]), generator=gen)
            elif name.endswith("M_inputs"):
                p.normal_(0.0, p.shape[0] ** -0.5, generator=gen)
            elif name.endswith(("c_proj.weight", "down_proj.weight")):
                p.normal_(0.0, branch * p.shape[1] ** -0.5, generator=gen)
            else:
                p.normal_(0.0, p.shape[-1] ** -0.5, generator=gen)
    return module.eval()


def prepare(case, seed):
    dev = torch.device("cuda")
    gen = torch.Generator(device=dev).manual_seed(seed)
    dt, kind = DTYPES[case["dtype"]], case["kind"]
    randn = lambda *shape: torch.randn(*shape, generator=gen, device=dev)
    if kind in ("generate", "score"):
        L = case["L"]
        config = F.FlashSTUConfig(
            n_embd=case["d"], n_layers=case["layers"], n_heads=case["heads"], seq_len=L, window_size=case["window"],
            vocab_size=VOCAB, mlp_scale=case["mlp"], num_eigh=24, torch_dtype=dt,
            filter_path=FILTERS_8192 if L == 8192 else None)
        with torch.device(dev):
            model = F.FlashSTU(config)
        _fill(model, gen, 0.02, case["layers"])
        ids = torch.randint(0, VOCAB, (case["batch"], case.get("prompt") or case["length"]), generator=gen, device=dev)
        return dict(case=case, model=model, ids=ids, seed=seed, gen=torch.Generator(device=dev))
    if kind == "block":
        config = F.FlashSTUConfig(
            n_embd=case["d"], n_layers=1, n_heads=case["heads"], seq_len=case["L"], window_size=case["window"],
            vocab_size=1, mlp_scale=case["mlp"], num_eigh=24, torch_dtype=dt, use_attn=case["op"] == "attention",
            use_approx=case["op"] != "full")
        with torch.device(dev):
            block = F.FlashSTUBlock(config=config, phi=_filters(case["L"], 24, dev).to(dt))
        _fill(block, gen, 1.0, 1)
        x = randn(case["batch"], case["prompt"], case["d"]).to(dt)
        tokens = randn(case["steps"], case["batch"], 1, case["d"]).to(dt)
        return dict(case=case, block=block, x=x, tokens=tokens)
    if kind == "mini":
        torch.manual_seed(seed)
        m = F.MiniSTU(case["L"], case["K"], case["d_in"], case["d_out"], dtype=dt, device=dev,
                      precomputed_filters=_filters(case["L"], case["K"], dev))
        return dict(case=case, m=m.eval(), x=randn(case["batch"], case["length"], case["d_in"]).to(dt))
    torch.manual_seed(seed)
    m = F.MiniSTU(case["L"], 24, case["d_in"], case["d_out"], dtype=dt, device=dev, backend="lds")
    x = (0.5 * randn(case["batch"], case["length"], case["d_in"])).to(dt)
    tokens = (0.5 * randn(case["steps"], case["batch"], 1, case["d_in"])).to(dt)
    return dict(case=case, m=m.eval(), x=x, tokens=tokens)


# ---------------------------------------------------------------------------------------------------- one pass
SAMPLING = {"greedy": dict(do_sample=False), "top_k": dict(temperature=0.8, top_k=40),
            "top_p": dict(temperature=0.9, top_k=100, top_p=0.9)}


@torch.no_grad()
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "generate":
        state["gen"].manual_seed(state["seed"])
        return state["model"].generate(state["ids"], max_length=case["prompt"] + case["new"], generator=state["gen"],
                                       return_logits=case["logits"], **SAMPLING[case["sampling"]])
    if kind == "score":
        if case["calls"] == 1:
            return state["model"](state["ids"], use_cache=False).logits
        past, logits = None, []
        for part in state["ids"].chunk(case["calls"], dim=1):
            out = state["model"](part, past_key_values=past, use_cache=True)
            past = out.past_key_values
            logits.append(out.logits)
        return logits
    if kind == "block":
        # the layers update their input in place: a pass works on a copy, token rows are laid out one after the other
        x = state["x"].clone()
        y, past = state["block"](x, use_cache=True)
        rows = state["tokens"].clone()
        for row in rows.unbind(0):
            _, past = state["block"](row, past_key_value=past, use_cache=True)
        return (y, rows, past[:-1]) if case["steps"] else (y, past[:-1])   # all of the cache but its position words
    if kind == "mini":
        return state["m"](state["x"])
    y, past = state["m"](state["x"], use_cache=True)
    rows = []
    for row in state["tokens"].unbind(0):
        r, past = state["m"](row, past_key_value=past, use_cache=True)
        rows.append(r)
    return (y, torch.stack(rows), past[0]) if rows else (y, past[0])


# ---------------------------------------------------------------------------------------------------- work
def _attended(T0, T, window):
    """Keys that T queries from position T0 on attend to in one sequence: the query's own and `window` before it."""
    short = max(0, min(T, window + 1 - T0))
    return short * (2 * T0 + short + 1) // 2 + (T - short) * (window + 1)


def _layer(op, d, mlp, window, e, B, t0, T, K=24):
    """(weight bytes, state bytes, flops) of T new positions of one layer with t0 positions in its cache."""
    pairs = T * t0 + T * (T + 1) // 2
    flops = 2 * B * T * 3 * mlp * d * d
    weights = 3 * mlp * d * d * e
    if op == "attention":
        seen = min(t0, window)
        return (weights + 4 * d * d * e, 2 * B * (seen + T) * d * e,
                flops + 2 * B * T * 4 * d * d + 4 * B * d * _attended(t0, T, window))
    if op == "approx":   # even taps only: one parity of the history for a single position
        seen = t0 // 2 if T == 1 else t0
        return (weights + d * d * e, B * (seen + T) * d * e + d * (t0 + T) // 2 * e,
                flops + 2 * B * T * d * d + B * d * pairs)
    # K filters, both branches: the convolutions share their even and odd tap sums
    return (weights + 2 * K * d * d * e, B * (t0 + T) * d * e + K * (t0 + T) * e,
            flops + 2 * B * T * 2 * K * d * d + 2 * B * d * K * pairs)


def _model(case, B, t0, T, logit_rows):
    d, e = case["d"], SIZE[case["dtype"]]
    bytes_ = VOCAB * d * e + logit_rows * VOCAB * e + B * T * d * e
    flops = 2 * logit_rows * VOCAB * d
    for i in range(case["layers"]):
        w, s, f = _layer("attention" if i % 2 else "approx", d, case["mlp"], case["window"], e, B, t0, T)
        bytes_, flops = bytes_ + w + s, flops + f
    return bytes_, flops


def work(case):
    kind, B, e = case["kind"], case["batch"], SIZE[case["dtype"]]
    total = [0, 0]

    def add(bytes_, flops):
        total[0] += bytes_
        total[1] += flops

    if kind == "generate":
        add(*_model(case, B, 0, case["prompt"], B))
        for i in range(case["new"] - 1):
            add(*_model(case, B, case["prompt"] + i, 1, B))
    elif kind == "score":
        part = -(-case["length"] // case["calls"])
        for t0 in range(0, case["length"], part):
            T = min(part, case["length"] - t0)
            add(*_model(case, B, t0, T, B * T))
    elif kind == "block":
        for t0, T in [(0, case["prompt"])] + [(case["prompt"] + i, 1) for i in range(case["steps"])]:
            w, s, f = _layer(case["op"], case["d"], case["mlp"], case["window"], e, B, t0, T)
            add(w + s + 2 * B * T * case["d"] * e, f)
    elif kind == "mini":
        T, K, di, do = case["length"], case["K"], case["d_in"], case["d_out"]
        add((B * T * (di + do) + 2 * K * di * do + K * T) * e,
            2 * B * T * 2 * K * di * do + 2 * B * di * K * T * (T + 1) // 2)
    else:
        T, di, do, D, N = case["length"], case["d_in"], case["d_out"], 160, 48
        steps = case["steps"]
        add((B * (T + steps) * (di + do) + (1 + steps) * N * di * do) * e + B * di * D * 8 * (1 + 2 * steps),
            B * (T + steps) * (2 * N * di * do + 2 * N * D * di + 2 * D * di))
    return {"bytes": total[0], "flops": total[1]}


def tolerance(case):
    """bf16 results carry a rounding of 2^-9 at every layer boundary; fp32 sums run over up to 10^4 terms.  Tokens are
    whole numbers: a near-tie may fall the other way and change what follows it in that sequence."""
    rel = 1e-2 if case["dtype"] == "bf16" else 2e-5
    if case["kind"] == "lds" and case["dtype"] == "fp32":
        rel = 1e-4   # the features are differences of modes 10^4 times their size
    return {"rel": rel, "differ": 0.01} if case["kind"] == "generate" else {"rel": rel}
