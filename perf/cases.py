"""The work whose speed matters: what a user of the engine has it do, over the range it is used in.

A case is a batch of requests of a Qwen2 model and the steps that the step function
(`ModelRunner.step`) runs for it, or a call of `LLM.generate`. Qwen2 is the architecture of the
reference and of the benchmark; the sizes are the benchmark's (the layers of Qwen2.5-1.5B and -7B) and
the tests' (tiny). Eight layers, as where the benchmark puts architectures side by side: through
random weights a rounding error grows with the root of the depth, and at 28 layers two correct
bfloat16 implementations part by 4 % (8 layers: 2 %). Weights are N(0, 0.02), norm weights around 1,
as everywhere in this repository.

The fields of a case that runs steps:

  size, dtype       the model's sizes, "bfloat16" or "float32"
  decoding          requests that bring one token a step, each with a context in the cache already,
                    of context_low to context_high tokens
  prompts           requests that bring a portion of their prompt in the first step, of prompt_low to
                    prompt_high tokens after the `start` tokens that are in the cache already,
                    and one token in each further step
  steps             how many steps one pass runs. The tokens are given (as in a replay), the logits
                    of each request's last token come back from every step.
  pattern           what the lengths between low and high are drawn from

and of one that generates: size, dtype, prompts, prompt_low, prompt_high, new_tokens, pattern.
"""

import math
import random

import numpy as np
import torch

from paged_attention_engine_b200 import LLM, Engine, StepEntry

PAGE = 16
STD = 0.02
# Keys and values of a context that is in the cache already: what a projection of normed rows by
# N(0, 0.02) weights gives at these widths.
CACHE_STD = 0.8
MAX_BATCHED_TOKENS = 8192


def _qwen2(layers, hidden, heads, kv_heads, head_dim, ff, vocab, theta, eps, positions, tied):
    return dict(
        architectures=["Qwen2ForCausalLM"], num_hidden_layers=layers, hidden_size=hidden, num_attention_heads=heads,
        num_key_value_heads=kv_heads, head_dim=head_dim, intermediate_size=ff, vocab_size=vocab, rope_theta=theta,
        rms_norm_eps=eps, max_position_embeddings=positions, tie_word_embeddings=tied, use_sliding_window=False,
    )


SIZES = {
    "1.5b": _qwen2(8, 1536, 12, 2, 128, 8960, 151936, 1e6, 1e-6, 32768, True),
    "7b": _qwen2(8, 3584, 28, 4, 128, 18944, 152064, 1e6, 1e-6, 32768, False),
    "tiny": _qwen2(3, 96, 3, 1, 32, 256, 509, 1e6, 1e-5, 256, False),
}


def _steps(name, size="1.5b", dtype="bfloat16", decoding=0, context=(0, 0), prompts=0, prompt=(0, 0), start=0, steps=1, pattern=0):
    return dict(name=name, size=size, dtype=dtype, decoding=decoding, context_low=context[0], context_high=context[1], prompts=prompts,
                prompt_low=prompt[0], prompt_high=prompt[1], start=start, steps=steps, pattern=pattern)


def listed():
    return [
        # One user's chat: decoding at batch 1, at the benchmark's context.
        _steps("decode 1", decoding=1, context=(4080, 4080), steps=16),
        # The benchmark's default workload.
        _steps("decode 8", decoding=8, context=(4080, 4080), steps=16),
        # The benchmark's largest batch, where the cache outweighs the weights.
        _steps("decode 64", decoding=64, context=(4088, 4088), steps=8),
        # A server's ordinary step: requests of all ages.
        _steps("decode 40 ragged", decoding=40, context=(16, 3000), steps=16, pattern=1),
        # A short question's time to its first token.
        _steps("prompt 100", prompts=1, prompt=(100, 100)),
        # The benchmark's prefill.
        _steps("prompt 2048", prompts=1, prompt=(2048, 2048)),
        # A long document; also a whole step of the token budget.
        _steps("prompt 8192", prompts=1, prompt=(8192, 8192)),
        # A queue of new requests of mixed lengths admitted in one step.
        _steps("prompts ragged", prompts=9, prompt=(16, 1500), pattern=2),
        # Continuous batching: a portion of a long prompt beside requests that decode.
        _steps("mixed", decoding=48, context=(16, 2048), prompts=1, prompt=(509, 509), start=512, pattern=3),
        # The 7B stream of the benchmark in its steady state: 64 requests of ragged lengths.
        _steps("7b decode 64 ragged", size="7b", decoding=64, context=(16, 2048), steps=8, pattern=4),
        # The float32 engine, with which a user checks a model: a prompt and the first decoded tokens.
        _steps("float32 check", dtype="float32", prompts=1, prompt=(60, 60), steps=9),
        # The smallest calls: the tests' tiny model through the entry point, scheduler and sampler.
        dict(name="tiny generate", size="tiny", dtype="float32", prompts=5, prompt_low=1, prompt_high=64, new_tokens=12, pattern=5),
    ]


def _log_uniform(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(("decode", "decode", "decode", "prompt", "prompt", "prompts", "mixed", "7b decode", "7b prompt", "float32", "generate"))
    pattern = rng.randrange(1, 10**6)
    if kind == "generate":
        low = _log_uniform(rng, 1, 16)
        case = dict(size="tiny", dtype="float32", prompts=rng.randint(1, 8), prompt_low=low, prompt_high=rng.randint(low, 96),
                    new_tokens=rng.randint(4, 16), pattern=pattern)
        return case
    if kind == "float32":
        case = _steps("", dtype="float32", prompts=1, prompt=(_log_uniform(rng, 3, 60),) * 2, steps=rng.randint(2, 9), pattern=pattern)
    elif kind in ("decode", "7b decode"):
        big = kind == "7b decode"
        high = _log_uniform(rng, 32, 2048 if big else 4088)
        low = high if rng.random() < 0.4 else _log_uniform(rng, 16, high)
        case = _steps("", size="7b" if big else "1.5b", decoding=_log_uniform(rng, 1, 64), context=(low, high), steps=8, pattern=pattern)
    elif kind in ("prompt", "7b prompt"):
        big = kind == "7b prompt"
        n = _log_uniform(rng, 17, 2048 if big else 8192)
        start = 0 if big or rng.random() < 0.7 else PAGE * rng.randint(1, 128)
        case = _steps("", size="7b" if big else "1.5b", prompts=1, prompt=(n, n), start=start, pattern=pattern)
    elif kind == "prompts":
        low = _log_uniform(rng, 16, 512)
        case = _steps("", prompts=rng.randint(2, 12), prompt=(low, _log_uniform(rng, low, 2048)), steps=rng.choice((1, 1, 3)), pattern=pattern)
    else:
        high = _log_uniform(rng, 64, 2048)
        n = _log_uniform(rng, 17, 2048)
        case = _steps("", decoding=_log_uniform(rng, 2, 63), context=(_log_uniform(rng, 16, high), high), prompts=1, prompt=(n, n),
                      start=rng.choice((0, PAGE * rng.randint(1, 64))), pattern=pattern)
    case.pop("name")
    return case


# ------------------------------------------------------------------------------------------- #
# Inputs
# ------------------------------------------------------------------------------------------- #

def _lengths(case):
    """Per request (tokens in the cache already, tokens of the first step): decoding requests first."""
    rng = random.Random(case["pattern"])
    out = [(rng.randint(case["context_low"], case["context_high"]), 1) for _ in range(case["decoding"])]
    budget = MAX_BATCHED_TOKENS - len(out)
    for _ in range(case["prompts"]):
        n = min(budget, rng.randint(case["prompt_low"], case["prompt_high"]))
        if n > 0:
            out.append((case["start"], n))
        budget -= n
    return out


def _token_ids(case, seed):
    """Per request, the tokens that one pass gives it."""
    gen = np.random.default_rng([seed, 1])
    vocab = SIZES[case["size"]]["vocab_size"]
    return [gen.integers(0, vocab, first + case["steps"] - 1).tolist() for _, first in _lengths(case)]


def _cached(case, seed, dtype):
    """Per request, [layers, keys and values, pages, kv heads, page, head size]: what its pages hold
    before the pass (the places behind its context are overwritten before they are read), or None."""
    m = SIZES[case["size"]]
    gen = torch.Generator(device="cuda").manual_seed(seed * 1000003 + 17)
    for (context, _), ids in zip(_lengths(case), _token_ids(case, seed)):
        if context == 0:
            yield None
            continue
        pages = -(-(context + len(ids)) // PAGE)
        shape = (m["num_hidden_layers"], 2, pages, m["num_key_value_heads"], PAGE, m["head_dim"])
        yield torch.empty(shape, dtype=dtype, device="cuda").normal_(0.0, CACHE_STD, generator=gen)


def _prompts_to_generate(case, seed):
    rng = random.Random(case["pattern"])
    gen = np.random.default_rng([seed, 2])
    vocab = SIZES[case["size"]]["vocab_size"]
    return [tuple(gen.integers(0, vocab, rng.randint(case["prompt_low"], case["prompt_high"])).tolist()) for _ in range(case["prompts"])]


def prepare(case, seed):
    if "new_tokens" in case:
        longest = case["prompt_high"] + case["new_tokens"]
        llm = LLM.from_random(SIZES[case["size"]], seed=seed, dtype=case["dtype"], block_size=PAGE, max_num_seqs=case["prompts"],
                              num_blocks=case["prompts"] * (-(-longest // PAGE) + 1) + 8)
        return {"llm": llm, "prompts": _prompts_to_generate(case, seed), "new_tokens": case["new_tokens"]}
    lengths, ids = _lengths(case), _token_ids(case, seed)
    engine = Engine.from_random(SIZES[case["size"]], seed=seed, dtype=case["dtype"])
    # The pool holds exactly the pages that the requests take, so a request that is opened again
    # finds its own pages and its context again.
    cache = engine.new_paged_cache(sum(-(-(c + len(t)) // PAGE) for (c, _), t in zip(lengths, ids)), PAGE, len(lengths))
    runner = engine.new_runner(cache)
    requests = [(f"request {i}", c, len(t)) for i, ((c, _), t) in enumerate(zip(lengths, ids))]
    _open(runner, requests)
    for (key, _, _), held in zip(requests, _cached(case, seed, engine.dtype)):
        if held is not None:
            cache.pools[0][:, :, list(cache.manager.block_table(key))] = held
    _close(runner, requests)
    steps = []
    for s in range(case["steps"]):
        entries = []
        for (key, _, _), (_, first), t in zip(requests, lengths, ids):
            mine = tuple(t[:first]) if s == 0 else (t[first + s - 1],)
            entries.append(StepEntry(key, mine, (len(mine) - 1,)))
        steps.append(entries)
    # Where the pass fills the whole pool, the pages are an output.
    return {"runner": runner, "requests": requests, "steps": steps, "pages": None if any(c for c, _ in lengths) else cache.pools[0]}


def _open(runner, requests):
    for key, context, new in requests:
        assert runner.begin_request(key)
        assert runner.manager.reserve(key, context + new).ok
        runner.manager.advance(key, context)


def _close(runner, requests):
    for key, _, _ in requests:
        runner.end_request(key)


def run(state):
    if "llm" in state:
        return [np.asarray(t) for t in state["llm"].generate(state["prompts"], state["new_tokens"])]
    runner, requests = state["runner"], state["requests"]
    _open(runner, requests)
    # A step's logits are valid until the next step: who keeps them copies them.
    logits = [runner.step(entries).logits.clone() for entries in state["steps"]]
    _close(runner, requests)
    return {"logits": logits, "pages": state["pages"]}


# ------------------------------------------------------------------------------------------- #
# What a pass cannot do without
# ------------------------------------------------------------------------------------------- #

def work(case):
    m = SIZES[case["size"]]
    size = 4 if case["dtype"] == "float32" else 2
    d, heads, kv = m["head_dim"], m["num_attention_heads"], m["num_key_value_heads"]
    layer = m["hidden_size"] * (2 * heads + 2 * kv) * d + 3 * m["hidden_size"] * m["intermediate_size"]
    head = m["hidden_size"] * m["vocab_size"]
    key_bytes = 2 * m["num_hidden_layers"] * kv * d * size       # a token's keys and values
    if "new_tokens" in case:
        steps = [[(0, n) for n in (len(p) for p in _prompts_to_generate(case, 0))]]
        steps += [[(c + n + s, 1) for c, n in steps[0]] for s in range(case["new_tokens"] - 1)]
    else:
        first = _lengths(case)
        steps = [first] + [[(c + n + s, 1) for c, n in first] for s in range(case["steps"] - 1)]
    total_bytes = total_flops = 0.0
    for step in steps:
        tokens = sum(n for _, n in step)
        pairs = sum(n * c + n * (n + 1) // 2 for c, n in step)
        total_bytes += size * (m["num_hidden_layers"] * layer + head + tokens * m["hidden_size"])
        total_bytes += key_bytes * sum(c + n for c, n in step) + 4.0 * len(step) * m["vocab_size"]
        total_flops += 2.0 * tokens * m["num_hidden_layers"] * layer + 2.0 * len(step) * head
        total_flops += 4.0 * m["num_hidden_layers"] * heads * d * pairs
    return {"bytes": total_bytes, "flops": total_flops}


def tolerance(case):
    if "new_tokens" in case:
        return "exact"           # token ids
    if case["dtype"] == "float32":
        return {"rel": 1e-5}
    # Eight layers whose every result is rounded to bfloat16: 1.4e-2 to 2e-2 between the few-token and the
    # split-K products, or between the two prefill attentions; 1.1e-2 to 1.9e-2 from 64 bits.
    return {"rel": 0.03}


# ------------------------------------------------------------------------------------------- #
# The same in 64 bits
# ------------------------------------------------------------------------------------------- #

def _weights(m, seed, dtype):
    """The tensors that `from_random` draws: in the order of their names, from one generator."""
    d, hidden, ff = m["head_dim"], m["hidden_size"], m["intermediate_size"]
    nq, nkv = m["num_attention_heads"] * d, m["num_key_value_heads"] * d
    shapes = {"model.embed_tokens.weight": (m["vocab_size"], hidden), "model.norm.weight": (hidden,)}
    if not m["tie_word_embeddings"]:
        shapes["lm_head.weight"] = (m["vocab_size"], hidden)
    for i in range(m["num_hidden_layers"]):
        p = f"model.layers.{i}."
        for name, rows in (("q", nq), ("k", nkv), ("v", nkv)):
            shapes[f"{p}self_attn.{name}_proj.weight"] = (rows, hidden)
            shapes[f"{p}self_attn.{name}_proj.bias"] = (rows,)
        shapes[p + "self_attn.o_proj.weight"] = (hidden, nq)
        shapes[p + "mlp.gate_proj.weight"] = shapes[p + "mlp.up_proj.weight"] = (ff, hidden)
        shapes[p + "mlp.down_proj.weight"] = (hidden, ff)
        shapes[p + "input_layernorm.weight"] = shapes[p + "post_attention_layernorm.weight"] = (hidden,)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    out = {}
    for name in sorted(shapes):
        t = torch.randn(shapes[name], generator=gen, device="cuda", dtype=torch.float32) * STD
        out[name] = (t + 1.0 if name.endswith("norm.weight") else t).to(dtype)
    return out


def _rms(x, weight, eps):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps) * weight.double()


def _rotate(x, positions, theta):
    half = x.shape[-1] // 2
    angle = positions.double()[:, None] * theta ** (-torch.arange(half, device=x.device, dtype=torch.float64) / half)
    c, s = angle.cos()[:, None], angle.sin()[:, None]
    lo, hi = x[..., :half], x[..., half:]
    return torch.cat((lo * c - hi * s, hi * c + lo * s), -1)


def _attend(q, k, v, context, d):
    """q [tokens, heads, d] at positions context, context + 1, ...; k, v [keys, kv heads, d] -> [tokens, heads * d]"""
    tokens, heads, _ = q.shape
    group = heads // k.shape[1]
    out = torch.empty_like(q)
    at = torch.arange(k.shape[0], device=q.device)
    for t in range(0, tokens, 1024):
        n = min(1024, tokens - t)
        hidden = at[None, :] > (context + t + torch.arange(n, device=q.device))[:, None]
        for g in range(k.shape[1]):
            mine = q[t : t + n, g * group : (g + 1) * group].transpose(0, 1)
            scores = (mine @ k[:, g].T) * d**-0.5
            weights = scores.masked_fill_(hidden, -math.inf).softmax(-1)
            out[t : t + n, g * group : (g + 1) * group] = (weights @ v[:, g]).transpose(0, 1)
    return out.reshape(tokens, heads * d)


def _forward(m, w, ids, contexts, held, rows, keep=None):
    """Logits at the rows `rows` of all requests' tokens laid end to end. `held`: per request its pages
    before, or None; `keep`, a list, gets every layer's (keys, values)."""
    d, heads, kv = m["head_dim"], m["num_attention_heads"], m["num_key_value_heads"]
    counts = [len(t) for t in ids]
    ends = np.cumsum(counts).tolist()
    positions = torch.cat([c + torch.arange(n, device="cuda") for c, n in zip(contexts, counts)])
    x = w["model.embed_tokens.weight"][torch.tensor([t for r in ids for t in r], device="cuda")].double()
    for layer in range(m["num_hidden_layers"]):
        p = f"model.layers.{layer}."

        def product(y, name):
            return y @ w[p + name + ".weight"].double().T

        y = _rms(x, w[p + "input_layernorm.weight"], m["rms_norm_eps"])
        q, k, v = ((product(y, f"self_attn.{n}_proj") + w[f"{p}self_attn.{n}_proj.bias"].double()).view(len(y), -1, d) for n in "qkv")
        q, k = _rotate(q, positions, m["rope_theta"]), _rotate(k, positions, m["rope_theta"])
        if keep is not None:
            keep.append((k, v))
        parts = []
        for context, n, end, pages in zip(contexts, counts, ends, held):
            kk, vv = k[end - n : end], v[end - n : end]
            if context:
                old = pages[layer].double().transpose(2, 3).reshape(2, -1, kv, d)[:, :context]
                kk, vv = torch.cat((old[0], kk)), torch.cat((old[1], vv))
            parts.append(_attend(q[end - n : end], kk, vv, context, d))
        x = x + product(torch.cat(parts), "self_attn.o_proj")
        y = _rms(x, w[p + "post_attention_layernorm.weight"], m["rms_norm_eps"])
        gate = product(y, "mlp.gate_proj")
        x = x + product(gate * torch.sigmoid(gate) * product(y, "mlp.up_proj"), "mlp.down_proj")
    y = _rms(x[rows], w["model.norm.weight"], m["rms_norm_eps"])
    return y @ w["model.embed_tokens.weight" if m["tie_word_embeddings"] else "lm_head.weight"].double().T


@torch.inference_mode()
def exact(case, seed):
    m, dtype = SIZES[case["size"]], getattr(torch, case["dtype"])
    w = _weights(m, seed, dtype)
    if "new_tokens" in case:
        out = []
        for prompt in _prompts_to_generate(case, seed):
            ids = list(prompt)
            for _ in range(case["new_tokens"]):
                ids.append(int(_forward(m, w, [ids], [0], [None], [len(ids) - 1]).argmax()))
            out.append(np.asarray(ids[len(prompt) :]))
        return out
    lengths, ids = _lengths(case), _token_ids(case, seed)
    contexts = [c for c, _ in lengths]
    begin = np.concatenate(([0], np.cumsum([len(t) for t in ids]))).tolist()
    rows = [begin[i] + first - 1 + s for s in range(case["steps"]) for i, (_, first) in enumerate(lengths)]
    keep = None if any(contexts) else []
    logits = _forward(m, w, ids, contexts, list(_cached(case, seed, dtype)), rows, keep)
    pages = None
    if keep is not None:
        counts = [-(-len(t) // PAGE) for t in ids]
        pages = torch.zeros((len(keep), 2, sum(counts), m["num_key_value_heads"], PAGE, m["head_dim"]), dtype=torch.float64, device="cuda")
        for layer, written in enumerate(keep):
            for kind, all_rows in enumerate(written):
                at = 0
                for t, b, n in zip(ids, begin, counts):
                    padded = torch.zeros((n * PAGE, *all_rows.shape[1:]), dtype=torch.float64, device="cuda")
                    padded[: len(t)] = all_rows[b : b + len(t)]
                    pages[layer, kind, at : at + n] = padded.view(n, PAGE, *all_rows.shape[1:]).transpose(1, 2)
                    at += n
    return {"logits": list(logits.split(len(lengths))), "pages": pages}
