"""The work that programs have this engine do, as cases that can be timed and checked one by one.

A case names a model, a precision and one pass: a step of the engine (decoded tokens, portions of prompts, or both
together), a whole request, or a whole call of ``LLM.generate``.  The models are the shapes that the framework's own
benchmark and tests use: Llama-3 decoders of 1B, 3B and 8B size, a tiny one, and a Bomotar (attention behind short
convolutions beside a delta rule) of the benchmark's smaller width with dense feed-forwards.  (Routed experts are
left out: where two experts' scores lie close, rounding decides between them, and no tolerance describes that.)

Weights are ``N(0, 0.02)`` as the random-weights mode draws them from the seed, token ids are uniform.  Tokens are given
and not sampled back into the model, so that one close call does not change all that follows.  ``exact`` draws the
same weights itself and runs whole sequences in 64 bits, without a cache and without this package's code.
"""

from __future__ import annotations

import math
from typing import Dict, List, Sequence, Tuple

import numpy as np
import torch

F64 = torch.float64
PAGE = 16
MOST_TOKENS = 2112          # tokens of one step: a portion of 2,048 beside 64 decoded ones

LLAMA3 = dict(low=1.0, high=4.0, original=8192)
MODELS: Dict[str, dict] = {
    "tiny": dict(layers=2, dim=64, heads=4, kv_heads=2, head_dim=16, hidden=192, vocab=512, eps=1e-5, theta=1e4, factor=None, tied=False),
    "1b": dict(layers=16, dim=2048, heads=32, kv_heads=8, head_dim=64, hidden=8192, vocab=128256, eps=1e-5, theta=5e5, factor=32.0, tied=True),
    "3b": dict(layers=28, dim=3072, heads=24, kv_heads=8, head_dim=128, hidden=8192, vocab=128256, eps=1e-5, theta=5e5, factor=32.0, tied=True),
    "8b": dict(layers=32, dim=4096, heads=32, kv_heads=8, head_dim=128, hidden=14336, vocab=128256, eps=1e-5, theta=5e5, factor=8.0, tied=False),
    "bomotar": dict(layers=4, dim=2048, heads=16, kv_heads=4, head_dim=128, hidden=8192, vocab=32000, eps=1e-6, taps=4, buckets=65536,
                    mul_prev=31, mul_cur=7, residual=0.7, side=0.7, rot_dims=64, rot_base=1e6, rot_factor=4.0, rot_original=8192.0,
                    rot_fast=32.0, rot_slow=1.0),
}


def _step(name: str, model: str, precision: str = "bfloat16", decode: int = 0, shortest: int = 0, longest: int = 0, portions: int = 0,
          portion: int = 0, start: int = 0, score: bool = False, temperature: float = -1.0) -> dict:
    """One step of the engine: ``decode`` requests with contexts from ``shortest`` to ``longest`` tokens bring one token
    each, ``portions`` requests bring ``portion`` tokens (the second and later ones a few less) behind ``start`` earlier
    ones.  ``score``: logits at every token, else at each request's last.  ``temperature`` >= 0: the step's logits are
    sampled from too."""
    return dict(name=name, kind="step", model=model, precision=precision, decode=decode, shortest=shortest, longest=longest,
                portions=portions, portion=portion, start=start, score=score, temperature=temperature)


def listed() -> List[dict]:
    return [
        # the smallest call: a handful of short prompts through LLM.generate on a tiny 32-bit model (what a first try
        # and a continuous test of an application do); host work and launches decide
        dict(name="tiny_generate", kind="generate", model="tiny", precision="float32", requests=4, longest=64, new=16),
        # one user talking to a small model
        _step("1b_decode_1", "1b", decode=1, shortest=333, longest=333),
        # serving: requests that decode beside portions of newly arrived prompts, all of odd lengths, sampled
        _step("1b_mixed", "1b", decode=24, shortest=130, longest=1900, portions=2, portion=611, temperature=0.8),
        # a short chat turn on the large model: time to the first token
        _step("8b_prompt_77", "8b", portions=1, portion=77),
        # a few requests deep into long documents
        _step("3b_decode_4_long", "3b", decode=4, shortest=5003, longest=7890),
        # a long document being read: a portion behind what was read before
        _step("3b_portion_far", "3b", portions=1, portion=2000, start=5001),
        # the headline: eight requests behind prompts of 2,048 tokens
        _step("8b_decode_8", "8b", decode=8, shortest=2048, longest=2048),
        # a full batch of chats, sampled
        _step("8b_decode_64", "8b", decode=64, shortest=40, longest=600, temperature=1.0),
        # a whole prompt at once
        _step("8b_prompt_2048", "8b", portions=1, portion=2048),
        # 32-bit: scoring a text (logits at every token), and decoding, as one does to check a 16-bit deployment
        _step("1b_score_f32", "1b", "float32", portions=1, portion=300, score=True),
        _step("1b_decode_4_f32", "1b", "float32", decode=4, shortest=50, longest=700),
        # a recurrent design: a prompt and its first tokens
        dict(name="bomotar_request", kind="request", model="bomotar", precision="bfloat16", portion=601, new=4),
    ]


def _log(rng, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    u = rng.random()
    if u < 0.08:
        case = dict(kind="generate", model="tiny", precision="float32", requests=rng.randint(1, 8), longest=_log(rng, 7, 100), new=rng.randint(4, 20))
        return case
    if u < 0.16:
        return dict(kind="request", model="bomotar", precision="bfloat16", portion=_log(rng, 9, 900), new=rng.randint(1, 5))
    f32 = u < 0.28
    model = "1b" if f32 else rng.choice(["1b", "1b", "3b", "8b", "8b"])
    kind = rng.choice(["decode", "prompt"] if f32 else ["decode", "decode", "prompt", "prompt", "mixed"])
    case = _step("", model, "float32" if f32 else "bfloat16")
    del case["name"]
    if kind != "prompt":
        case["longest"] = _log(rng, 30, 900 if f32 else 7900)
        case["shortest"] = _log(rng, 9, case["longest"])
        n = _log(rng, 1, 12 if f32 else 64)
        while n > 1 and n * (case["longest"] + case["shortest"]) > 48000:
            n //= 2
        case["decode"] = n
        if n >= 16:
            case["temperature"] = rng.choice([0.0, 0.7, 1.0])
    if kind != "decode":
        case["portions"] = rng.choice([1, 1, 2])
        case["portion"] = _log(rng, 9 if f32 else 5, 290 if f32 else 2040) // case["portions"] + rng.randint(1, 9)
        if rng.random() < 0.4 and not f32 and (model != "8b" or case["portion"] < 1000):
            case["start"] = _log(rng, 40, 6000 if case["portions"] == 1 else 2500)
        case["score"] = f32
    return case


# ------------------------------------------------------------------------------------------------- shapes of a case

def _contexts(case: dict) -> List[int]:
    """How many tokens each decoding request holds before the pass."""
    n, lo, hi = case.get("decode", 0), case.get("shortest", 0), case.get("longest", 0)
    return [hi] if n == 1 else [lo + (hi - lo) * i // (n - 1) for i in range(n)]


def _portions(case: dict) -> List[int]:
    return [max(1, case["portion"] - 37 * i) for i in range(case.get("portions", 1))]


def _generate_lengths(case: dict) -> List[int]:
    """Lengths of the prompts, from one token to the longest."""
    n, hi = case["requests"], case["longest"]
    return [hi if i == n - 1 else 1 + (hi - 1) * i * i // max((n - 1) ** 2, 1) for i in range(n)]


def _ids(case: dict, seed: int) -> Dict[str, List[List[int]]]:
    """Token ids of the pass: what each request holds before, and what it brings."""
    rng = np.random.default_rng([seed, 77])
    vocab = MODELS[case["model"]]["vocab"]

    def some(n):
        return rng.integers(0, vocab, n).tolist()

    if case["kind"] == "generate":
        return {"prompts": [some(n) for n in _generate_lengths(case)]}
    if case["kind"] == "request":
        return {"prompts": [some(case["portion"])], "follow": [some(case["new"])]}
    held = _contexts(case) + [case["start"]] * case["portions"]
    brings = [1] * case["decode"] + _portions(case) if case["portions"] else [1] * case["decode"]
    return {"held": [some(n) for n in held], "brings": [some(n) for n in brings]}


def _config(case: dict, max_len: int):
    m = MODELS[case["model"]]
    if case["model"] == "bomotar":
        from torchllms_b200.models.bomotar import AttentionConfig, BomotarConfig, DeltaConfig, LayerConfig, MlpConfig, ParallelConfig, RampScaling
        hd = m["head_dim"]
        left = AttentionConfig(heads=m["heads"], kv_heads=m["kv_heads"], dim=hd, vdim=hd, scale=hd ** -0.5, conv=m["taps"], rot_dims=m["rot_dims"],
                               rot_base=m["rot_base"], scaling=RampScaling(m["rot_factor"], m["rot_original"], m["rot_fast"], m["rot_slow"]))
        right = DeltaConfig(heads=m["heads"], kv_heads=m["kv_heads"], dim=hd, vdim=hd, conv=m["taps"])
        layers = tuple(LayerConfig(ParallelConfig(left, right, m["side"], m["side"]), MlpConfig("dense", m["hidden"])) for _ in range(m["layers"]))
        return BomotarConfig("Bomotar", m["vocab"], m["dim"], m["eps"], m["residual"], buckets=m["buckets"], mul_prev=m["mul_prev"],
                             mul_cur=m["mul_cur"], layers=layers, max_seq_len=max_len)
    from torchllms_b200.models.llama_config import LlamaConfig, RopeScaling
    scaling = RopeScaling() if m["factor"] is None else RopeScaling("llama3", m["factor"], LLAMA3["low"], LLAMA3["high"], LLAMA3["original"])
    return LlamaConfig(architecture="LlamaForCausalLM", n_layers=m["layers"], dim=m["dim"], n_heads=m["heads"], n_kv_heads=m["kv_heads"],
                       head_dim=m["head_dim"], ffn_hidden=m["hidden"], vocab_size=m["vocab"], norm_eps=m["eps"], rope_theta=m["theta"],
                       rope_scaling=scaling, tie_word_embeddings=m["tied"], max_seq_len=max_len)


# ------------------------------------------------------------------------------------------------- the engine's side

def prepare(case: dict, seed: int) -> dict:
    """The loaded model with its cache and decode graphs, requests that hold their earlier tokens, and the ids to bring."""
    from torchllms_b200.engine.step import StepEntry
    from torchllms_b200.inference import LLM
    from torchllms_b200.sampling.sampler import SamplingParams
    m, ids = MODELS[case["model"]], _ids(case, seed)
    if case["kind"] == "generate":
        longest, requests, held = case["longest"] + case["new"], case["requests"], 0
        max_len = 128
    elif case["kind"] == "request":
        longest, requests, held = case["portion"] + case["new"], 1, 0
        max_len = 1024
    else:
        lengths = [len(a) + len(b) for a, b in zip(ids["held"], ids["brings"])]
        longest, requests, held = max(lengths), len(lengths), sum(lengths)
        max_len = 8192
    # the pool holds what the pass needs, and room for the throw-away requests that record the decode graphs
    token_bytes = 2 * m["layers"] * m["kv_heads"] * m["head_dim"] * (4 if case["precision"] == "float32" else 2)
    pool = max(held + 4 * PAGE * (requests + 1) + 4096, max_len)
    llm = LLM(config=_config(case, max_len), random_seed=seed, precision=case["precision"], max_len=max_len, max_bsz=requests + 1, page_size=PAGE,
              kv_memory_gb=pool * token_bytes / (1 << 30), max_num_batched_tokens=MOST_TOKENS, eos_ids=[], seed=seed)
    state = dict(case=case, llm=llm, engine=llm.engine, ids=ids)
    if case["kind"] != "step":
        llm.warmup([case["requests"] if case["kind"] == "generate" else 1], [longest])
        return state
    if case["decode"] and not case["portions"]:
        llm.warmup([case["decode"]], [longest])
    engine = llm.engine
    kept = case["decode"] + (case["portions"] if case["start"] else 0)
    handles = [engine.claim() for _ in range(kept)]
    waiting, batch, room = [(h, t) for h, t in zip(handles, ids["held"])], [], 2048
    while waiting:                       # earlier tokens, in steps of up to 2,048
        h, tokens = waiting.pop(0)
        batch.append(StepEntry(h, tokens[:room], []))
        if len(tokens) > room:
            waiting.insert(0, (h, tokens[room:]))
        room -= len(batch[-1].tokens)
        if room == 0 or not waiting:
            engine.step(batch)
            batch, room = [], 2048
    state["handles"], state["held"] = handles, [len(t) for t in ids["held"][:kept]]
    state["params"] = [SamplingParams(max(case["temperature"], 0.0), None, seed)] * requests
    state["requests"] = list(range(requests))
    return state


def run(state: dict):
    from torchllms_b200.engine.step import StepEntry
    case, engine, ids = state["case"], state["engine"], state["ids"]
    if case["kind"] == "generate":
        # generation, then the score of what was generated: the logits that each new token was chosen from
        prompts = ids["prompts"]
        results = state["llm"].generate(prompt_token_ids=prompts, max_new_tokens=case["new"], temperature=0.0, disable_tqdm=True)
        handles = [engine.claim() for _ in prompts]
        logits = engine.step([StepEntry(h, p + r.token_ids[:-1], list(range(len(p) - 1, len(p) + case["new"] - 1)))
                              for h, p, r in zip(handles, prompts, results)])
        for h in handles:
            engine.release(h)
        return {"tokens": np.asarray([r.token_ids for r in results], dtype=np.int64), "logits": logits}
    if case["kind"] == "request":
        handle = engine.claim()
        rows = [engine.step([StepEntry(handle, ids["prompts"][0])])]
        for token in ids["follow"][0]:
            rows.append(engine.step([StepEntry(handle, [token])]).clone())
        engine.release(handle)
        return {"logits": rows}
    handles, fresh = state["handles"], []
    while len(handles) + len(fresh) < len(ids["brings"]):
        fresh.append(engine.claim())
    logits = engine.step([StepEntry(h, tokens, list(range(len(tokens))) if case["score"] else None)
                          for h, tokens in zip(handles + fresh, ids["brings"])])
    out = {"logits": logits}
    if case["temperature"] >= 0.0:
        out["tokens"] = state["llm"].sampler.launch(logits, state["params"], state["requests"], state["held"] + [0] * len(fresh))
    for h, n in zip(handles, state["held"]):       # the requests go on from where they were in the next pass
        engine.cache.truncate(h, n)
    for h in fresh:
        engine.release(h)
    return out


# ------------------------------------------------------------------------------------------------- what a pass needs

def _layer_weights(m: dict) -> int:
    d, hd = m["dim"], m["head_dim"]
    if "taps" in m:
        q, kv = m["heads"] * hd, m["kv_heads"] * hd
        left = d * (q + 2 * kv) + 2 * d * q                    # q, k, v, gate, out
        right = d * (2 * kv + q) + d * m["heads"] + d * q + 2 * (d * hd + hd * q)
        return left + right + 2 * d * m["hidden"]
    return d * hd * (2 * m["heads"] + 2 * m["kv_heads"]) + 3 * d * m["hidden"]


def work(case: dict) -> dict:
    m = MODELS[case["model"]]
    size = 4 if case["precision"] == "float32" else 2
    layer, head = m["layers"] * _layer_weights(m), m["vocab"] * m["dim"]
    kv_token = 2 * m["layers"] * m["kv_heads"] * m["head_dim"] * size
    pair = 4 * m["layers"] * m["heads"] * m["head_dim"]          # flops of one query and one key, both products

    def step(held: Sequence[int], brings: Sequence[int], wanted: int) -> Tuple[float, float]:
        tokens = sum(brings)
        pairs = sum(n * h + n * (n + 1) // 2 for h, n in zip(held, brings))
        moved = (layer + head) * size + (sum(held) + tokens) * kv_token + tokens * m["dim"] * size + wanted * m["vocab"] * 4
        flops = 2.0 * layer * tokens + 2.0 * head * wanted + float(pair) * pairs
        if "taps" in m:
            # the delta rule: a matrix per head read, corrected and read again for every token; it is kept in 32 bits
            state = m["layers"] * m["heads"] * m["head_dim"] ** 2
            moved, flops = moved + 8 * state * len(brings), flops + 8.0 * state * tokens
        return float(moved), flops

    if case["kind"] == "generate":
        lengths = _generate_lengths(case)
        steps = [step([0] * len(lengths), lengths, len(lengths))]
        steps += [step([n + i for n in lengths], [1] * len(lengths), len(lengths)) for i in range(case["new"] - 1)]
        steps += [step([0] * len(lengths), [n + case["new"] - 1 for n in lengths], len(lengths) * case["new"])]
    elif case["kind"] == "request":
        steps = [step([0], [case["portion"]], 1)] + [step([case["portion"] + i], [1], 1) for i in range(case["new"])]
    else:
        held = _contexts(case) + [case["start"]] * case["portions"]
        brings = [1] * case["decode"] + (_portions(case) if case["portions"] else [])
        steps = [step(held, brings, sum(brings) if case["score"] else len(brings))]
    return {"bytes": sum(b for b, _ in steps), "flops": sum(f for _, f in steps)}


def tolerance(case: dict):
    """16-bit storage alone moves the logits of the deep models by 2 to 6 per cent (against ``exact``), those of the
    four layers of the Bomotar by 0.7; in 32 bits it is 1e-5, most of it the angles of late positions."""
    if case["precision"] == "float32":
        return {"rel": 2e-5, "max": 2e-4, "differ": 0.05}
    if case["model"] == "bomotar":
        return {"rel": 0.025, "max": 0.25, "differ": 0.25}
    return {"rel": 0.1, "max": 0.8, "differ": 0.25}


# ------------------------------------------------------------------------------------------------- the same in 64 bits

class _Drawn:
    """The random-weights mode's tensors one after the other: one generator, drawn in 32 bits, scaled, cast."""

    def __init__(self, seed: int, precision: str):
        self.device = "cuda" if torch.cuda.is_available() else "cpu"
        self.dtype = torch.float32 if precision == "float32" else torch.bfloat16
        self.gen = torch.Generator(device=self.device)
        self.gen.manual_seed(int(seed))

    def __call__(self, shape, scale: float, offset: float = 0.0) -> torch.Tensor:
        t = torch.randn(shape, generator=self.gen, device=self.device, dtype=torch.float32)
        return (t * scale if offset == 0.0 else offset + t * scale).to(self.dtype).to(F64)


def _rms(x: torch.Tensor, w: torch.Tensor, eps: float) -> torch.Tensor:
    return x / torch.sqrt(x.pow(2).mean(-1, keepdim=True) + eps) * w


def _causal(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor) -> torch.Tensor:
    """Softmax attention of one whole sequence; ``q [n, H, d]``, ``k, v [n, G, d]``."""
    n, H, d = q.shape
    per = H // k.shape[1]
    out = torch.empty(n, H, v.shape[2], dtype=F64, device=q.device)
    step = max(1, min(n, (1 << 28) // max(n, 1)))
    for h in range(H):
        kh, vh = k[:, h // per], v[:, h // per]
        for a in range(0, n, step):
            b = min(n, a + step)
            s = q[a:b, h] @ kh[:b].T * d ** -0.5
            later = torch.arange(b, device=q.device)[None, :] > torch.arange(a, b, device=q.device)[:, None]
            out[a:b, h] = torch.softmax(s.masked_fill_(later, float("-inf")), dim=-1) @ vh[:b]
    return out


def _llama_frequencies(m: dict) -> torch.Tensor:
    """Rotary frequencies with the llama3 bands, 32-bit numbers as the design has them."""
    f = 1.0 / (m["theta"] ** (torch.arange(0, m["head_dim"], 2).float() / m["head_dim"]))
    if m["factor"] is None:
        return f
    turns = LLAMA3["original"] / (2 * math.pi / f)
    s = ((turns - LLAMA3["low"]) / (LLAMA3["high"] - LLAMA3["low"])).clamp(0.0, 1.0)
    return (1 - s) * f / m["factor"] + s * f


def _llama(m: dict, drawn: _Drawn, sequences: List[List[int]], wanted: List[List[int]]) -> torch.Tensor:
    """Logits of whole sequences at the wanted places."""
    dev, d, H, G, hd, eps = drawn.device, m["dim"], m["heads"], m["kv_heads"], m["head_dim"], m["eps"]
    table = drawn((m["vocab"], d), 0.02)
    x = table[torch.tensor([t for s in sequences for t in s], device=dev)]
    if not m["tied"]:
        del table
    ends = np.cumsum([0] + [len(s) for s in sequences]).tolist()
    pos = torch.cat([torch.arange(len(s)) for s in sequences]).to(dev, F64)
    angle = pos[:, None] * _llama_frequencies(m).to(dev, F64)[None, :]
    cos, sin = torch.cos(angle)[:, None, :], torch.sin(angle)[:, None, :]

    def turned(y):
        a, b = y[..., 0::2], y[..., 1::2]
        return torch.stack([a * cos - b * sin, a * sin + b * cos], dim=-1).flatten(-2)

    for _ in range(m["layers"]):
        wq, wk, wv, wo = (drawn(s, 0.02) for s in ((H * hd, d), (G * hd, d), (G * hd, d), (d, H * hd)))
        w1, w2, w3 = (drawn(s, 0.02) for s in ((m["hidden"], d), (d, m["hidden"]), (m["hidden"], d)))
        n1, n2 = drawn((d,), 0.1, 1.0), drawn((d,), 0.1, 1.0)
        h = _rms(x, n1, eps)
        q, k, v = turned((h @ wq.T).view(-1, H, hd)), turned((h @ wk.T).view(-1, G, hd)), (h @ wv.T).view(-1, G, hd)
        o = torch.cat([_causal(q[a:b], k[a:b], v[a:b]) for a, b in zip(ends, ends[1:])])
        x = x + o.flatten(1) @ wo.T
        for a in range(0, x.shape[0], 4096):
            h = _rms(x[a:a + 4096], n2, eps)
            x[a:a + 4096] += (torch.nn.functional.silu(h @ w1.T) * (h @ w3.T)) @ w2.T
    last = drawn((d,), 0.1, 1.0)
    head = table if m["tied"] else drawn((m["vocab"], d), 0.02)
    rows = torch.tensor([ends[i] + w for i, places in enumerate(wanted) for w in places], device=dev)
    return _rms(x[rows], last, eps) @ head.T


def _bomotar_frequencies(m: dict) -> Tuple[torch.Tensor, float]:
    dims, base = m["rot_dims"], m["rot_base"]
    f = base ** (-2.0 * torch.arange(dims // 2, dtype=F64) / dims)

    def pair_of(turns):
        return dims * math.log(m["rot_original"] / (2.0 * math.pi * turns)) / (2.0 * math.log(base))

    lo, hi = max(math.floor(pair_of(m["rot_fast"])), 0), min(math.ceil(pair_of(m["rot_slow"])), dims - 1)
    ramp = ((torch.arange(dims // 2, dtype=F64) - lo) / max(hi - lo, 0.001)).clamp(0.0, 1.0)
    return f / m["rot_factor"] * ramp + f * (1.0 - ramp), 0.1 * math.log(m["rot_factor"]) + 1.0


def _conv(u: torch.Tensor, w: torch.Tensor) -> torch.Tensor:
    """Causal convolution over time, a channel at a time; the last tap is the current token's."""
    n, taps = u.shape[0], w.shape[1]
    y = torch.zeros_like(u)
    for j in range(taps):
        back = taps - 1 - j
        if back < n:
            y[back:] += u[:n - back] * w[:, j]
    return y


def _bomotar(m: dict, drawn: _Drawn, tokens: List[int], wanted: List[int]) -> torch.Tensor:
    dev, d, H, G, hd, eps, n = drawn.device, m["dim"], m["heads"], m["kv_heads"], m["head_dim"], m["eps"], len(tokens)
    matrix = lambda rows, cols: drawn((rows, cols), cols ** -0.5)  # noqa: E731
    gain = lambda size: drawn((size,), 0.1, 1.0)                   # noqa: E731
    ids = torch.tensor(tokens, device=dev)
    pairs = torch.full_like(ids, m["buckets"])
    pairs[1:] = (ids[:-1] * m["mul_prev"] + ids[1:] * m["mul_cur"]) % m["buckets"]
    x = drawn((m["vocab"], d), 1.0)[ids]
    x = x + drawn((m["buckets"] + 1, d), 0.3)[pairs]
    freq, grow = _bomotar_frequencies(m)
    angle = torch.arange(n, dtype=F64, device=dev)[:, None] * freq.to(dev)[None, :]
    cos, sin, half = grow * torch.cos(angle)[:, None, :], grow * torch.sin(angle)[:, None, :], m["rot_dims"] // 2

    def turned(y):
        u, v = y[..., :half], y[..., half:2 * half]
        return torch.cat([u * cos - v * sin, v * cos + u * sin, y[..., 2 * half:]], dim=-1)

    def unit(y):
        return y / torch.sqrt(y.pow(2).sum(-1, keepdim=True) + 1e-6)

    silu = torch.nn.functional.silu
    for _ in range(m["layers"]):
        norm1, norm1b, norm2, norm2b = gain(d), gain(d), gain(d), gain(d)
        h = _rms(x, norm1, eps)
        branch = []
        for rows in (H * hd, G * hd, G * hd):
            w = matrix(rows, d)
            branch.append(_conv(h @ w.T, drawn((rows, m["taps"]), 0.3)))
        o = _causal(turned(branch[0].view(n, H, hd)), turned(branch[1].view(n, G, hd)), branch[2].view(n, G, hd)).flatten(1)
        gate, out = matrix(H * hd, d), matrix(d, H * hd)
        left = (o * torch.sigmoid(h @ gate.T)) @ out.T
        branch = []
        for rows in (G * hd, G * hd, H * hd):
            w = matrix(rows, d)
            branch.append(silu(_conv(h @ w.T, drawn((rows, m["taps"]), 0.3))))
        beta = torch.sigmoid(h @ matrix(H, d).T)
        a_log, norm = drawn((H,), 0.3), gain(hd)
        a1, a2 = matrix(hd, d), matrix(H * hd, hd)
        # (drawn around zero, moved in 32 bits, then cast: as one tensor)
        bias = drawn((H * hd,), 1.0, -3.0)
        g1, g2, out = matrix(hd, d), matrix(H * hd, hd), matrix(d, H * hd)
        decay = torch.exp(-torch.exp(a_log)[:, None] * torch.nn.functional.softplus(h @ a1.T @ a2.T + bias).view(n, H, hd))
        q = (unit(branch[0].view(n, G, hd)) * hd ** -0.5).repeat_interleave(H // G, dim=1)
        k = unit(branch[1].view(n, G, hd)).repeat_interleave(H // G, dim=1)
        v = branch[2].view(n, H, hd)
        S, o = torch.zeros(H, hd, hd, dtype=F64, device=dev), torch.empty(n, H, hd, dtype=F64, device=dev)
        for t in range(n):
            S = decay[t][:, :, None] * S
            u = beta[t][:, None] * (v[t] - (k[t][:, None, :] @ S)[:, 0])
            S = S + k[t][:, :, None] * u[:, None, :]
            o[t] = (q[t][:, None, :] @ S)[:, 0]
        right = ((_rms(o, norm, eps)).flatten(1) * torch.sigmoid(h @ g1.T @ g2.T)) @ out.T
        x = x + m["residual"] * _rms(m["side"] * left + m["side"] * right, norm1b, eps)
        up, down = matrix(m["hidden"], d), matrix(d, m["hidden"])
        y = torch.nn.functional.gelu(_rms(x, norm2, eps) @ up.T, approximate="tanh") @ down.T
        x = x + m["residual"] * _rms(y, norm2b, eps)
    last, head = gain(d), matrix(m["vocab"], d)
    return _rms(x[torch.tensor(wanted, device=dev)], last, eps) @ head.T


@torch.no_grad()
def exact(case: dict, seed: int):
    m, ids = MODELS[case["model"]], _ids(case, seed)
    drawn = lambda: _Drawn(seed, case["precision"])  # noqa: E731
    if case["kind"] == "generate":
        seqs, n = [list(p) for p in ids["prompts"]], case["new"]
        for _ in range(n):
            best = _llama(m, drawn(), seqs, [[len(s) - 1] for s in seqs]).argmax(-1).tolist()
            seqs = [s + [t] for s, t in zip(seqs, best)]
        places = [list(range(len(s) - n - 1, len(s) - 1)) for s in seqs]
        return {"tokens": None, "logits": _llama(m, drawn(), [s[:-1] for s in seqs], places)}
    if case["kind"] == "request":
        tokens = ids["prompts"][0] + ids["follow"][0]
        logits = _bomotar(m, drawn(), tokens, list(range(case["portion"] - 1, len(tokens))))
        return {"logits": [row[None] for row in logits]}
    if sum(len(t) for t in ids["held"]) * _layer_weights(m) * m["layers"] > 2.5e14:
        return None                     # over about 20 seconds in 64 bits
    sequences = [a + b for a, b in zip(ids["held"], ids["brings"])]
    wanted = [list(range(len(a), len(s))) if case["score"] else [len(s) - 1] for a, s in zip(ids["held"], sequences)]
    out = {"logits": _llama(m, drawn(), sequences, wanted)}
    if case["temperature"] >= 0.0:
        out["tokens"] = None
    return out
