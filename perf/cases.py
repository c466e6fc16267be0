"""Workloads of this library, as a user's program runs them: steps of prompts, single decode steps and whole generations
of the served architectures, through `Engine.step`, `DecodeSession` and `Engine.generate`.

A case is a dict of plain values:

  model      a Llama shape by its name (all of its layers) or another architecture, at `width` and `layers`
  dtype      "bfloat16", or "float32": the exact engine
  do         "prefill"   prompts enter as one `Engine.step`, logits at each prompt's last token
             "pieces"    the same prompts cut into `pieces` steps, each on what the cache holds already
             "score"     one step, logits at every position
             "decode"    one token for each live sequence, through the replayed decode step
             "sample"    the same with drawn tokens (temperature, top-p, min-p, repetition penalty)
             "generate"  prompts to token ids, greedy, `new` tokens each
  sequences  how many prompts
  tokens     length of a prompt, or of the longest one where `ragged` says that they differ

Weights are the engine's seeded random ones, as `bench.py` uses them.  Feed-forwards that route tokens to experts run in
float32 only: which expert a token goes to is a comparison of scores, and where two of them nearly tie two correct bfloat16
implementations go different ways, so that no tolerance says whether their outputs agree.  For the same reason bfloat16 cases
return logits (of a decode step that is fed given tokens) and not the tokens chosen from them.
"""
from __future__ import annotations

import math

import torch

F64 = torch.float64
VOCAB = 32000
# Deviation of the random matrices.  With 0.02 a 32-layer stack of them amplifies bfloat16 rounding until two correct orders
# of summation differ by 4 % in the logits; with 0.01 it is 0.5 to 0.7 % at every Llama shape.
STD = 0.01

_LLAMA3 = dict(rope_type="llama3", low_freq_factor=1.0, high_freq_factor=4.0, original_max_position_embeddings=8192)
LLAMAS = {
    "llama-3.1-8b": dict(num_hidden_layers=32, hidden_size=4096, num_attention_heads=32, num_key_value_heads=8, head_dim=128,
                         intermediate_size=14336, vocab_size=128256, rope_theta=500000.0, rope_scaling=dict(_LLAMA3, factor=8.0),
                         tie_word_embeddings=False),
    "llama-2-7b": dict(num_hidden_layers=32, hidden_size=4096, num_attention_heads=32, num_key_value_heads=32, head_dim=128,
                       intermediate_size=11008, vocab_size=32000, rope_theta=10000.0, tie_word_embeddings=False),
    "llama-3.2-1b": dict(num_hidden_layers=16, hidden_size=2048, num_attention_heads=32, num_key_value_heads=8, head_dim=64,
                         intermediate_size=8192, vocab_size=128256, rope_theta=500000.0, rope_scaling=dict(_LLAMA3, factor=32.0),
                         tie_word_embeddings=True)}
OTHERS = ("gevonex", "fizadra", "tubusun", "degavik", "salipel")      # bfloat16; mogevik's feed-forwards are all routed
# architectures that keep fixed-size state per sequence: their sequences cannot be rewound
KEEP_STATE = ("gevonex", "mogevik", "tubusun", "degavik", "salipel")


# ---- the cases ----------------------------------------------------------------------------------------------------------
def _case(name, model, do, sequences, tokens, dtype="bfloat16", width=0, layers=0, ragged=False, pieces=1, new=0):
    c = dict(model=model, do=do, sequences=sequences, tokens=tokens, dtype=dtype, width=width, layers=layers, ragged=ragged,
             pieces=pieces, new=new)
    return dict(c, name=name) if name else c


def listed():
    return [
        # an interactive server at its ordinary load: a few conversations, one token each (`bench.py`'s default)
        _case("decode_8b_batch8", "llama-3.1-8b", "decode", 8, 512),
        # the largest call: a long prompt enters an 8B model
        _case("prefill_8b_2048", "llama-3.1-8b", "prefill", 1, 2048),
        # the smallest call: one user, a small model; launches and latency
        _case("decode_1b_single", "llama-3.2-1b", "decode", 1, 99),
        # a loaded server of a small model, tokens drawn as its users ask
        _case("sample_1b_batch64", "llama-3.2-1b", "sample", 64, 1000),
        # several users' prompts of unequal lengths arrive at once
        _case("prefill_1b_ragged", "llama-3.2-1b", "prefill", 6, 707, ragged=True),
        # full multi-head attention over long, unequal contexts: the cache weighs as much as the weights
        _case("decode_7b_ragged", "llama-2-7b", "decode", 8, 2040, ragged=True),
        # state-space, latent-attention and minGRU layers take in a prompt
        _case("prefill_gevonex", "gevonex", "prefill", 1, 2048, width=2048, layers=4),
        # latent attention and mixed scores, a token at a time
        _case("decode_fizadra_batch8", "fizadra", "decode", 8, 600, width=2048, layers=4),
        # a document enters in pieces; windowed attention beside linear attention
        _case("pieces_tubusun", "tubusun", "pieces", 1, 3001, width=2048, layers=4, pieces=2),
        # delta rule, mixed weights and retention over unequal prompts
        _case("prefill_degavik_ragged", "degavik", "prefill", 4, 801, width=2048, layers=4, ragged=True),
        # chunked and differential attention and the matrix memory with many live sequences
        _case("decode_salipel_batch32", "salipel", "decode", 32, 300, width=2048, layers=4),
        # the exact engine end to end: routed feed-forwards, prompts to tokens
        _case("generate_mogevik_float32", "mogevik", "generate", 4, 61, dtype="float32", width=1024, layers=3, ragged=True, new=8),
    ]


def _spread(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    if rng.random() < 0.15:
        return _case(None, rng.choice(["mogevik", "mogevik"] + list(OTHERS)), rng.choice(["generate", "score", "prefill"]),
                     rng.randint(1, 4), _spread(rng, 9, 160), dtype="float32", width=rng.choice([512, 768, 1024]),
                     layers=rng.randint(3, 4), ragged=True, new=rng.randint(2, 9))
    model = rng.choice(list(LLAMAS) + list(LLAMAS) + list(OTHERS))
    size = {} if model in LLAMAS else dict(width=rng.choice([1024, 1536, 2048, 3072, 4096]), layers=rng.randint(3, 5))
    most = 2048 if model in ("llama-3.1-8b", "llama-2-7b") else 6000       # tokens of all prompts together
    do = rng.choice(["prefill", "prefill", "pieces", "score", "decode", "decode", "decode", "sample"])
    sequences = _spread(rng, 1, 64 if do in ("decode", "sample") else 8)
    if do in ("decode", "sample"):
        tokens = _spread(rng, 20, max(40, min(2000, 16000 // sequences)))
    elif do == "score":
        sequences, tokens = min(sequences, 3), _spread(rng, 5, 300)
    else:
        tokens = _spread(rng, 5, most // sequences)
    return _case(None, model, do, sequences, tokens, ragged=rng.random() < 0.5 and sequences > 1,
                 pieces=rng.randint(2, 3) if do == "pieces" else 1, **size)


def _lengths(case):
    """Lengths of the prompts: all the same, or spread evenly from 1/8 of the longest to the longest, the long ones in between."""
    n, longest = case["sequences"], case["tokens"]
    if not case["ragged"] or n == 1:
        return [longest] * n
    order = sorted(range(n), key=lambda i: (i * 5 + 2) % n * n + i)
    lengths = [0] * n
    for rank, i in enumerate(order):
        lengths[i] = max(1, longest // 8 + (longest - longest // 8) * rank // (n - 1))
    return lengths


# ---- configurations: `bench.py`'s, with dense feed-forwards but for the float32 ones ------------------------------------
def config(case):
    model = case["model"]
    if model in LLAMAS:
        return dict(LLAMAS[model], architectures=["LlamaForCausalLM"], model_type="llama", rms_norm_eps=1e-5,
                    max_position_embeddings=131072 if "rope_scaling" in LLAMAS[model] else 4096)
    w, n, routed = case["width"], case["layers"], case["dtype"] == "float32"
    H = w // 128
    G = max(1, H // 4)
    spread = lambda first, span, ratio: [1.0 - first * ratio ** (h / max(1, span - 1)) for h in range(span)]  # noqa: E731
    if model == "gevonex":
        kinds = ["mamba2", "latent_attention", "mingru", "mamba2"]
        mixers = {"mamba2": dict(heads=w // 32, vdim=64, state=128, groups=1, norm_groups=1, conv=4),
                  "latent_attention": dict(heads=H, dim=128, vdim=128, kv_rank=128, scale=128 ** -0.5), "mingru": dict(width=w)}
        layers = [dict(type=kinds[i % 4], mixer=mixers[kinds[i % 4]], mlp=dict(kind="dense", ff=4 * w)) for i in range(n)]
        return dict(architecture="Gevonex", vocab=VOCAB, width=w, norm=dict(eps=1e-5), logit_softcap=30.0,
                    loop=dict(start=0, stop=n, times=1), layers=layers)
    if model == "fizadra":
        rot = dict(base=10000.0, dims=32)
        scaled = dict(rot, scaling=dict(factor=4.0, original=2048, fast=32.0, slow=1.0))
        latent = dict(heads=H, dim=96, rot_dim=32, vdim=128, kv_rank=96, q_rank=max(64, w // 256 * 64), scale=128 ** -0.5)
        kinds = ["latent_attention", "attention", "latent_attention", "latent_attention_2"]
        mixers = [dict(latent, rot=scaled),
                  dict(heads=H, kv_heads=G, dim=128, vdim=128, scale=128 ** -0.5, rot=dict(base=500000.0, dims=64)),
                  dict(latent, rot=scaled), dict(latent, rot=rot)]
        layers = [dict(type=kinds[i % 4], mixer=dict(mixers[i % 4], kv_from=i - 2) if i % 4 == 2 else mixers[i % 4],
                       mlp=dict(kind="dense", ff=4 * w)) for i in range(n)]
        return dict(architecture="Fizadra", vocab=VOCAB, width=w, norm=dict(eps=1e-5, groups=4), layers=layers)
    if model == "mogevik":
        kinds = ["rglru", "rglru", "attention"]
        mixers = {"rglru": dict(width=w, blocks=max(1, w // 256), conv=4),
                  "attention": dict(heads=H, kv_heads=G, dim=128, vdim=128, scale=128 ** -0.5, mask=dict(size=1024))}
        mlp = dict(kind="moe", expert=dict(ff=w // 2), shared=dict(ff=(2 * w // 3 + 63) // 64 * 64),
                   router=dict(experts=14, identity=2, top=4, groups=dict(count=4, keep=3)))
        return dict(architecture="Mogevik", vocab=VOCAB, width=w, norm=dict(eps=1e-5), embedding=dict(scale=float(w) ** 0.5),
                    loop=dict(start=0, stop=n, times=1), layers=[dict(type=kinds[i % 3], mixer=mixers[kinds[i % 3]], mlp=mlp) for i in range(n)])
    if model == "tubusun":
        left = dict(heads=H, kv_heads=G, dim=128, vdim=128, scale=0.09, mask=dict(size=1024), rot=dict(dims=64, base=10000.0))
        mixer = dict(left=left, right=dict(heads=H, dim=128, vdim=128, decay=spread(0.1, H, 0.01)), left_scale=0.6, right_scale=0.5)
        moe = dict(kind="moe", expert=dict(ff=w // 2, limit=7.0), router=dict(experts=16, top=4, groups=dict(count=4, keep=3)))
        return dict(architecture="Tubusun", vocab=VOCAB, width=w, norm=dict(eps=1e-6), embedding=dict(scale=1.0), logit_softcap=30.0,
                    layers=[dict(type="parallel", mixer=mixer, mlp=moe if routed and i % 2 == 0 else dict(kind="dense", ff=4 * w))
                            for i in range(n)])
    if model == "degavik":
        mixers = {"channel_delta": dict(heads=H, kv_heads=H, dim=128, vdim=128, conv=4, decay_rank=128, gate_rank=128),
                  "attention": dict(heads=H, kv_heads=G, dim=128, vdim=128, scale=0.09, softcap=30.0,
                                    mask=dict(size=1024, keep_first=4), rot=dict(dims=64, base=10000.0)),
                  "retention": dict(heads=H, dim=128, vdim=128, rot=dict(dims=128, base=10000.0), decay=spread(0.03, H, 1.0 / 60.0))}
        kinds = ["channel_delta", "attention", "retention", "channel_delta"]
        moe = dict(kind="moe", expert=dict(ff=w // 2), router=dict(experts=16, top=4), shared=dict(ff=w // 2))
        dense = dict(kind="dense", ff=(8 * w // 3 + 63) // 64 * 64)
        return dict(architecture="Degavik", vocab=VOCAB, width=w, norm=dict(eps=1e-5),
                    layers=[dict(type=kinds[i % 4], mixer=mixers[kinds[i % 4]], mlp=moe if routed and i % 2 else dense) for i in range(n)])
    assert model == "salipel", model
    rot = dict(dims=64, base=10000.0)
    far = dict(dims=64, base=500000.0, scaling=dict(factor=8.0, low=1.0, high=4.0, original=8192))
    mixers = {"attention": dict(heads=H, kv_heads=G, dim=128, vdim=128, scale=128 ** -0.5, mask=dict(size=1024)),
              "attention_2": dict(heads=H, kv_heads=G, dim=64, vdim=128, scale=64 ** -0.5, diff=0.5, softcap=50.0, rot=rot),
              "parallel": dict(left=dict(heads=H, kv_heads=G, dim=128, vdim=128, scale=128 ** -0.5,
                                         mask=dict(size=1024, keep_first=4), rot=far),
                               right=dict(heads=H, dim=128, vdim=128, gate_cap=15.0), left_scale=0.8, right_scale=0.6)}
    kinds = ["attention", "attention_2", "parallel", "attention_2"]
    moe = dict(kind="moe", expert=dict(ff=3 * w // 4), router=dict(experts=16, top=4, scale=1.0))
    dense = dict(kind="dense", ff=(8 * w // 3 + 255) // 256 * 256)
    return dict(architecture="Salipel", vocab=VOCAB, width=w, norm=dict(eps=1e-6), residual_mult=0.7,
                layers=[dict(type=kinds[i % 4], mixer=mixers[kinds[i % 4]], mlp=moe if routed and i % 2 == 0 else dense) for i in range(n)])


# ---- a user's program ----------------------------------------------------------------------------------------------------
def _tokens(case, seed):
    """The prompts, and the token that each sequence is fed in a decode step."""
    g = torch.Generator().manual_seed(int(seed) * 7919 + 17)
    vocab = LLAMAS[case["model"]]["vocab_size"] if case["model"] in LLAMAS else VOCAB
    ids = lambda n: torch.randint(0, vocab, (n,), generator=g).tolist()  # noqa: E731
    return [ids(n) for n in _lengths(case)], ids(case["sequences"])


def _admit(state):
    """New sequences take in the prompts."""
    from mdma_b200 import StepEntry
    eng = state["engine"]
    for s in state["slots"]:
        eng.release(s)
    state["slots"] = [eng.acquire() for _ in state["prompts"]]
    eng.step([StepEntry(s, p, [len(p) - 1]) for s, p in zip(state["slots"], state["prompts"])])


def prepare(case, seed):
    from mdma_b200 import Engine, SamplingParams
    prompts, fed = _tokens(case, seed)
    longest = max(len(p) for p in prompts)
    state = dict(case=case, prompts=prompts, fed=fed, slots=[])
    context, rows = longest, len(prompts)
    if case["do"] in ("decode", "sample"):
        # sequences that cannot be rewound go on to the end of their context and start anew
        context = -(-(longest + 65) // 1024) * 1024 if case["model"] in KEEP_STATE else longest + 1
    elif case["do"] == "generate":
        context = longest + case["new"]
    elif case["do"] == "score":
        rows = sum(len(p) for p in prompts)
    eng = state["engine"] = Engine(config=config(case), seed=int(seed), dtype=case["dtype"], max_batch=len(prompts),
                                   max_context=context, logit_rows=rows, init_std=STD)
    state["context"] = context
    if case["do"] == "generate":        # a server has its decode step ready
        eng.generate([p[:2] for p in prompts], max_tokens=3, stop_ids=())
    elif case["do"] in ("decode", "sample"):
        state["params"] = (SamplingParams(temperature=0.8, top_p=0.95, min_p=0.05, repetition_penalty=1.1, repetition_window=64,
                                          seed=int(seed)) if case["do"] == "sample" else SamplingParams.greedy())
        state["histories"] = prompts if case["do"] == "sample" else None
        _admit(state)
        _decode(state)
        _decode(state)
        _admit(state)
    return state


def _decode(state):
    eng, slots = state["engine"], state["slots"]
    if state["case"]["model"] in KEEP_STATE:
        if max(eng.cache.length(s) for s in slots) >= state["context"]:
            _admit(state)
            slots = state["slots"]
    else:
        for s, p in zip(slots, state["prompts"]):
            eng.cache.truncate(s, len(p))
    session = eng.decode_session()
    session.start(slots, state["fed"], params=state["params"])
    session.run(1, state["histories"])
    session.read()
    return session.logits[:len(slots)]


def run(state):
    from mdma_b200 import StepEntry
    case, eng, prompts = state["case"], state["engine"], state["prompts"]
    if case["do"] in ("decode", "sample"):
        return _decode(state)
    if case["do"] == "generate":
        outs = eng.generate(prompts, max_tokens=case["new"], stop_ids=())
        return {"tokens": torch.tensor([o.tokens for o in outs]), "logits": eng.logits[:len(prompts)]}
    slots = [eng.acquire() for _ in prompts]
    cuts = [[len(p) * k // case["pieces"] for k in range(case["pieces"] + 1)] for p in prompts]
    for k in range(case["pieces"]):
        entries = []
        for slot, prompt, at in zip(slots, prompts, cuts):
            piece = prompt[at[k]:at[k + 1]]
            want = range(len(piece)) if case["do"] == "score" else [len(piece) - 1] if k == case["pieces"] - 1 else []
            if piece:
                entries.append(StepEntry(slot, piece, want))
        logits = eng.step(entries)
    for s in slots:
        eng.release(s)
    return logits


def work(case):
    """Matrices read once (of experts, the share that the tokens use), cached rows and states read and written once, the
    logits; two operations for each matrix element and token and for each visible pair's key and value numbers."""
    from mdma_b200 import load_config
    from mdma_b200.engine.model import DecoderModel
    cfg = config(case)
    arch, typed = load_config(cfg)
    model = DecoderModel(arch.describe(typed))
    elem = 4 if case["dtype"] == "float32" else 2
    lengths = _lengths(case)
    vocab = model.spec.vocab_size
    decode = case["do"] in ("decode", "sample")
    passes = case["new"] if case["do"] == "generate" else 1
    new = len(lengths) if decode else sum(lengths)             # tokens that enter (in the first pass)
    outs = sum(lengths) if case["do"] == "score" else len(lengths)
    nbytes = flops = 0.0

    def matrices(tokens, rows):
        b = f = 0.0
        for name, ts in model.expected_tensors().items():
            if len(ts.shape) < 2 or ts.kind != "matrix":
                continue
            n = math.prod(ts.shape)
            if "embed" in name:
                if cfg.get("tie_word_embeddings") or case["model"] in ("tubusun", "mogevik"):
                    b, f = b + n * elem, f + 2.0 * n * rows
                continue
            use = seen = 1.0
            p = name.split(".")
            if len(p) > 3 and p[1] == "mlp" and p[2][0] == "e" and p[2][1:].isdigit():
                r = cfg["layers"][int(p[0][1:])]["mlp"]["router"]
                use = r["top"] / (r["experts"] + r.get("identity", 0))
                seen = 1.0 - (1.0 - use) ** tokens
            if "head" in name:
                b, f = b + n * elem, f + 2.0 * n * rows
            else:
                b, f = b + n * elem * seen, f + 2.0 * n * tokens * use
        return b, f

    for step in range(passes):
        b, f = matrices(new if step == 0 else len(lengths), outs)
        nbytes, flops = nbytes + b + 4.0 * outs * vocab, flops + f
        for run_, need in zip(model.spec.schedule, model.kv_needs()):
            if need is None:
                continue
            wide = need.n_kv_heads * need.head_dim + ((need.n_v_heads or need.n_kv_heads) * (need.v_dim or need.head_dim) if need.values else 0)
            mixer = model.blocks[run_.layer].mixer
            shapes = (mixer.attention_shapes() if hasattr(mixer, "attention_shapes") else
                      [(mixer.n_heads, mixer.n_kv_heads, mixer.head_dim)] if hasattr(mixer, "n_kv_heads") else [])
            heads = shapes[0][0] if shapes else getattr(mixer, "n_heads", need.n_kv_heads)
            limit = need.window or need.chunk or 1 << 40
            for n in lengths:
                last = n + step if step or decode else n
                nbytes += elem * wide * min(last, limit)
                pairs = (sum(min(i + 1, limit) for i in range(n)) if step == 0 and not decode else min(last + 1, limit))
                flops += 4.0 * heads * need.head_dim * pairs
        for need in model.state_needs():
            if need is not None:
                nbytes += 2.0 * math.prod(need.shape) * torch.empty((), dtype=need.dtype).element_size() * len(lengths)
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    # bfloat16: the engine is 0.3 to 1.0 % off 64 bits, by shape and depth, and the same prompts cut in other pieces (other
    # orders of summation) differ by 0.5 to 0.7 %.  float32: 2e-7 to 7e-7 off.
    if case["dtype"] == "float32":
        return {"rel": 1e-5, "max": 1e-4, "differ": 0.01}
    return {"rel": 0.03, "max": 0.3}


# ---- the same in 64 bits, plainly: whole sequences, no cache ------------------------------------------------------------
class _Weights(dict):
    """The engine's seeded tensors, as it holds them, widened when asked for."""

    def __init__(self, case, seed):
        from mdma_b200 import load_config
        from mdma_b200.engine.model import expected_tensors
        from mdma_b200.weights import random_tensor, resident_dtype
        arch, typed = load_config(config(case))
        dtype = getattr(torch, case["dtype"])
        super().__init__({name: random_tensor(name, ts, int(seed), resident_dtype(ts, torch.bfloat16, dtype), torch.device("cuda"), STD)
                          for name, ts in expected_tensors(arch.describe(typed)).items()})

    def __getitem__(self, name):
        return super().__getitem__(name).to(F64)

    def row(self, name, ids):
        return super().__getitem__(name)[torch.tensor(ids, device="cuda")].to(F64)


def _unit(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _silu(z):
    return z * torch.sigmoid(z)


def _gelu(z):
    return 0.5 * z * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (z + 0.044715 * z ** 3)))


def _softplus(z):
    return torch.log1p(torch.exp(-z.abs())) + z.clamp(min=0.0)


def _rot_of(m, kind):
    """(turn per position of every pair, factor on both parts) of a rotation; `kind`: whose way of stretching the slow pairs."""
    dims, base, s = int(m["dims"]), float(m["base"]), m.get("scaling")
    f = [base ** (-2.0 * i / dims) for i in range(dims // 2)]
    if s and kind == "ramp":
        at = lambda turns: dims * math.log(s["original"] / (2 * math.pi * turns)) / (2 * math.log(base))  # noqa: E731
        lo, hi = max(math.floor(at(s["fast"])), 0), min(math.ceil(at(s["slow"])), dims - 1)
        ramp = [min(max((i - lo) / max(hi - lo, 0.001), 0.0), 1.0) for i in range(dims // 2)]
        f = [a / s["factor"] * r + a * (1.0 - r) for a, r in zip(f, ramp)]
        return torch.tensor(f, dtype=F64, device="cuda"), 0.1 * math.log(s["factor"]) + 1.0
    if s:
        for i, a in enumerate(f):
            turns = s["original"] * a / (2.0 * math.pi)
            share = min(max((turns - s["low"]) / (s["high"] - s["low"]), 0.0), 1.0)
            f[i] = (1.0 - share) * a / s["factor"] + share * a
    return torch.tensor(f, dtype=F64, device="cuda"), 1.0


def _rotate(x, m, adjacent, kind=""):
    """x [T, heads, d] at positions 0..: pairs of neighbours, or half a turned width apart."""
    f, mag = _rot_of(m, kind)
    dims = 2 * len(f)
    a = torch.arange(len(x), dtype=F64, device="cuda")[:, None, None] * f
    c, s = torch.cos(a) * mag, torch.sin(a) * mag
    one, two = (slice(0, dims, 2), slice(1, dims, 2)) if adjacent else (slice(0, dims // 2), slice(dims // 2, dims))
    out = x.clone()
    out[..., one] = x[..., one] * c - x[..., two] * s
    out[..., two] = x[..., two] * c + x[..., one] * s
    return out


def _sees(T, window=0, keep=0, chunk=0):
    i, j = torch.arange(T, device="cuda")[:, None], torch.arange(T, device="cuda")[None, :]
    see = j <= i
    if window:
        see = see & ((i - j < window) | (j < keep))
    return see & (i // chunk == j // chunk) if chunk else see


def _attend(q, k, v, scale, see, cap=None, slopes=None, sinks=None, talk=None, mix=None):
    """q [T, H, D], k [T, G, D], v [T, G, V] -> [T, H, V]; `talk` mixes the heads' scores, `mix` their weights."""
    T, H, _ = q.shape
    out = torch.empty(T, H, v.shape[-1], dtype=F64, device="cuda")
    groups = [range(H)] if talk is not None or mix is not None else [range(h, min(h + 8, H)) for h in range(0, H, 8)]
    per = H // k.shape[1]
    i = torch.arange(T, dtype=F64, device="cuda")
    for hs in groups:
        of = torch.tensor([h // per for h in hs], device="cuda")
        here = slice(hs[0], hs[-1] + 1)
        s = torch.matmul(q[:, here].transpose(0, 1), k[:, of].permute(1, 2, 0)) * scale
        if talk is not None:
            s = torch.matmul(talk, s.flatten(1)).view_as(s)
        if cap:
            s = cap * torch.tanh(s / cap)
        if slopes is not None:
            s = s - slopes[here, None, None] * (i[:, None] - i)
        s = s.masked_fill(~see, -math.inf)
        top = s.amax(-1, keepdim=True)
        if sinks is not None:
            top = torch.maximum(top, sinks[here, None, None])
        e = torch.exp(s - top)
        e = e / (e.sum(-1, keepdim=True) + (torch.exp(sinks[here, None, None] - top) if sinks is not None else 0.0))
        if mix is not None:
            e = torch.matmul(mix, e.flatten(1)).view_as(e)
        out[:, here] = torch.matmul(e, v[:, of].transpose(0, 1)).transpose(0, 1)
    return out


def _heads(h, w, n):
    return (h @ w.T).reshape(len(h), n, -1)


def _conv(x, taps, bias=None):
    y = torch.zeros_like(x)
    for back in range(min(taps.shape[1], len(x))):
        y[back:] += x[:len(x) - back] * taps[:, taps.shape[1] - 1 - back]
    return y if bias is None else y + bias


def _linear_state(q, k, v, decay):
    """S = decay_t S + k_t v_t', o_t = S' q_t from S = 0; decay [T, H]."""
    S = torch.zeros(q.shape[1], q.shape[2], v.shape[2], dtype=F64, device="cuda")
    out = torch.empty(v.shape, dtype=F64, device="cuda")
    for t in range(len(q)):
        S = decay[t][:, None, None] * S + k[t][:, :, None] * v[t][:, None, :]
        out[t] = torch.matmul(q[t][:, None, :], S)[:, 0]
    return out


def _top(h, W, p, r, scores, choose, weigh):
    """Which experts a token goes to, and how much of each: [T, experts] of shares, zero where it does not go."""
    s = scores(h @ W[p + "router"].T)
    c = choose(s)
    groups = r.get("groups")
    if groups and groups["keep"] < groups["count"]:
        parts = c.reshape(len(c), groups["count"], -1)
        value = parts.sort(-1, descending=True).values[..., :1 if "correction" in r else 2].sum(-1)
        out = value.sort(-1, descending=True).indices[:, groups["keep"]:]
        c = parts.scatter(1, out[:, :, None].expand(-1, -1, parts.shape[-1]), -math.inf).reshape(c.shape)
    at = c.sort(-1, descending=True).indices[:, :r["top"]]
    return torch.zeros_like(s).scatter(1, at, weigh(s.gather(1, at)))


def _experts(h, share, n, of):
    out = torch.zeros_like(h)
    for e in range(n):
        rows = share[:, e] != 0
        if rows.any():
            out[rows] += share[rows, e, None] * of(h[rows], e)
    return out


def _llama(cfg, W, ids):
    H, G, D, eps = cfg["num_attention_heads"], cfg["num_key_value_heads"], cfg["head_dim"], cfg["rms_norm_eps"]
    s = cfg.get("rope_scaling")
    rot = dict(dims=D, base=cfg["rope_theta"])
    if s:
        rot["scaling"] = dict(factor=s["factor"], low=s["low_freq_factor"], high=s["high_freq_factor"],
                              original=s["original_max_position_embeddings"])
    x = W.row("model.embed_tokens.weight", ids)
    see = _sees(len(ids))
    for i in range(cfg["num_hidden_layers"]):
        w = lambda n: W[f"model.layers.{i}.{n}.weight"]  # noqa: E731, B023
        h = _unit(x, eps) * w("input_layernorm")
        q, k = _rotate(_heads(h, w("self_attn.q_proj"), H), rot, False), _rotate(_heads(h, w("self_attn.k_proj"), G), rot, False)
        a = _attend(q, k, _heads(h, w("self_attn.v_proj"), G), D ** -0.5, see)
        x = x + a.flatten(1) @ w("self_attn.o_proj").T
        h = _unit(x, eps) * w("post_attention_layernorm")
        x = x + (_silu(h @ w("mlp.gate_proj").T) * (h @ w("mlp.up_proj").T)) @ w("mlp.down_proj").T
    return _unit(x, eps) * W["model.norm.weight"], W["model.embed_tokens.weight" if cfg["tie_word_embeddings"] else "lm_head.weight"]


def _gevonex_mix(h, W, p, kind, m, eps):
    T = len(h)
    if kind == "mingru":
        z, u = torch.sigmoid(h @ W[p + "z"].T + W[p + "z.b"]), h @ W[p + "x"].T + W[p + "x.b"]
        take = z * torch.where(u >= 0, u + 0.5, torch.sigmoid(u))
        s, rows = torch.zeros_like(u[0]), []
        for t in range(T):
            s = (1.0 - z[t]) * s + take[t]
            rows.append(s)
        return (torch.stack(rows) * _silu(h @ W[p + "g"].T)) @ W[p + "o"].T
    if kind == "latent_attention":
        c = _unit(h @ W[p + "dkv"].T, eps) * W[p + "dkv.norm"]
        o = _attend(_heads(h, W[p + "q"], m["heads"]), _heads(c, W[p + "uk"], m["heads"]), _heads(c, W[p + "uv"], m["heads"]),
                    m["scale"], _sees(T), sinks=W[p + "sink"])
        return o.flatten(1) @ W[p + "o"].T
    H, V, N = m["heads"], m["vdim"], m["state"]
    inner, proj = H * V, h @ W[p + "in"].T
    z, xbc, dt = proj[:, :inner], proj[:, inner:2 * inner + 2 * N], proj[:, 2 * inner + 2 * N:]
    xbc = _silu(_conv(xbc, W[p + "conv"], W[p + "conv.b"]))
    v = xbc[:, :inner].reshape(T, H, V)
    B, C = (xbc[:, inner + N * j:inner + N * (j + 1)][:, None].expand(T, H, N) for j in (0, 1))
    dt = _softplus(dt + W[p + "dt_bias"])
    y = _linear_state(C, B * dt[:, :, None], v, torch.exp(-torch.exp(W[p + "A_log"]) * dt)) + W[p + "D"][:, None] * v
    return (_unit(y.reshape(T, inner) * _silu(z), eps) * W[p + "norm"]) @ W[p + "o"].T


def _gevonex(cfg, W, ids):
    eps = cfg["norm"]["eps"]
    norm = lambda x, n: torch.tanh(W[n + ".alpha"] * x) * W[n] + W[n + ".b"]  # noqa: E731
    x = x0 = W.row("embed", ids)
    x = torch.cat([x, x0], -1) @ W["loop.in"].T + W["loop.step"][0]
    for i, layer in enumerate(cfg["layers"]):
        p = f"l{i}."
        h = norm(x, p + "norm1")
        shifted = h + (torch.cat([torch.zeros_like(h[:1]), h[:-1]]) - h) * W[p + "shift"]
        x = x + torch.sigmoid(h @ W[p + "rg1"].T + W[p + "rg1.b"]) * _gevonex_mix(shifted, W, p + "mix.", layer["type"], layer["mixer"], eps)
        h = norm(x, p + "norm2")
        x = x + torch.sigmoid(h @ W[p + "rg2"].T + W[p + "rg2.b"]) * (_gelu(h @ W[p + "mlp.up"].T) @ W[p + "mlp.down"].T)
    return norm(x, "final.norm"), W["head"]


def _fizadra(cfg, W, ids):
    eps, T, see = cfg["norm"]["eps"], len(ids), _sees(len(ids))
    norm = lambda x, n: _unit(x.reshape(T, cfg["norm"]["groups"], -1), eps).reshape(T, -1) * W[n]  # noqa: E731
    x = W.row("embed", ids)
    history, cached = [x], {}
    for i, layer in enumerate(cfg["layers"]):
        p, q_, m = f"l{i}.", f"l{i}.mix.", layer["mixer"]
        H, h = m["heads"], norm(x, f"l{i}.norm1")
        if layer["type"] == "attention":
            heads = lambda n, k: (h @ W[q_ + n].T + W[q_ + n + ".b"]).reshape(T, k, -1)  # noqa: E731, B023
            q = _rotate(_unit(heads("q", H), eps) * W[q_ + "q.norm"], m["rot"], False)
            k = _rotate(_unit(heads("k", m["kv_heads"]), eps) * W[q_ + "k.norm"], m["rot"], False)
            o = _attend(q, k, heads("v", m["kv_heads"]), m["scale"], see, talk=W[q_ + "talk"], sinks=torch.zeros(H, dtype=F64, device="cuda"))
        else:
            first, R, D = layer["type"] == "latent_attention", m["kv_rank"], m["dim"]
            q = _heads(_unit(h @ W[q_ + "dq"].T, eps) * W[q_ + "dq.norm"], W[q_ + "uq"], H)
            q = torch.cat([q[..., :D], _rotate(q[..., D:], m["rot"], first, "ramp")], -1)
            if "kv_from" not in m:
                kv = h @ W[q_ + "dkv"].T
                cached[i] = (_unit(kv[:, :R], eps) * W[q_ + "dkv.norm"], _rotate(kv[:, None, R:], m["rot"], first, "ramp"))
            c, turned = cached[i] = cached[m.get("kv_from", i)]
            k = torch.cat([_heads(c, W[q_ + "uk"], H), turned.expand(T, H, -1)], -1)
            o = _attend(q, k, _heads(c, W[q_ + "uv"], H), m["scale"], see, sinks=W[q_ + "sink"] if first else None)
            g = torch.sigmoid(h @ W[q_ + "g"].T)
            o = o * (g.reshape(T, H, -1) if first else g[:, :, None])
        x = x + norm(o.flatten(1) @ W[q_ + "o"].T, p + "norm1b")
        y = torch.relu(norm(x, p + "norm2") @ W[p + "mlp.up"].T) ** 2 @ W[p + "mlp.down"].T
        history.append(x + norm(y, p + "norm2b"))
        x = sum(a * b for a, b in zip(W[p + "dwa"], history))
    return norm(x, "final.norm"), W["head"]


def _mogevik(cfg, W, ids):
    eps, T = cfg["norm"]["eps"], len(ids)

    def norm(x, n):
        x = x - x.mean(-1, keepdim=True)
        return _unit(x, eps) * W[n]
    gated = lambda h, p: (_silu(h @ W[p + "gate"].T) * (h @ W[p + "up"].T)) @ W[p + "down"].T  # noqa: E731
    x = W.row("embed", ids) * cfg["embedding"]["scale"] + W["loop.step"][0]
    for i, layer in enumerate(cfg["layers"]):
        p, m, f = f"l{i}.mix.", layer["mixer"], layer["mlp"]
        h = norm(x, f"l{i}.norm1")
        if layer["type"] == "rglru":
            u = _conv(h @ W[p + "x"].T + W[p + "x.b"], W[p + "conv"], W[p + "conv.b"])
            r, take = (torch.sigmoid(torch.einsum("tbn,bmn->tbm", u.reshape(T, m["blocks"], -1), W[p + n]) + W[p + n + ".b"]).reshape(T, -1)
                       for n in ("ra", "ri"))
            log_a = -8.0 * r * _softplus(W[p + "lam"])
            take = torch.sqrt(-torch.expm1(2.0 * log_a)) * take * u
            s, rows = torch.zeros_like(u[0]), []
            for t in range(T):
                s = torch.exp(log_a[t]) * s + take[t]
                rows.append(s)
            mix = torch.stack(rows) * _gelu(h @ W[p + "y"].T + W[p + "y.b"])
        else:
            q, k, v = (((h @ W[p + n].T + W[p + n + ".b"]).reshape(T, k_, -1)) for n, k_ in (("q", m["heads"]), ("k", m["kv_heads"]), ("v", m["kv_heads"])))
            slopes = torch.tensor([2.0 ** (-8.0 * (a + 1) / m["heads"]) for a in range(m["heads"])], dtype=F64, device="cuda")
            mix = _attend(q, k, v, m["scale"], _sees(T, m["mask"]["size"]), slopes=slopes).flatten(1) * torch.sigmoid(h @ W[p + "g"].T)
        ff = f"l{i}.mlp."
        r = dict(f["router"], correction=True)
        share = _top(h, W, ff, r, lambda z: torch.softmax(z, -1), lambda s: s + W[ff + "correction"],  # noqa: B023
                     lambda s: s / (s.sum(-1, keepdim=True) + 1e-20))
        y = _experts(h, share, r["experts"] + r["identity"], lambda rows, e: gated(rows, f"{ff}e{e}.") if e < r["experts"] else rows)  # noqa: B023
        x = x + mix @ W[p + "o"].T + y + torch.sigmoid(h @ W[ff + "shared.sg"].T) * gated(h, ff + "shared.")
    return norm(x, "final.norm"), W["embed"]


def _tubusun(cfg, W, ids):
    eps, T = cfg["norm"]["eps"], len(ids)
    x = W.row("embed", ids) * cfg["embedding"]["scale"]
    for i, layer in enumerate(cfg["layers"]):
        p, f = f"l{i}.", layer["mlp"]
        h = _unit(x, eps) * W[p + "norm1"]
        l, r, a, b = layer["mixer"]["left"], layer["mixer"]["right"], p + "mix.left.", p + "mix.right."
        q, k = (_unit(_rotate(_heads(h, W[a + n], c), l["rot"], True), eps) for n, c in (("q", l["heads"]), ("k", l["kv_heads"])))
        o = _attend(q, k, _heads(h, W[a + "v"], l["kv_heads"]), l["scale"], _sees(T, l["mask"]["size"]), sinks=W[a + "sink"])
        y = layer["mixer"]["left_scale"] * ((o * torch.sigmoid(h @ W[a + "g"].T)[:, :, None]).flatten(1) @ W[a + "o"].T)
        q, k, v = (_silu(_heads(h, W[b + n], r["heads"])) for n in ("q", "k", "v"))
        o = _linear_state(q, k, v, torch.tensor(r["decay"], dtype=F64, device="cuda").expand(T, -1)).flatten(1)
        o = _unit(o, eps) * W[b + "norm"] * torch.sigmoid(h @ W[b + "g"].T)
        y = y + layer["mixer"]["right_scale"] * (o @ W[b + "o"].T)
        x = x + _unit(y, eps) * W[p + "norm1b"]
        h = _unit(x, eps) * W[p + "norm2"]
        p_ = p + "mlp."
        if f["kind"] == "dense":
            z = h @ W[p_ + "up"].T + W[p_ + "up.b"]
            y = (0.5 * z * (1.0 + torch.erf(z / math.sqrt(2.0)))) @ W[p_ + "down"].T + W[p_ + "down.b"]
        else:
            def expert(rows, e):
                g, u = rows @ W[f"{p_}e{e}.gate"].T, rows @ W[f"{p_}e{e}.up"].T  # noqa: B023
                g, u = g.clamp(max=f["expert"]["limit"]), u.clamp(-f["expert"]["limit"], f["expert"]["limit"])  # noqa: B023
                return (g * torch.sigmoid(1.702 * g) * (u + 1.0)) @ W[f"{p_}e{e}.down"].T  # noqa: B023
            y = _experts(h, _top(h, W, p_, f["router"], torch.sigmoid, lambda s: s, lambda s: s), f["router"]["experts"], expert)
        x = x + _unit(y, eps) * W[p + "norm2b"]
    return _unit(x, eps) * W["final.norm"], W["embed"]


def _degavik_mix(h, W, p, kind, m, eps):
    T, H = len(h), m["heads"]
    if kind == "attention":
        q = _rotate(_unit(_heads(h, W[p + "q"], H), eps) * W[p + "q.norm"], m["rot"], True)
        k = _rotate(_unit(_heads(h, W[p + "k"], m["kv_heads"]), eps) * W[p + "k.norm"], m["rot"], True)
        o = _attend(q * W[p + "temp"][:, None], k, _heads(h, W[p + "v"], m["kv_heads"]), m["scale"],
                    _sees(T, m["mask"]["size"], m["mask"]["keep_first"]), cap=m["softcap"], mix=W[p + "talk"])
        return o.flatten(1) @ W[p + "o"].T
    if kind == "retention":
        q, k = (_rotate(_heads(h, W[p + n], H), m["rot"], False) for n in ("q", "k"))
        o = _linear_state(q, k * m["dim"] ** -0.5, _heads(h, W[p + "v"], H), torch.tensor(m["decay"], dtype=F64, device="cuda").expand(T, -1))
        return (_unit(o, eps).flatten(1) * _silu(h @ W[p + "g"].T)) @ W[p + "o"].T
    q, k, v = (_silu(_conv(h @ W[p + n].T, W[p + n + ".conv"])).reshape(T, H, -1) for n in ("q", "k", "v"))
    q, k = (a / torch.sqrt((a * a).sum(-1, keepdim=True) + 1e-6) for a in (q, k))
    q, beta = q * m["dim"] ** -0.5, torch.sigmoid(h @ W[p + "b"].T)
    step = _softplus((h @ W[p + "a1"].T) @ W[p + "a2"].T + W[p + "dt_bias"]).reshape(T, H, -1)
    keep = torch.exp(-torch.exp(W[p + "A_log"])[:, None] * step)
    S, o = torch.zeros(H, q.shape[2], v.shape[2], dtype=F64, device="cuda"), torch.empty_like(v)
    for t in range(T):
        S = keep[t][:, :, None] * S
        u = beta[t][:, None] * (v[t] - torch.matmul(k[t][:, None], S)[:, 0])
        S = S + k[t][:, :, None] * u[:, None, :]
        o[t] = torch.matmul(q[t][:, None], S)[:, 0]
    gate = torch.sigmoid((h @ W[p + "g1"].T) @ W[p + "g2"].T).reshape(T, H, -1)
    return (_unit(o, eps) * W[p + "norm"] * gate).flatten(1) @ W[p + "o"].T


def _degavik(cfg, W, ids):
    eps = cfg["norm"]["eps"]
    gated = lambda h, p: (_silu(h @ W[p + "gate"].T) * (h @ W[p + "up"].T)) @ W[p + "down"].T  # noqa: E731
    x = W.row("embed", ids)
    for i, layer in enumerate(cfg["layers"]):
        p, f, ff = f"l{i}.", layer["mlp"], f"l{i}.mlp."
        x = x + _unit(_degavik_mix(x, W, p + "mix.", layer["type"], layer["mixer"], eps), eps) * W[p + "norm1"]
        if f["kind"] == "dense":
            y = gated(x, ff)
        else:
            share = _top(x, W, ff, f["router"], lambda z: z + W[ff + "router.b"], lambda s: s, lambda s: torch.softmax(s, -1))  # noqa: B023
            y = _experts(x, share, f["router"]["experts"], lambda rows, e: gated(rows, f"{ff}e{e}.")) + gated(x, ff + "shared.")  # noqa: B023
        x = x + _unit(y, eps) * W[p + "norm2"]
    return _unit(x, eps) * W["final.norm"], W["head"]


def _salipel_mix(h, W, p, kind, m, eps):
    T = len(h)
    if kind == "parallel":
        return (m["left_scale"] * _salipel_mix(h, W, p + "left.", "left", m["left"], eps)
                + m["right_scale"] * _salipel_mix(h, W, p + "right.", "right", m["right"], eps))
    H, G = m["heads"], m.get("kv_heads", m["heads"])
    if kind == "attention":
        slopes = torch.tensor([2.0 ** (-8.0 * (a + 1) / H) for a in range(H)], dtype=F64, device="cuda")
        o = _attend(_heads(h, W[p + "q"], H), _heads(h, W[p + "k"], G), _unit(_heads(h, W[p + "v"], G), eps), m["scale"],
                    _sees(T, chunk=m["mask"]["size"]), slopes=slopes, sinks=W[p + "sink"])
        return o.flatten(1) @ W[p + "o"].T
    if kind == "attention_2":
        q = _rotate(_unit(_heads(h, W[p + "q"], 2 * H), eps) * W[p + "q.norm"], m["rot"], False)
        k = _rotate(_unit(_heads(h, W[p + "k"], 2 * G), eps) * W[p + "k.norm"], m["rot"], False)
        one, two = (_attend(q[:, j::2], k[:, j::2], _heads(h, W[p + "v"], G), m["scale"], _sees(T), cap=m["softcap"]) for j in (0, 1))
        lam = torch.exp(W[p + "lq1"] @ W[p + "lk1"]) - torch.exp(W[p + "lq2"] @ W[p + "lk2"]) + m["diff"]
        o = _unit(one - lam * two, eps) * (1.0 - m["diff"])
        return (o.flatten(1) * torch.sigmoid(h @ W[p + "g"].T)) @ W[p + "o"].T
    if kind == "left":
        raw = _heads(h, W[p + "k"], G)
        q = _rotate(_unit(_heads(h, W[p + "q"], H), eps) * W[p + "q.norm"], m["rot"], False)
        k = _rotate(_unit(raw, eps) * W[p + "k.norm"], m["rot"], False)
        o = _attend(q, k, raw, m["scale"], _sees(T, m["mask"]["size"], m["mask"]["keep_first"]))
        return (o.flatten(1) * torch.sigmoid(h @ W[p + "g"].T)) @ W[p + "o"].T
    q, k, v = _heads(h, W[p + "q"], H) * m["dim"] ** -0.5, _heads(h, W[p + "k"], H), _heads(h, W[p + "v"], H)
    soft = lambda n: m["gate_cap"] * torch.tanh((h @ W[p + n].T + W[p + n + ".b"]) / m["gate_cap"])  # noqa: E731
    li, lf = soft("i"), -_softplus(-soft("f"))
    S, n = torch.zeros(H, m["dim"], v.shape[-1], dtype=F64, device="cuda"), torch.zeros(H, m["dim"], dtype=F64, device="cuda")
    top, o = torch.zeros(H, dtype=F64, device="cuda"), torch.empty_like(v)
    for t in range(T):
        new = torch.maximum(lf[t] + top, li[t])
        keep, take = torch.exp(lf[t] + top - new), torch.exp(li[t] - new)
        S = keep[:, None, None] * S + (take[:, None] * k[t])[:, :, None] * v[t][:, None, :]
        n, top = keep[:, None] * n + take[:, None] * k[t], new
        o[t] = torch.matmul(q[t][:, None], S)[:, 0] / (torch.maximum((n * q[t]).sum(-1).abs(), torch.exp(-top)) + 1e-6)[:, None]
    return (_unit(o, eps).flatten(1) * W[p + "norm"] * torch.sigmoid(h @ W[p + "g"].T)) @ W[p + "o"].T


def _salipel(cfg, W, ids):
    eps = cfg["norm"]["eps"]
    x = W.row("embed", ids)
    for i, layer in enumerate(cfg["layers"]):
        p, f, ff = f"l{i}.", layer["mlp"], f"l{i}.mlp."
        h = _unit(x, eps) * W[p + "norm1"]
        y = _salipel_mix(h, W, p + "mix.", layer["type"], layer["mixer"], eps)
        if f["kind"] == "dense":
            y = y + (_gelu(h @ W[ff + "gate"].T) * (h @ W[ff + "up"].T)) @ W[ff + "down"].T
        else:
            r = f["router"]
            share = _top(h, W, ff, r, lambda z: torch.softmax(z, -1), lambda s: s + W[ff + "correction"],  # noqa: B023
                         lambda s: s / (s.sum(-1, keepdim=True) + 1e-20) * r["scale"])  # noqa: B023
            y = y + _experts(h, share, r["experts"], lambda rows, e: torch.relu(rows @ W[f"{ff}e{e}.up"].T) ** 2 @ W[f"{ff}e{e}.down"].T)  # noqa: B023
        x = x + cfg["residual_mult"] * y
    return _unit(x, eps) * W["final.norm"], W["head"]


def exact(case, seed):
    cfg, W = config(case), _Weights(case, seed)
    plain = _llama if case["model"] in LLAMAS else globals()["_" + case["model"]]
    prompts, fed = _tokens(case, seed)

    def logits(ids, every=False):
        h, head = plain(cfg, W, ids)
        z = (h if every else h[-1:]) @ head.T
        cap = cfg.get("logit_softcap")
        return cap * torch.tanh(z / cap) if cap else z
    if case["do"] == "generate":
        rows = []
        for p in prompts:
            ids = list(p)
            for _ in range(case["new"]):
                z = logits(ids)
                ids.append(int(z[0].argmax()))
            rows.append(z)
        return {"tokens": None, "logits": torch.cat(rows)}
    if case["do"] in ("decode", "sample"):
        prompts = [p + [t] for p, t in zip(prompts, fed)]
    return torch.cat([logits(p, case["do"] == "score") for p in prompts])
