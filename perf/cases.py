"""What is timed: the steps, sessions and sampling calls that programs make with this library.

A case is a dict of plain values.  ``kind`` says what one pass is:

* ``decode``: one new token for each of ``batch`` sequences that hold ``low`` to ``high`` tokens (``LlogosModel.step``); the
  sequences are then rolled back by that token (``truncate``), so a pass can be made again.
* ``prompt``: ``batch`` new sequences of ``low`` to ``high`` tokens in one step, logits of every sequence's last token (or of all
  tokens: ``every``), sequences closed again.
* ``append``: ``batch`` sequences of ``low`` to ``high`` tokens that each bring ``new`` more in one step, rolled back afterwards.
* ``session``: ``batch`` prompts of ``low`` to ``high`` tokens in one step, then ``steps`` decode steps over given tokens, the logits
  of all of them, sequences closed again: what generation does, without the draw of the next token.
* ``sample``: one token for each of ``batch`` rows of logits, with the library's default filters and penalties.

Sequence lengths are spread between ``low`` and ``high`` by the case's own numbers; weights, tokens and logits come from the seed.
``exact`` is the same arithmetic in plain torch float64 on whole sequences, one function per design.
"""
import math
import random

import torch

# ---- the models -----------------------------------------------------------------------------------

LLAMA3 = {"rope_type": "llama3", "factor": 8.0, "low_freq_factor": 1.0, "high_freq_factor": 4.0, "original_max_position_embeddings": 8192}
DENSE = {
    "llama-3.1-8b": {"architectures": ["LlamaForCausalLM"], "num_hidden_layers": 32, "hidden_size": 4096, "num_attention_heads": 32,
                     "num_key_value_heads": 8, "head_dim": 128, "intermediate_size": 14336, "vocab_size": 128256,
                     "rope_theta": 500000.0, "rms_norm_eps": 1e-5, "max_position_embeddings": 131072, "rope_scaling": LLAMA3},
    "qwen3-8b": {"architectures": ["Qwen3ForCausalLM"], "num_hidden_layers": 36, "hidden_size": 4096, "num_attention_heads": 32,
                 "num_key_value_heads": 8, "head_dim": 128, "intermediate_size": 12288, "vocab_size": 151936,
                 "rope_theta": 1000000.0, "rms_norm_eps": 1e-6, "max_position_embeddings": 40960},
    "qwen2.5-14b": {"architectures": ["Qwen2ForCausalLM"], "num_hidden_layers": 48, "hidden_size": 5120, "num_attention_heads": 40,
                    "num_key_value_heads": 8, "head_dim": 128, "intermediate_size": 13824, "vocab_size": 152064,
                    "rope_theta": 1000000.0, "rms_norm_eps": 1e-6, "max_position_embeddings": 131072},
    "llama-3.2-1b": {"architectures": ["LlamaForCausalLM"], "num_hidden_layers": 16, "hidden_size": 2048, "num_attention_heads": 32,
                     "num_key_value_heads": 8, "head_dim": 64, "intermediate_size": 8192, "vocab_size": 128256,
                     "rope_theta": 500000.0, "rms_norm_eps": 1e-5, "max_position_embeddings": 131072, "tie_word_embeddings": True,
                     "rope_scaling": dict(LLAMA3, factor=32.0)},
}
# sizes of the other designs: width, heads, key/value heads, head size, feed-forward size, window
SIZES = {"1b-like": (2048, 32, 8, 64, 8192, 1024), "8b-like": (4096, 32, 8, 128, 14336, 2048)}
VOCAB, EXPERTS, TOP = 32000, 16, 4


def karitar(size):
    width, heads, kv, hd, ff, window = SIZES[size]
    att = {"heads": heads, "kv_heads": kv, "dim": hd, "vdim": hd, "scale": hd ** -0.5, "mask": {"size": window}}
    return {"architecture": "Karitar", "vocab": VOCAB, "width": width, "norm": {"eps": 1e-5}, "streams": 2,
            "layers": [{"type": "attention", "mixer": dict(att), "mlp": {"kind": "dense", "ff": ff}} for _ in range(4)]}


def piratar(size):
    width, heads, kv, hd, ff, _ = SIZES[size]
    rot = {"base": 1000000.0, "dims": hd}
    left = {"heads": heads, "kv_heads": kv, "dim": hd, "vdim": hd, "scale": hd ** -0.5, "conv": 4, "rot": dict(rot)}
    right = {"heads": heads // 4, "dim": hd, "vdim": hd, "decay": [1.0 - 2.0 ** -(5 + i % 6) for i in range(heads // 4)], "rot": dict(rot)}
    both = ("parallel", {"left": left, "right": right})
    return {"architecture": "Piratar", "vocab": VOCAB, "width": width, "norm": {"eps": 1e-6},
            "embedding": {"scale": float(width) ** 0.5, "bigram": {"buckets": 100003, "mul_prev": 1009, "mul_cur": 101}},
            "token_side": {"dim": 64},
            "layers": [{"type": t, "mixer": m, "mlp": {"kind": "dense", "ff": ff}}
                       for t, m in (both, ("rglru", {"width": width, "blocks": 16, "conv": 4}), both, both)]}


def penasun(size):
    width, heads, kv, hd, ff, _ = SIZES[size]
    ssm = {"heads": 2 * width // 64, "vdim": 64, "state": 128, "groups": 8, "conv": 4, "norm_groups": 8}
    att = {"heads": heads, "kv_heads": kv, "dim": hd // 2, "vdim": hd, "scale": (hd // 2) ** -0.5, "diff": 0.5,
           "q_temp": {"coef": 0.1, "every": 4096}}
    mlp = {"kind": "moe", "router": {"experts": EXPERTS, "top": TOP, "identity": 4, "scale": 2.5, "groups": {"count": 4, "keep": 2}},
           "expert": {"ff": ff // 8, "limit": 7.0}}
    return {"architecture": "Penasun", "vocab": VOCAB, "width": width, "norm": {"eps": 1e-5},
            "layers": [{"type": t, "mixer": dict(m), "mlp": mlp} for t, m in (("mamba2", ssm), ("attention", att)) * 2]}


DESIGNS = {"karitar": karitar, "penasun": penasun, "piratar": piratar}


def config_of(case):
    if case["model"] in DENSE:
        return dict(DENSE[case["model"]], num_hidden_layers=case["layers"])
    return DESIGNS[case["model"]](case["size"])


def vocab_of(cfg):
    return cfg["vocab_size"] if "vocab_size" in cfg else cfg["vocab"]


# ---- the cases ------------------------------------------------------------------------------------

def listed():
    return [
        # the next token of a single chat with a small model: latency is what its user waits for
        {"name": "decode_1b_one", "kind": "decode", "model": "llama-3.2-1b", "layers": 16, "dtype": "bfloat16",
         "batch": 1, "low": 611, "high": 611},
        # the workload that the library's numbers are quoted on: eight sequences at a context of 8,192
        {"name": "decode_8b_eight_long", "kind": "decode", "model": "llama-3.1-8b", "layers": 32, "dtype": "bfloat16",
         "batch": 8, "low": 8190, "high": 8190},
        # a server's full batch of requests of unequal lengths
        {"name": "decode_8b_ragged_64", "kind": "decode", "model": "llama-3.1-8b", "layers": 32, "dtype": "bfloat16",
         "batch": 64, "low": 128, "high": 2048},
        # a document's prompt: the quoted prompt workload
        {"name": "prompt_8b_2048", "kind": "prompt", "model": "llama-3.1-8b", "layers": 32, "dtype": "bfloat16",
         "batch": 1, "low": 2048, "high": 2048, "every": False},
        # scoring a handful of short texts: logits of every token, odd lengths
        {"name": "prompt_1b_short", "kind": "prompt", "model": "llama-3.2-1b", "layers": 16, "dtype": "bfloat16",
         "batch": 5, "low": 3, "high": 90, "every": True},
        # long ragged prompts of a larger model (some of its layers): the largest step
        {"name": "prompt_14b_long", "kind": "prompt", "model": "qwen2.5-14b", "layers": 8, "dtype": "bfloat16",
         "batch": 6, "low": 256, "high": 8192, "every": False},
        # the next turns of four running chats: a few hundred tokens behind thousands that the cache holds
        {"name": "append_8b_turns", "kind": "append", "model": "qwen3-8b", "layers": 12, "dtype": "bfloat16",
         "batch": 4, "low": 1000, "high": 4000, "new": 83},
        # the 32-bit path, which answers are checked against: short prompts and decoding
        {"name": "session_1b_float32", "kind": "session", "model": "llama-3.2-1b", "layers": 16, "dtype": "float32",
         "batch": 3, "low": 7, "high": 96, "steps": 8},
        # drawing the next tokens of a batch with the default filters and penalties
        {"name": "sample_8", "kind": "sample", "vocab": 128256, "batch": 8},
        # prompts and decoding of models with other mixers, residuals and feed-forwards
        {"name": "session_karitar", "kind": "session", "model": "karitar", "size": "8b-like", "dtype": "bfloat16",
         "batch": 8, "low": 64, "high": 700, "steps": 12},
        {"name": "session_piratar", "kind": "session", "model": "piratar", "size": "1b-like", "dtype": "bfloat16",
         "batch": 4, "low": 300, "high": 1500, "steps": 12},
        {"name": "session_penasun", "kind": "session", "model": "penasun", "size": "1b-like", "dtype": "bfloat16",
         "batch": 8, "low": 100, "high": 1000, "steps": 12},
    ]


def _log(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(("decode", "decode", "prompt", "prompt", "append", "float32", "sample", "design", "design"))
    if kind == "sample":
        return {"kind": "sample", "vocab": rng.choice((32000, 128256, 151936, 152064)), "batch": _log(rng, 1, 64)}
    if kind == "design":
        model, size = rng.choice(sorted(DESIGNS)), rng.choice(sorted(SIZES))
        batch = _log(rng, 1, 12) if model != "penasun" else rng.randint(6, 12)
        high = _log(rng, 20, min(3000, 6000 // batch))
        return {"kind": "session", "model": model, "size": size, "dtype": "bfloat16", "batch": batch,
                "low": max(3, _log(rng, max(3, high // 10), high)), "high": high, "steps": rng.randint(4, 16)}
    if kind == "float32":
        high = _log(rng, 8, 160)
        return {"kind": "session", "model": "llama-3.2-1b", "layers": rng.randint(2, 16), "dtype": "float32",
                "batch": _log(rng, 1, 6), "low": rng.randint(3, high), "high": high, "steps": rng.randint(2, 12)}
    model = rng.choice(sorted(DENSE))
    case = {"kind": kind, "model": model, "layers": rng.randint(4, 8) if model == "qwen2.5-14b" else rng.randint(4, 16), "dtype": "bfloat16"}
    if kind == "decode":
        batch = _log(rng, 1, 64)
        high = _log(rng, 40, min(8190, 48000 // batch))
        case.update(batch=batch, low=_log(rng, max(20, high // 16), high), high=high)
    elif kind == "prompt":
        batch = _log(rng, 1, 8)
        high = _log(rng, 20, min(8192, 16000 // batch))
        case.update(batch=batch, low=_log(rng, max(3, high // 16), high), high=high, every=False)
    else:
        batch = _log(rng, 1, 8)
        high = _log(rng, 200, min(6000, 20000 // batch))
        case.update(batch=batch, low=_log(rng, max(50, high // 8), high), high=high, new=_log(rng, 2, 400))
    return case


def lengths_of(case):
    """The sequences' tokens ahead of the pass (of a prompt: in it): spread over low..high by the case's own numbers."""
    r = random.Random(1000003 * case["batch"] + 1009 * case["low"] + case["high"])
    return [r.randint(case["low"], case["high"]) for _ in range(case["batch"])]


# ---- what a program has in hand, and a pass -------------------------------------------------------

class State:
    pass


def _tokens(seed, counts, vocab):
    g = torch.Generator().manual_seed(seed)
    return [torch.randint(0, vocab, (n,), generator=g).tolist() for n in counts]


def _given(case, seed):
    """(tokens of every sequence ahead of the pass's own, tokens that the pass brings behind them)."""
    lens, vocab = lengths_of(case), vocab_of(config_of(case))
    more = {"decode": 1, "prompt": 0, "append": case.get("new"), "session": case.get("steps")}[case["kind"]]
    toks = _tokens(seed, [n + more for n in lens], vocab)
    return [t[:n] for t, n in zip(toks, lens)], [t[n:] for t, n in zip(toks, lens)]


def prepare(case, seed):
    import llogos_b200 as llogos
    st = State()
    st.case = case
    if case["kind"] == "sample":
        b, v = case["batch"], case["vocab"]
        g = torch.Generator(device="cuda").manual_seed(seed)
        st.sampler = llogos.LlogosModel.random(dict(DENSE["llama-3.2-1b"], num_hidden_layers=1, hidden_size=64, num_attention_heads=2,
                                                    num_key_value_heads=1, head_dim=32, intermediate_size=64, vocab_size=v),
                                               seed, max_context=64, max_batch=b).sampler
        st.logits = torch.randn(b, v, device="cuda", generator=g) * 2.5      # a trained model's logits: a few stand out
        st.params = llogos.GenerationParams(seed=seed)
        st.sampler.begin(_tokens(seed, [40 + 9 * i for i in range(b)], v), st.params)
        st.rows, st.drawn = list(range(b)), 0
        return st
    cfg = config_of(case)
    st.before, st.brings = _given(case, seed)
    longest = max(len(a) + len(b) for a, b in zip(st.before, st.brings))
    st.model = llogos.LlogosModel.random(cfg, seed, dtype=case["dtype"], std=0.02, norm_std=0.1,
                                         max_context=(longest + 63) // 64 * 64, max_batch=case["batch"])
    if case["kind"] in ("decode", "append"):
        st.slots = []
        for toks in st.before:
            st.slots.append(st.model.open())
            st.model.step([(st.slots[-1], toks)], want=[[]])
    if case["kind"] == "prompt":
        st.want = [list(range(len(t))) if case["every"] else [len(t) - 1] for t in st.before]
    if case["kind"] == "session":
        st.logits = torch.empty(case["steps"] + 1, case["batch"], vocab_of(cfg), device="cuda")
    return st


def run(st):
    kind = st.case["kind"]
    if kind == "sample":
        st.drawn += 1
        return st.sampler.sample_device(st.logits, st.params, seed=st.params.seed, step=st.drawn, seq_ids=st.rows, ring_rows=st.rows)
    m = st.model
    if kind in ("decode", "append"):
        logits = m.step(list(zip(st.slots, st.brings)))
        for slot, toks in zip(st.slots, st.before):
            m.truncate(slot, len(toks))
        return logits
    slots = [m.open() for _ in st.before]
    if kind == "prompt":
        out = m.step(list(zip(slots, st.before)), st.want)
    else:
        out = st.logits                                          # a step's logits are valid until the next step
        out[0].copy_(m.step(list(zip(slots, st.before))))
        for k in range(st.case["steps"]):
            out[k + 1].copy_(m.step([(s, t[k:k + 1]) for s, t in zip(slots, st.brings)]))
    for s in slots:
        m.close(s)
    return out


# ---- what a pass cannot do without ----------------------------------------------------------------

def _pairs(counts, before, window):
    """(query, key) pairs that a causal step scores, and the cached keys that it reads."""
    pairs = rows = 0
    for c, b in zip(counts, before):
        w = window or b + c
        if b + c <= w:
            pairs += c * b + c * (c + 1) // 2
        else:
            pairs += sum(min(b + i + 1, w) for i in range(c))
        rows += min(b, w)
    return pairs, rows


def _step_work(case, cfg, counts, before, wanted):
    """(bytes, flops) of one step: every matrix a token uses read once, cached keys and values read, new ones written, logits
    written; products, attention, and the recurrences' updates."""
    e = 2 if case["dtype"] == "bfloat16" else 4
    n, v = sum(counts), vocab_of(cfg)
    if "vocab_size" in cfg:
        h, hd, nh, kv = cfg["hidden_size"], cfg["head_dim"], cfg["num_attention_heads"], cfg["num_key_value_heads"]
        layers = cfg["num_hidden_layers"]
        mats = layers * (h * hd * (nh + 2 * kv) + nh * hd * h + 3 * h * cfg["intermediate_size"])
        pairs, rows = _pairs(counts, before, 0)
        moved = (mats + v * h) * e + layers * 2 * kv * hd * e * (rows + n) + 4 * wanted * v + n * h * e
        return moved, 2.0 * n * mats + 2.0 * wanted * v * h + 4.0 * layers * nh * hd * pairs
    d = cfg["width"]
    moved, flops = v * d * e + 4.0 * wanted * v + n * d * e, 2.0 * wanted * v * d
    seqs = len(counts)
    for lay in cfg["layers"]:
        ml, mixers = lay["mlp"], [(lay["type"], lay["mixer"])]
        if ml["kind"] == "moe":
            experts, identity, expert = ml["router"]["experts"], ml["router"]["identity"], 3 * d * ml["expert"]["ff"]
            share = TOP * experts / (experts + identity)                                     # of a token's choices, those with matrices
            moved += e * (min(experts, int(n * share)) * expert + d * (experts + identity))
            flops += 2.0 * n * (share * expert + d * (experts + identity))
        else:
            mats = (2 if cfg["architecture"] == "Karitar" else 3) * d * ml["ff"]
            moved, flops = moved + e * mats, flops + 2.0 * n * mats
        if lay["type"] == "parallel":
            mixers = [("attention", lay["mixer"]["left"]), ("retention", lay["mixer"]["right"])]
        for kind, mx in mixers:
            state = 0
            if kind == "attention":
                nh, maps = mx["heads"], 2 if "diff" in mx else 1
                row, gate = mx["kv_heads"] * (maps * mx["dim"] + mx["vdim"]), nh * mx["vdim"] if "conv" in mx else nh
                mats = d * (nh * maps * mx["dim"] + row + (0 if "diff" in mx else gate)) + nh * mx["vdim"] * d
                pairs, rows = _pairs(counts, before, mx.get("mask", {}).get("size", 0))
                moved += e * row * (rows + n)
                flops += 2.0 * nh * maps * (mx["dim"] + mx["vdim"]) * pairs
            elif kind == "retention":
                mats, state = 2 * d * mx["heads"] * (mx["dim"] + mx["vdim"]) + mx["heads"] * mx["vdim"] * d, mx["heads"] * mx["dim"] * mx["vdim"]
            elif kind == "rglru":
                mats, state = 3 * d * mx["width"] + 2 * mx["width"] ** 2 // mx["blocks"], mx["width"]
            else:
                mats = d * (2 * mx["heads"] * mx["vdim"] + 2 * mx["groups"] * mx["state"] + mx["heads"]) + mx["heads"] * mx["vdim"] * d
                state = mx["heads"] * mx["state"] * mx["vdim"]
            moved += e * mats + 2 * 4 * seqs * state
            flops += 2.0 * n * mats + 4.0 * n * state
    return moved, flops


def work(case):
    if case["kind"] == "sample":
        return {"bytes": 4.0 * case["batch"] * case["vocab"], "flops": 0.0}
    cfg, lens = config_of(case), lengths_of(case)
    b = len(lens)
    if case["kind"] == "decode":
        moved, flops = _step_work(case, cfg, [1] * b, lens, b)
    elif case["kind"] == "append":
        moved, flops = _step_work(case, cfg, [case["new"]] * b, lens, b)
    else:
        moved, flops = _step_work(case, cfg, lens, [0] * b, sum(lens) if case.get("every") else b)
        for k in range(case.get("steps", 0)):
            x, y = _step_work(case, cfg, [1] * b, [n + k for n in lens], b)
            moved, flops = moved + x, flops + y
    return {"bytes": float(moved), "flops": float(flops)}


def tolerance(case):
    if case["kind"] == "sample":
        return "exact"
    if case["dtype"] == "float32":
        return {"rel": 3e-5}      # sums of 2,048 to 8,192 float32 products in another order, through all layers
    # bfloat16 operands; of two correct runs of a model with a mixture, a token takes another last expert in one now and then
    return {"rel": 0.03, "max": 0.95 if case["model"] == "penasun" else 0.4}


# ---- the same in float64 --------------------------------------------------------------------------

F64 = torch.float64
_M = (1 << 64) - 1


def _signed(x):
    x &= _M
    return x - (1 << 64) if x >> 63 else x


def _mix(x):
    x = (x + 0x9E3779B97F4A7C15) & _M
    x = ((x ^ (x >> 30)) * 0xBF58476D1CE4E5B9) & _M
    x = ((x ^ (x >> 27)) * 0x94D049BB133111EB) & _M
    return x ^ (x >> 31)


def _mix_tensor(x):
    low = lambda y, k: (y >> k) & ((1 << (64 - k)) - 1)      # noqa: E731  (a shift that brings in zeros)
    x = x + _signed(0x9E3779B97F4A7C15)
    x = (x ^ low(x, 30)) * _signed(0xBF58476D1CE4E5B9)
    x = (x ^ low(x, 27)) * _signed(0x94D049BB133111EB)
    return x ^ low(x, 31)


class Weights:
    """The random weights by name, as the library's random models hold them: element i of a tensor is Box-Muller of two
    splitmix64 numbers of (seed, name, i), rounded to bfloat16."""

    def __init__(self, seed, device):
        self.seed, self.device = seed, device

    def __call__(self, name, *shape, mean=0.0, std=0.02):
        h = 0xCBF29CE484222325
        for byte in name.encode():
            h = ((h ^ byte) * 0x100000001B3) & _M
        key, n = _signed(_mix(_mix(self.seed & _M) ^ h)), math.prod(shape)
        out = torch.empty(n, dtype=torch.bfloat16, device=self.device)
        for lo in range(0, n, 1 << 26):
            i = torch.arange(lo, min(n, lo + (1 << 26)), device=self.device) * 2 + key
            a, b = _mix_tensor(i), _mix_tensor(i + 1)
            u = ((((a >> 11) & ((1 << 53) - 1)) + 1).to(F64)) * 2.0 ** -53
            v = (((b >> 11) & ((1 << 53) - 1)).to(F64)) * 2.0 ** -53
            z = torch.sqrt(-2.0 * torch.log(u)) * torch.cos(2.0 * math.pi * v)
            out[lo:lo + (1 << 26)] = (mean + std * z).float().bfloat16()
        return out.view(shape).to(F64)

    def norm(self, name, *shape):
        return self(name, *shape, mean=1.0, std=0.1)


def _unit(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _silu(x):
    return x * torch.sigmoid(x)


def _turn(x, freqs, neighbours=False):
    """x: [T, heads, d]; the first 2 len(freqs) elements of every head are rotated, halves or neighbouring elements."""
    half = len(freqs)
    ang = torch.arange(x.shape[0], dtype=F64, device=x.device)[:, None] * torch.tensor(freqs, dtype=F64, device=x.device)
    c, s = torch.cos(ang)[:, None], torch.sin(ang)[:, None]
    y = x.clone()
    one, two = (slice(0, 2 * half, 2), slice(1, 2 * half, 2)) if neighbours else (slice(0, half), slice(half, 2 * half))
    y[..., one] = x[..., one] * c - x[..., two] * s
    y[..., two] = x[..., two] * c + x[..., one] * s
    return y


def _powers(base, dims):
    return [base ** (-2.0 * i / dims) for i in range(dims // 2)]


def _attend(q, k, v, scale, sees=None, sink=None, mix=None):
    """Causal softmax attention.  q: [T, heads, d], k, v: [T, kv heads, .]; ``sees(i, j)``: which earlier keys; ``sink``: one more
    summand per head in the denominator; ``mix``: what becomes of all heads' scores ahead of the softmax."""
    t, heads = q.shape[:2]
    rep = heads // k.shape[1]
    out = torch.empty(t, heads, v.shape[2], dtype=F64, device=q.device)
    kk, vv = k.repeat_interleave(rep, 1).transpose(0, 1), v.repeat_interleave(rep, 1).transpose(0, 1)
    block = max(16, (1 << 27) // (t * heads))
    j = torch.arange(t, device=q.device)[None]
    for lo in range(0, t, block):
        i = torch.arange(lo, min(t, lo + block), device=q.device)[:, None]
        s = q[lo:lo + block].transpose(0, 1) @ kk.transpose(1, 2) * scale
        s = s if mix is None else mix(s)
        s = s.masked_fill(~((j <= i) & (sees(i, j) if sees else True)), -math.inf)
        m = s.amax(-1, keepdim=True)
        if sink is not None:
            m = torch.maximum(m, sink[:, None, None])
        e = torch.exp(s - m)
        z = e.sum(-1, keepdim=True)
        if sink is not None:
            z = z + torch.exp(sink[:, None, None] - m)
        out[lo:lo + block] = ((e / z) @ vv).transpose(0, 1)
    return out


def _llama3(freqs, sc):
    out = []
    for f in freqs:
        wave, orig = 2.0 * math.pi / f, sc["original_max_position_embeddings"]
        if wave > orig / sc["low_freq_factor"]:
            f = f / sc["factor"]
        elif wave >= orig / sc["high_freq_factor"]:
            s = (orig / wave - sc["low_freq_factor"]) / (sc["high_freq_factor"] - sc["low_freq_factor"])
            f = (1.0 - s) * f / sc["factor"] + s * f
        out.append(f)
    return out


def _dense(cfg, w, seqs, rows):
    """Logits of ``rows[i]`` of every sequence, the sequences side by side through each layer (its weights are made once)."""
    h, hd, nh, kv, ff = (cfg[k] for k in ("hidden_size", "head_dim", "num_attention_heads", "num_key_value_heads", "intermediate_size"))
    eps, arch = cfg["rms_norm_eps"], cfg["architectures"][0]
    freqs = _powers(cfg["rope_theta"], hd)
    freqs = _llama3(freqs, cfg["rope_scaling"]) if "rope_scaling" in cfg else freqs
    cuts = [len(s) for s in seqs]
    emb = w("model.embed_tokens.weight", cfg["vocab_size"], h)
    x = emb[torch.tensor([t for s in seqs for t in s], device=w.device)]
    if not cfg.get("tie_word_embeddings"):
        del emb
    for li in range(cfg["num_hidden_layers"]):
        p = "model.layers.%d." % li
        a = p + "self_attn."
        y = _unit(x, eps) * w.norm(p + "input_layernorm.weight", h)
        q = (y @ w(a + "q_proj.weight", nh * hd, h).t()).view(-1, nh, hd)
        k = (y @ w(a + "k_proj.weight", kv * hd, h).t()).view(-1, kv, hd)
        v = (y @ w(a + "v_proj.weight", kv * hd, h).t()).view(-1, kv, hd)
        if arch == "Qwen3ForCausalLM":
            q, k = _unit(q, eps) * w.norm(a + "q_norm.weight", hd), _unit(k, eps) * w.norm(a + "k_norm.weight", hd)
        if arch == "Qwen2ForCausalLM":
            q, k, v = (t + w(a + n + "_proj.bias", t.shape[1] * hd).view(-1, hd) for t, n in ((q, "q"), (k, "k"), (v, "v")))
        o = torch.cat([_attend(_turn(a_, freqs), _turn(b_, freqs), c_, hd ** -0.5)
                       for a_, b_, c_ in zip(q.split(cuts), k.split(cuts), v.split(cuts))])
        x = x + o.view(-1, nh * hd) @ w(a + "o_proj.weight", h, nh * hd).t()
        y = _unit(x, eps) * w.norm(p + "post_attention_layernorm.weight", h)
        g = _silu(y @ w(p + "mlp.gate_proj.weight", ff, h).t()) * (y @ w(p + "mlp.up_proj.weight", ff, h).t())
        x = x + g @ w(p + "mlp.down_proj.weight", h, ff).t()
    x = torch.cat([t[r] for t, r in zip(x.split(cuts), rows)])
    head = emb if cfg.get("tie_word_embeddings") else w("lm_head.weight", cfg["vocab_size"], h)
    return (_unit(x, eps) * w.norm("model.norm.weight", h)) @ head.t()


def _karitar(cfg, w, seqs, rows):
    d, eps, cuts, n = cfg["width"], cfg["norm"]["eps"], [len(s) for s in seqs], cfg["streams"]
    x = w("embed", cfg["vocab"], d)[torch.tensor([t for s in seqs for t in s], device=w.device)][None].repeat(n, 1, 1)
    for li, lay in enumerate(cfg["layers"]):
        p, m, mx, ff = "l%d." % li, "l%d.mix." % li, lay["mixer"], lay["mlp"]["ff"]
        heads, kv, dim, vd, size = mx["heads"], mx["kv_heads"], mx["dim"], mx["vdim"], mx["mask"]["size"]

        def mixer(h):
            q = _unit(h @ w(m + "q", heads * dim, d).t() + w(m + "q.b", heads * dim), eps) * w.norm(m + "q.norm", heads * dim)
            k = _unit(h @ w(m + "k", kv * dim, d).t() + w(m + "k.b", kv * dim), eps) * w.norm(m + "k.norm", kv * dim)
            v = h @ w(m + "v", kv * vd, d).t() + w(m + "v.b", kv * vd)
            o = torch.cat([_attend(a.view(-1, heads, dim), b.view(-1, kv, dim), c.view(-1, kv, vd), mx["scale"],
                                   lambda i, j: i - j < size, torch.zeros(heads, dtype=F64, device=w.device))
                           for a, b, c in zip(q.split(cuts), k.split(cuts), v.split(cuts))])
            o = o * torch.sigmoid(h @ w(m + "g", heads, d).t())[:, :, None]
            return o.view(-1, heads * vd) @ w(m + "o", d, heads * vd).t()

        def feed(h):
            return torch.relu(h @ w(p + "mlp.up", ff, d).t()).square() @ w(p + "mlp.down", d, ff).t()

        for hc, norm, f in (("hc1.", "norm1", mixer), ("hc2.", "norm2", feed)):
            mix = w(p + hc + "mix", n, n, std=0.1)
            mix = (mix.bfloat16() + torch.eye(n, dtype=torch.bfloat16, device=w.device)).to(F64)
            y = f(_unit(torch.einsum("s,std->td", w.norm(p + hc + "in", n), x), eps) * w.norm(p + norm, d))
            x = torch.einsum("sr,std->rtd", mix, x) + w.norm(p + hc + "out", n)[:, None, None] * y
    x = torch.cat([t[r] for t, r in zip(x.sum(0).split(cuts), rows)])
    return (_unit(x, eps) * w.norm("final.norm", d)) @ w("head", cfg["vocab"], d).t()


def _conv(u, taps, bias=0.0):
    """A causal convolution per channel; taps' last column weighs the current token."""
    k = taps.shape[1]
    padded = torch.cat([u.new_zeros(k - 1, u.shape[1]), u])
    return bias + sum(padded[j:j + len(u)] * taps[:, j] for j in range(k))


def _gelu(x):
    return torch.nn.functional.gelu(x, approximate="tanh")


def _retention(q, k, v, decay):
    s = torch.zeros(q.shape[1], q.shape[2], v.shape[2], dtype=F64, device=q.device)
    out = torch.empty_like(v)
    for i in range(q.shape[0]):
        s = decay[:, None, None] * s + k[i][:, :, None] * v[i][:, None]
        out[i] = (q[i][:, None] @ s)[:, 0]
    return out


def _side_by_side(h, w, m, mx, d, eps, cuts):
    l, r = mx["left"], mx["right"]
    heads, kv, dim, vd = l["heads"], l["kv_heads"], l["dim"], l["vdim"]
    freqs, p = _powers(l["rot"]["base"], l["rot"]["dims"]), m + "left."
    sides = []
    q, k, v = ((h @ w(p + n, c * e, d).t()).split(cuts) for n, c, e in (("q", heads, dim), ("k", kv, dim), ("v", kv, vd)))
    taps = [w(p + n + ".conv", c * e, l["conv"], std=0.5) for n, c, e in (("q", heads, dim), ("k", kv, dim), ("v", kv, vd))]
    o = torch.cat([_attend(_turn(_conv(a, taps[0]).view(-1, heads, dim), freqs), _turn(_conv(b, taps[1]).view(-1, kv, dim), freqs),
                           _conv(c, taps[2]).view(-1, kv, vd), l["scale"]) for a, b, c in zip(q, k, v)]).view(-1, heads * vd)
    sides.append((o * torch.sigmoid(h @ w(p + "g", heads * vd, d).t())) @ w(p + "o", d, heads * vd).t())
    heads, dim, vd = r["heads"], r["dim"], r["vdim"]
    freqs, p = _powers(r["rot"]["base"], r["rot"]["dims"]), m + "right."
    decay = torch.tensor(r["decay"], dtype=F64, device=w.device)
    q, k, v = ((h @ w(p + n, heads * e, d).t()).view(-1, heads, e).split(cuts) for n, e in (("q", dim), ("k", dim), ("v", vd)))
    o = torch.cat([_retention(_turn(a, freqs), _turn(b, freqs) * dim ** -0.5, c, decay) for a, b, c in zip(q, k, v)])
    o = _unit(o, eps).view(-1, heads * vd) * _silu(h @ w(p + "g", heads * vd, d).t())
    sides.append(o @ w(p + "o", d, heads * vd).t())
    return sum(_unit(y, eps) * w.norm(m + n, d) for y, n in zip(sides, ("left.out", "right.out"))) / 2.0


def _rglru(h, w, m, mx, d, cuts):
    n, blocks = mx["width"], mx["blocks"]
    e = n // blocks
    y = _gelu(h @ w(m + "y", n, d).t() + w(m + "y.b", n))
    taps, bias = w(m + "conv", n, mx["conv"], std=0.5), w(m + "conv.b", n)
    u = torch.cat([_conv(t, taps, bias) for t in (h @ w(m + "x", n, d).t() + w(m + "x.b", n)).split(cuts)])
    r, i = (torch.sigmoid(torch.einsum("boi,tbi->tbo", w(m + g, blocks, e, e), u.view(-1, blocks, e)) + w(m + g + ".b", blocks, e)).reshape(-1, n)
            for g in ("ra", "ri"))
    a = torch.exp(-8.0 * r * torch.nn.functional.softplus(w(m + "lam", n, mean=-3.0, std=1.0)))
    out = []
    for a_, drive in zip(a.split(cuts), (torch.sqrt(1.0 - a * a) * i * u).split(cuts)):
        s = torch.zeros(n, dtype=F64, device=w.device)
        for t in range(len(a_)):
            s = a_[t] * s + drive[t]
            out.append(s)
    return (torch.stack(out) * y) @ w(m + "o", d, n).t()


def _piratar(cfg, w, seqs, rows):
    d, eps, cuts, em, dim = cfg["width"], cfg["norm"]["eps"], [len(s) for s in seqs], cfg["embedding"], cfg["token_side"]["dim"]
    plus = lambda x, name: _unit(x, eps) * (1.0 + w(name, d))      # noqa: E731  (these norms hold their weights less one)
    bg, pairs = em["bigram"], []
    for s in seqs:
        pairs += [bg["buckets"]] + [(a * bg["mul_prev"] + b * bg["mul_cur"]) % bg["buckets"] for a, b in zip(s, s[1:])]
    tok, pairs = torch.tensor([t for s in seqs for t in s], device=w.device), torch.tensor(pairs, device=w.device)
    x = plus(w("embed", cfg["vocab"], d)[tok] * em["scale"] + w("bigram", bg["buckets"] + 1, d)[pairs], "embed.norm")
    side = w("side.embed", cfg["vocab"], dim * len(cfg["layers"]))[tok]
    for li, lay in enumerate(cfg["layers"]):
        p, m, ff = "l%d." % li, "l%d.mix." % li, lay["mlp"]["ff"]
        h = plus(x, p + "norm1")
        y = _rglru(h, w, m, lay["mixer"], d, cuts) if lay["type"] == "rglru" else _side_by_side(h, w, m, lay["mixer"], d, eps, cuts)
        h = plus(x, p + "norm2")
        g = _silu(h @ w(p + "mlp.gate", ff, d).t()) * (h @ w(p + "mlp.up", ff, d).t())
        x = x + y + g @ w(p + "mlp.down", d, ff).t()
        s = _gelu(x @ w(p + "side.gate", dim, d).t()) * side[:, li * dim:(li + 1) * dim]
        x = x + _unit(s @ w(p + "side.proj", d, dim).t(), eps) * w.norm(p + "side.norm", d)
    x = torch.cat([t[r] for t, r in zip(x.split(cuts), rows)])
    return plus(x, "final.norm") @ w("head", cfg["vocab"], d).t()


def exact(case, seed):
    # a mixture's choice of experts is a step function of rounded inputs: no one value is what a bfloat16 run is near
    if case["kind"] == "sample" or case["model"] == "penasun":
        return None
    cfg = config_of(case)
    before, brings = _given(case, seed)
    seqs = [a + b for a, b in zip(before, brings)]
    if _step_work(case, cfg, [len(s) for s in seqs], [0] * len(seqs), 1)[1] > 2e14:      # over about 20 seconds in float64
        return None
    w = Weights(seed, "cuda")
    with torch.no_grad():
        back = case["steps"] + 1 if case["kind"] == "session" else 1
        rows = [range(len(s)) if case.get("every") else range(len(s) - back, len(s)) for s in seqs]
        rows = [torch.tensor(list(r), device=w.device) for r in rows]
        out = (_dense if case["model"] in DENSE else _karitar if case["model"] == "karitar" else _piratar)(cfg, w, seqs, rows)
    return out if case["kind"] != "session" else out.view(len(seqs), back, -1).transpose(0, 1).contiguous()
