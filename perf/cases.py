"""What this library is timed on: the work that its users have it do, through its public entry points.

Two kinds of pass, over every architecture the library runs, with random weights at the benchmark's layer sizes:

* ``prompt``: ``Stepper.step`` over whole prompts of new sequences, logits at each prompt's end: the time to the first
  token.  Slots are taken and given back in the pass, token ids are host lists, as a server's are.
* ``decode``: one token more for every running sequence, replayed from a captured graph as ``Engine.generate`` does:
  the layers, the output head and the choice of the token.  The sequences' lengths stay where they are, so that every
  pass is the same step; a recurrent layer's state moves on with every pass.

The tokens of a pass are no output of it: random weights leave the first two candidates closer than the rounding of
bfloat16, so the chosen tokens' logits are returned beside all logits, and not their numbers.

``exact`` is every architecture's forward pass in 64 bits, whole sequences, no cache.
"""

from __future__ import annotations

import gc
import math
import random

import torch

from starter_b200.config import config_from_dict
from starter_b200.engine.context import lengths_uneven
from starter_b200.engine.graph import GraphDecoder
from starter_b200.engine.session import Session
from starter_b200.engine.step import StepEntry
from starter_b200.sampling import SamplingParams
from starter_b200.weights import RandomSource

DEVICE = "cuda:0"
F = torch.float64


# ---- the models: the sizes that bench.py measures ----------------------------------------------------------------

def _qwen3(hidden, ff, layers, heads, theta):
    return dict(architectures=["Qwen3ForCausalLM"], hidden_size=hidden, intermediate_size=ff, num_hidden_layers=layers,
                num_attention_heads=heads, num_key_value_heads=8, head_dim=128, vocab_size=151936, rms_norm_eps=1e-6,
                rope_theta=theta, tie_word_embeddings=True)


def _kudazen(width, ff, latent, wkv, attention):
    kinds = [{"type": "latent_attention", "mixer": dict(latent, scale=(latent["dim"] + latent["rot_dim"]) ** -0.5,
                                                        rot={"base": 10000.0, "dims": latent["rot_dim"]})},
             {"type": "wkv", "mixer": dict(wkv)},
             {"type": "attention", "mixer": dict(attention, scale=attention["dim"] ** -0.5)}]
    return {"architecture": "Kudazen", "vocab": 32000, "width": width, "norm": {"eps": 1e-5, "groups": 2},
            "layers": [dict(kinds[i % 3], mlp={"kind": "dense", "ff": ff, "limit": 7.0}) for i in range(6)]}


def _nazulorn(width, gla, attention, experts, expert_ff, shared_ff):
    kinds = [{"type": "gla", "mixer": dict(gla, tau=8.0)},
             {"type": "attention", "mixer": dict(attention, scale=attention["dim"] ** -0.5, diff=0.5,
                                                 rot={"base": 500000.0, "dims": attention["dim"],
                                                      "scaling": {"factor": 8.0, "original": 4096, "fast": 16.0, "slow": 2.0}})}]
    mlp = {"kind": "moe", "router": {"experts": experts, "identity": 2, "top": 4, "scale": 2.0},
           "expert": {"ff": expert_ff, "limit": 7.0}, "shared": {"ff": shared_ff, "limit": 7.0}}
    return {"architecture": "Nazulorn", "vocab": 32000, "width": width, "norm": {"eps": 1e-5}, "embedding": {"scale": 1.0},
            "residual_mult": 0.5, "streams": 2, "logit_scale": 1.0, "layers": [dict(kinds[min(i % 3, 1)], mlp=mlp) for i in range(6)]}


def _gulazen(width, attention, ff, experts, expert_ff, shared_ff):
    mixer = dict(attention, scale=attention["dim"] ** -0.5, softcap=30.0)
    dense = {"kind": "dense", "ff": ff}
    moe = {"kind": "moe", "router": {"experts": experts, "top": 4}, "expert": {"ff": expert_ff}, "shared": {"ff": shared_ff}}
    return {"architecture": "Gulazen", "vocab": 32000, "width": width, "norm": {"eps": 1e-5}, "canon": {"taps": 4},
            "layers": [{"type": "attention", "mixer": mixer, "mlp": moe if i % 2 else dense} for i in range(6)]}


def _paditar(width, attention, left, right, ff):
    two_maps = {"type": "attention", "mixer": dict(attention, scale=attention["dim"] ** -0.5, diff=0.5,
                                                   rot={"base": 500000.0, "dims": attention["dim"] // 2})}
    pair = {"type": "parallel", "mixer": {"left": dict(left, vdim=left["dim"], scale=left["dim"] ** -0.5, conv=4,
                                                       q_temp={"coef": 0.2, "every": 64}),
                                          "right": dict(right, gate_cap=15.0), "left_scale": 1.0, "right_scale": 0.6}}
    return {"architecture": "Paditar", "vocab": 32000, "width": width, "norm": {"eps": 1e-5}, "loop": {"start": 0, "stop": 2, "times": 2},
            "layers": [dict(kind, mlp={"kind": "dense", "ff": ff}) for kind in (pair, two_maps, pair, two_maps)]}


def _siparax(width, latent, delta, ff):
    def layer(kind, **more):
        return {"type": kind, "mixer": dict(latent, scale=(latent["dim"] + latent["rot_dim"]) ** -0.5,
                                            rot={"base": 1000000.0, "dims": latent["rot_dim"],
                                                 "scaling": {"factor": 4.0, "original": 8192, "fast": 24.0, "slow": 2.0}}, **more)}
    recurrent = {"type": "channel_delta", "mixer": dict(delta, conv=4)}
    kinds = [recurrent, layer("latent_attention_2"), layer("latent_attention"),
             recurrent, layer("latent_attention_2", kv_from=1), layer("latent_attention")]
    return {"architecture": "Siparax", "vocab": 32000, "width": width, "norm": {"eps": 1e-5}, "logit_softcap": 30.0,
            "layers": [dict(kind, mlp={"kind": "dense", "ff": ff}) for kind in kinds]}


def _nifalorn(width, lightning, mamba, attention, experts, expert_ff, shared_ff):
    decay = [1.0 - 2.0 ** -(1.0 + 7.0 * i / (lightning["heads"] - 1)) for i in range(lightning["heads"])]
    attn = {"type": "attention", "mixer": dict(attention, scale=attention["dim"] ** -0.5, diff=0.4,
                                               rot={"base": 500000.0, "dims": attention["dim"],
                                                    "scaling": {"factor": 8.0, "low": 1.0, "high": 4.0, "original": 4096}})}
    kinds = [{"type": "lightning", "mixer": dict(lightning, decay=decay)}, attn, attn,
             {"type": "mamba2", "mixer": dict(mamba, conv=4)}, attn, attn]
    mlp = {"kind": "moe", "router": {"experts": experts, "top": 4, "scale": 2.0, "groups": {"count": 4, "keep": 2}},
           "expert": {"ff": expert_ff}, "shared": {"ff": shared_ff}}
    return {"architecture": "Nifalorn", "vocab": 32000, "width": width, "norm": {"eps": 1e-5}, "embedding": {"scale": 1.0},
            "logit_scale": 1.0, "layers": [dict(kind, mlp=mlp) for kind in kinds]}


_CHUNKED = dict(heads=16, kv_heads=4, dim=64, vdim=64), dict(heads=16, kv_heads=8, dim=128, vdim=128)
_MAPS = dict(heads=8, kv_heads=2, dim=64, vdim=64), dict(heads=8, kv_heads=4, dim=128, vdim=128)
_LATENT = (dict(heads=8, dim=64, rot_dim=32, vdim=64, q_rank=384, kv_rank=256),
           dict(heads=16, dim=128, rot_dim=64, vdim=128, q_rank=768, kv_rank=512))
MODELS = {
    "qwen3-4b": _qwen3(2560, 9728, 36, 32, 5000000.0),
    "qwen3-1.7b": _qwen3(2048, 6144, 28, 16, 1000000.0),
    "qwen3-4b-2layers": _qwen3(2560, 9728, 2, 32, 5000000.0),   # what the 32-bit check (bench.py --check) runs
    "kudazen-1024": _kudazen(1024, 4096, _LATENT[0], dict(heads=16, dim=64, decay_rank=64), dict(_CHUNKED[0], mask={"size": 1024})),
    "kudazen-2048": _kudazen(2048, 8192, _LATENT[1], dict(heads=32, dim=64, decay_rank=64), dict(_CHUNKED[1], mask={"size": 2048})),
    "nazulorn-1024": _nazulorn(1024, dict(heads=8, dim=64, vdim=128, decay_rank=64), dict(_MAPS[0], mask={"size": 1024}), 16, 512, 2048),
    "nazulorn-2048": _nazulorn(2048, dict(heads=16, dim=64, vdim=128, decay_rank=64), dict(_MAPS[1], mask={"size": 2048}), 32, 1024, 4096),
    "gulazen-1024": _gulazen(1024, dict(_CHUNKED[0], mask={"size": 1024, "keep_first": 4}), 4096, 16, 512, 2048),
    "gulazen-2048": _gulazen(2048, dict(_CHUNKED[1], mask={"size": 2048, "keep_first": 4}), 8192, 32, 1024, 4096),
    "paditar-1024": _paditar(1024, _MAPS[0], dict(heads=8, kv_heads=2, dim=64), dict(heads=8, dim=64, vdim=128), 4096),
    "paditar-2048": _paditar(2048, _MAPS[1], dict(heads=8, kv_heads=4, dim=128), dict(heads=16, dim=64, vdim=128), 8192),
    "siparax-1024": _siparax(1024, _LATENT[0], dict(heads=16, kv_heads=16, dim=64, vdim=64, decay_rank=64, gate_rank=64), 4096),
    "siparax-2048": _siparax(2048, _LATENT[1], dict(heads=32, kv_heads=32, dim=64, vdim=64, decay_rank=64, gate_rank=64), 8192),
    "nifalorn-1024": _nifalorn(1024, dict(heads=8, dim=64, vdim=128), dict(heads=16, vdim=64, state=128, groups=2, norm_groups=2),
                               dict(_MAPS[0], mask={"size": 1024}), 16, 512, 2048),
    "nifalorn-2048": _nifalorn(2048, dict(heads=16, dim=64, vdim=128), dict(heads=32, vdim=64, state=128, groups=4, norm_groups=4),
                               dict(_MAPS[1], mask={"size": 2048}), 32, 1024, 4096),
}
FAMILIES = [n for n in MODELS if not n.startswith("qwen3")]


# ---- the cases -----------------------------------------------------------------------------------------------------

def _case(name, model, kind, batch, longest, ragged=False, dtype="bfloat16"):
    return dict(name=name, model=model, kind=kind, batch=batch, longest=longest, ragged=ragged, dtype=dtype)


def listed():
    return [
        # one user at a terminal: the latency of a token
        _case("qwen4b_decode_1", "qwen3-4b", "decode", 1, 4096),
        # the headline: a small server's batch near the end of the context
        _case("qwen4b_decode_8", "qwen3-4b", "decode", 8, 4096),
        # a full server: many users, each at a place of their own
        _case("qwen4b_decode_64_ragged", "qwen3-4b", "decode", 64, 2048, ragged=True),
        # the time to the first token of one long question
        _case("qwen4b_prompt_2048", "qwen3-4b", "prompt", 1, 2048),
        # a batch of documents of unequal length
        _case("qwen1.7b_prompts_16_ragged", "qwen3-1.7b", "prompt", 16, 2048, ragged=True),
        # the true 32-bit run that bfloat16 is held against
        _case("qwen4b_float32_prompt_300", "qwen3-4b-2layers", "prompt", 1, 300, dtype="float32"),
        # each further architecture as its users meet it: a prompt, several prompts, or a running batch
        _case("kudazen_prompt_2048", "kudazen-2048", "prompt", 1, 2048),
        _case("nazulorn_prompts_4_ragged", "nazulorn-1024", "prompt", 4, 1999, ragged=True),
        _case("gulazen_decode_8", "gulazen-2048", "decode", 8, 2048),
        _case("paditar_prompt_3333", "paditar-2048", "prompt", 1, 3333),
        _case("siparax_prompts_3_ragged", "siparax-2048", "prompt", 3, 1500, ragged=True),
        _case("nifalorn_decode_24_ragged", "nifalorn-1024", "decode", 24, 1024, ragged=True),
    ]


def _log_between(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    """A case of the same ranges: any architecture, both kinds of pass, one sequence to a full batch."""
    if rng.random() < 0.1:
        return {k: v for k, v in _case("", "qwen3-4b-2layers", "prompt", rng.randint(1, 3), _log_between(rng, 9, 400), dtype="float32").items() if k != "name"}
    model = rng.choice(["qwen3-4b", "qwen3-1.7b"]) if rng.random() < 0.35 else rng.choice(FAMILIES)
    kind = rng.choice(["prompt", "decode"])
    if kind == "prompt":
        batch = _log_between(rng, 1, 12)
        longest = _log_between(rng, 30, min(4096, (6000 if model == "qwen3-4b" else 12000) // batch))
    else:
        batch = _log_between(rng, 1, 64)
        longest = _log_between(rng, 40, min(4096, 100000 // batch))
    return {k: v for k, v in _case("", model, kind, batch, longest, ragged=batch > 1 and rng.random() < 0.6).items() if k != "name"}


def _lengths(case):
    """Tokens of every sequence: the longest first, the others anywhere from a sixteenth of it on where they are ragged."""
    longest = case["longest"]
    if not case["ragged"]:
        return [longest] * case["batch"]
    rng = random.Random(f"{case['batch']}:{longest}")
    return [longest] + [rng.randint(max(1, longest // 16), longest) for _ in range(case["batch"] - 1)]


# ---- a user's program ----------------------------------------------------------------------------------------------

class _Weights(RandomSource):
    """Random weights that keep a row's size from layer to layer, as a model is initialised for training: embedding rows
    of size one, matrices that keep their input's size, and those whose product returns to the residual (a mixer's and a
    feed-forward's last) smaller by the root of the number of branches.  A mixture's router is decisive, as a trained one
    is: every token leans towards experts of its own, so that the choice does not hang on the rounding of bfloat16."""

    def __init__(self, case, device="cpu"):
        raw = MODELS[case["model"]]
        self.config = config_from_dict(raw)
        super().__init__(self.config, seed=0, dtype=_dtype(case), device=device)
        self.given, self.branches = self.init, 2 * len(self.config.model_spec().layers)
        self.init = self._init
        self.router = next((layer["mlp"]["router"] for layer in raw.get("layers", ()) if "router" in layer["mlp"]), None)

    def _init(self, name, shape):
        last = name.removesuffix(".weight").rsplit(".", 1)[-1]
        if self.given is not None:
            mean, std = self.given(name, shape)
        elif len(shape) == 1:
            mean, std = 1.0, 0.1
        else:
            mean, std = 0.0, 1.0 if last == "embed_tokens" else float(shape[-1]) ** -0.5
        if last in ("o", "down", "o_proj", "down_proj"):
            std *= self.branches ** -0.5
        return mean, std

    def get(self, name):
        t = super().get(name)
        if self.router is None or not (name == "embed" or name.endswith("mlp.router")):
            return t
        r, width = self.router, t.shape[1]
        n = r["experts"] + r.get("identity", 0)
        g = torch.Generator(device=self.device).manual_seed(1)
        towards = torch.randn(n, width, generator=g, device=self.device)
        if name != "embed":
            return (towards * width ** -0.5).to(t.dtype)
        groups = r.get("groups", {"count": 1, "keep": 1})
        lean = torch.rand(t.shape[0], groups["count"], n // groups["count"], generator=g, device=self.device)
        own = lean >= lean.topk(r["top"] // groups["keep"], -1).values[..., -1:]
        kept = torch.rand(t.shape[0], groups["count"], 1, generator=g, device=self.device)
        own = own & (kept >= kept.topk(groups["keep"], 1).values[:, -1:])
        return (t.float() + 0.4 * own.reshape(t.shape[0], n).float() @ towards).to(t.dtype)


STATES = 4      # running batches that a session has room for
_session_of = {}


def _session(case):
    """The loaded model with its cache, kept from one batch of inputs to the next as a server keeps it."""
    key = (case["model"], case["dtype"], case["kind"], case["batch"], case["longest"], case["ragged"])
    if key not in _session_of:
        _session_of.clear()
        gc.collect()
        torch.cuda.empty_cache()
        pages = sum((n + 1 + 63) // 64 for n in _lengths(case)) * (STATES if case["kind"] == "decode" else 1)
        weights = _Weights(case, DEVICE)
        _session_of[key] = Session((weights.config, weights), dtype=case["dtype"],
                                   max_tokens=64 * pages, max_seqs=case["batch"] * (STATES if case["kind"] == "decode" else 1),
                                   max_seq_tokens=case["longest"] + 1, max_step_tokens=max(1024, case["longest"]), device=DEVICE, verbose=False)
    return _session_of[key]


def _dtype(case):
    return getattr(torch, case["dtype"])


def _tokens(case, seed):
    """Host token lists: the sequences, and the token that a decode step feeds to each."""
    vocab = config_from_dict(MODELS[case["model"]]).model_spec().vocab_size
    g = torch.Generator().manual_seed(int(seed))
    sequences = [torch.randint(0, vocab, (n,), generator=g).tolist() for n in _lengths(case)]
    return sequences, torch.randint(0, vocab, (case["batch"],), generator=g).tolist()


class _Running:
    """A batch of sequences that hold their tokens, and the captured graph of their next step."""

    def __init__(self, session, sequences, tokens):
        cache, model, ops = session.cache, session.model, session.runtime.ops
        self.cache, self.slots = cache, [cache.alloc() for _ in sequences]
        for slot, seq in zip(self.slots, sequences):
            cache.reserve(slot, len(seq) + 1)
        session.stepper.step([StepEntry(slot, seq) for slot, seq in zip(self.slots, sequences)])
        self.bucket = GraphDecoder(session, SamplingParams()).new_bucket(len(sequences), lengths_uneven([len(s) + 1 for s in sequences]))
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            self._step(model, ops)   # on the cache's null slot: no sequence is touched
        torch.cuda.current_stream().wait_stream(side)
        torch.cuda.synchronize()
        self.graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(self.graph):
            logits, score = self._step(model, ops)
        self.logits, self.score = logits[:len(sequences)], score[:len(sequences)]
        cache.flush()
        self.bucket.load(self.slots, tokens, list(range(len(sequences))), 0)

    def _step(self, model, ops):
        b = self.bucket
        with ops.status_into(b.status):
            logits = model.logits(b.ctx, model.hidden(b.ctx, b.tokens), None)
            chosen = ops.argmax(logits)
        return logits, torch.gather(logits, 1, chosen.long()[:, None])

    def __del__(self):
        for slot in self.slots:
            self.cache.free(slot)


def prepare(case, seed):
    session = _session(case)
    sequences, tokens = _tokens(case, seed)
    if case["kind"] == "decode":
        return _Running(session, sequences, tokens)
    return session, sequences


def run(state):
    if isinstance(state, _Running):
        state.graph.replay()
        return {"logits": state.logits, "score": state.score}
    session, prompts = state
    cache = session.cache
    slots = [cache.alloc() for _ in prompts]
    try:
        return {"logits": session.stepper.step([StepEntry(s, p, [len(p) - 1]) for s, p in zip(slots, prompts)])}
    finally:
        for s in slots:
            cache.free(s)


# ---- what a pass cannot do without -------------------------------------------------------------------------------------

def _pairs(lengths, kind, window=None, chunk=None):
    """(query, key) pairs that are visible, and keys that a pass has to read."""
    pairs = keys = 0
    for n in lengths:
        if kind == "decode":
            reach = n + 1
            if window:
                reach = min(reach, window)
            if chunk:
                reach = n % chunk + 1
            pairs, keys = pairs + reach, keys + reach
            continue
        if chunk:
            full, rest = divmod(n, chunk)
            pairs += full * chunk * (chunk + 1) // 2 + rest * (rest + 1) // 2
        else:
            w = min(window or n, n)
            pairs += w * (w + 1) // 2 + (n - w) * w
        keys += n
    return pairs, keys


def _mixer_work(entry, lengths, kind, size):
    """(bytes of cache and state, flops beside the matrices) of one layer run."""
    m, B = entry["mixer"], len(lengths)
    rows = sum(lengths) if kind == "prompt" else B
    if entry["type"] == "parallel":
        left = _mixer_work({"type": "attention", "mixer": dict(m["left"], maps=1)}, lengths, kind, size)
        right = _mixer_work({"type": "mlstm", "mixer": m["right"]}, lengths, kind, size)
        return left[0] + right[0], left[1] + right[1]
    if entry["type"] in ("wkv", "gla", "mlstm", "channel_delta", "lightning", "mamba2"):
        state = m["heads"] * m.get("dim", m.get("state", 0)) * m.get("vdim", m.get("dim"))
        return B * state * 4 * (2 if kind == "decode" else 1), 6.0 * rows * state
    if entry["type"].startswith("latent"):
        pairs, keys = _pairs(lengths, kind)
        per_pair = 2 * m["kv_rank"] + m["rot_dim"] if kind == "decode" else m["dim"] + m["rot_dim"] + m["vdim"]
        return keys * (m["kv_rank"] + m["rot_dim"]) * size, 2.0 * pairs * m["heads"] * per_pair
    mask = m.get("mask") or {}
    chunked = "maps" in m and m["maps"] == "chunk"
    pairs, keys = _pairs(lengths, kind, window=None if chunked else mask.get("size"), chunk=mask.get("size") if chunked else None)
    maps = 2 if "diff" in m else 1
    return keys * m["kv_heads"] * (maps * m["dim"] + m["vdim"]) * size, 2.0 * pairs * m["heads"] * maps * (m["dim"] + m["vdim"])


def work(case):
    raw, lengths, kind = MODELS[case["model"]], _lengths(case), case["kind"]
    entries = _Weights(case).entries
    size = 4 if case["dtype"] == "float32" else 2
    rows, B = (sum(lengths) if kind == "prompt" else case["batch"]), case["batch"]
    arch = raw.get("architecture", "Qwen3")
    if arch == "Qwen3":
        mixer = dict(heads=raw["num_attention_heads"], kv_heads=8, dim=128, vdim=128)
        layers = [{"type": "attention", "mixer": mixer}] * raw["num_hidden_layers"]
        embed, head, vocab, width = "model.embed_tokens.weight", "lm_head.weight", raw["vocab_size"], raw["hidden_size"]
    else:
        layers, embed, head, vocab, width = raw["layers"], "embed", "head", raw["vocab"], raw["width"]
    times = [1] * len(layers)
    if raw.get("loop"):
        for i in range(raw["loop"]["start"], raw["loop"]["stop"]):
            times[i] = raw["loop"]["times"]
    nbytes = 2.0 * B * vocab * 2 + rows * width * size      # 32-bit logits out, embedding rows in
    flops = 2.0 * B * vocab * width
    for name, (_, shape) in entries.items():
        n = math.prod(shape)
        if name == embed:
            nbytes += n * size if head not in entries else 0    # the output head reads the table
            continue
        share = 1.0
        parts = name.split(".")
        if "mlp" in parts and len(parts) == 4 and parts[2][:1] == "e" and parts[2][1:].isdigit():
            r = layers[int(parts[0][1:])]["mlp"]["router"]
            share = r["top"] / (r["experts"] + r.get("identity", 0))
            nbytes += n * size * (1.0 - (1.0 - share) ** rows)  # experts that no row chooses stay unread
        else:
            nbytes += n * size
        if len(shape) == 2 and name != head:
            runs = times[int(parts[0][1:])] if parts[0][1:].isdigit() else 1
            flops += 2.0 * rows * n * share * runs
    for entry, t in zip(layers, times):
        if arch == "Kudazen" and entry["type"] == "attention":
            entry = {"type": "attention", "mixer": dict(entry["mixer"], maps="chunk")}
        b, f = _mixer_work(entry, lengths, kind, size)
        nbytes, flops = nbytes + t * b, flops + t * f
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    """About four times what the library's logits are off exact()'s (2-norm; its own outputs are the same every time):
    the true 32-bit run 1.3e-6 (5e-6 with rows of other sizes); bfloat16 with a bfloat16 residual over 28 and 36 layers 0.013 and 0.015 (0.03 is the most
    that is allowed), with a 32-bit residual over 6 layers 0.002 to 0.006."""
    if case["dtype"] == "float32":
        return {"rel": 2e-5}
    if case["model"].startswith("qwen3"):
        return {"rel": 0.03, "max": 0.3}
    return {"rel": 0.02, "max": 0.3}


# ---- every architecture in 64 bits --------------------------------------------------------------------------------------

EXACT_FLOPS = 2.5e14     # a pass over whole sequences beyond this takes over about ten seconds in 64 bits


def _rms(x, eps):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps)


def _layer_norm(x, w, b, eps):
    x = x - x.mean(-1, keepdim=True)
    return _rms(x, eps) * w + b


def _silu(z):
    return z * torch.sigmoid(z)


def _frequencies(rot):
    """(radians a position per pair, size of cosines and sines): plain, stretched by pair index, or blended by wavelength."""
    dims, base, sc = int(rot["dims"]), float(rot["base"]), rot.get("scaling")
    out, size = [], 1.0
    if sc and "fast" in sc:
        def place(turns):
            return dims * math.log(sc["original"] / (2 * math.pi * turns)) / (2 * math.log(base))
        lo, hi = max(math.floor(place(sc["fast"])), 0), min(math.ceil(place(sc["slow"])), dims - 1)
        size = 0.1 * math.log(sc["factor"]) + 1.0
    for i in range(dims // 2):
        f = base ** (-2.0 * i / dims)
        if sc and "fast" in sc:
            ramp = min(max((i - lo) / max(hi - lo, 0.001), 0.0), 1.0)
            f = f / sc["factor"] * ramp + f * (1.0 - ramp)
        elif sc:
            length = 2 * math.pi / f
            if length > sc["original"] / sc["low"]:
                f = f / sc["factor"]
            elif length >= sc["original"] / sc["high"]:
                s = (sc["original"] / length - sc["low"]) / (sc["high"] - sc["low"])
                f = (1.0 - s) * f / sc["factor"] + s * f
        out.append(f)
    return torch.tensor(out, dtype=F, device=DEVICE), size


def _rotate(t, rot, halves):
    """t [T, ..., D]: the first rot.dims columns turn, pair i being columns (i, i + dims / 2) or (2 i, 2 i + 1)."""
    if not rot:
        return t
    f, size = _frequencies(rot)
    dims = int(rot["dims"])
    angle = torch.arange(t.shape[0], dtype=F, device=DEVICE)[:, None] * f
    shape = (t.shape[0],) + (1,) * (t.dim() - 2) + (dims // 2,)
    c, s = (torch.cos(angle) * size).reshape(shape), (torch.sin(angle) * size).reshape(shape)
    a, b = (slice(0, dims // 2), slice(dims // 2, dims)) if halves else (slice(0, dims, 2), slice(1, dims, 2))
    out = t.clone()
    out[..., a], out[..., b] = t[..., a] * c - t[..., b] * s, t[..., b] * c + t[..., a] * s
    return out


def _seen(T, window=None, chunk=None, keep=0):
    i, j = torch.arange(T, device=DEVICE)[:, None], torch.arange(T, device=DEVICE)[None, :]
    seen = j <= i
    if window:
        seen = seen & ((i - j < window) | (j < keep))
    if chunk:
        seen = seen & (i // chunk == j // chunk)
    return seen


def _weights(scores, seen, sink=None):
    """Softmax over the visible keys; ``sink``: one more term exp(sink) in the denominator."""
    scores = scores.masked_fill(~seen, -math.inf)
    top = scores.amax(-1, keepdim=True)
    if sink is not None:
        top = torch.clamp(top, min=float(sink))
    e = torch.exp(scores - top)
    total = e.sum(-1, keepdim=True)
    if sink is not None:
        total = total + torch.exp(sink - top)
    return e / total


def _attend(q, k, v, scale, seen, sink=None, bias=None):
    """q [T, H, D], k [T, G, D], v [T, Gv, V], one head after another; sink [H]; bias(head) is added to a head's scores."""
    H = q.shape[1]
    outs = []
    for h in range(H):
        s = (q[:, h] @ k[:, h * k.shape[1] // H].T) * scale
        if bias is not None:
            s = bias(h, s)
        outs.append(_weights(s, seen, None if sink is None else sink[h]) @ v[:, h * v.shape[1] // H])
    return torch.stack(outs, 1)


def _conv(u, w, bias=None):
    """Causal convolution of every column: the weight's last column meets the current row."""
    T, taps = u.shape[0], w.shape[1]
    out = torch.zeros_like(u) if bias is None else bias.expand_as(u).clone()
    for j in range(taps):
        back = taps - 1 - j
        if back < T:
            out[back:] += w[:, j] * u[:T - back]
    return out


def _memory(q, k, v, decay, add=None, bonus=None):
    """S <- decay_t S + add_t k_t v_t^T, out_t = S^T q_t, head by head at once: q, k [T, H, D], v [T, H, V], decay
    [T, H, D] or [T, H, 1].  ``bonus`` [H, D]: out_t reads the old S and bonus * k_t v_t^T instead of the new one."""
    T, H, D = q.shape
    S = torch.zeros(H, D, v.shape[2], dtype=F, device=DEVICE)
    out = torch.empty(T, H, v.shape[2], dtype=F, device=DEVICE)
    if add is not None:
        k = k * add[..., None]
    for t in range(T):
        kv = k[t, :, :, None] * v[t, :, None, :]
        if bonus is not None:
            out[t] = torch.einsum("hd,hdv->hv", q[t], S + bonus[:, :, None] * kv)
        S = torch.addcmul(kv, decay[t, :, :, None], S)
        if bonus is None:
            out[t] = (q[t, :, None, :] @ S)[:, 0]
    return out


def _two_maps(h, w, m, eps, rot_halves, **mask):
    T, H, G, D, V = h.shape[0], m["heads"], m["kv_heads"], m["dim"], m["vdim"]
    q = _rotate((h @ w["q"].T).reshape(T, H, 2, D), m.get("rot"), rot_halves)
    k = _rotate((h @ w["k"].T).reshape(T, G, 2, D), m.get("rot"), rot_halves)
    v = (h @ w["v"].T).reshape(T, G, V)
    lam = torch.exp((w["lq1"] * w["lk1"]).sum()) - torch.exp((w["lq2"] * w["lk2"]).sum()) + m["diff"]
    seen = _seen(T, **mask)
    a, b = (_attend(q[:, :, i], k[:, :, i], v, m["scale"], seen) for i in (0, 1))
    return (_rms(a - lam * b, eps) * (1.0 - m["diff"])).reshape(T, H * V)


def _latent(h, w, m, eps, halves, gated=False, sink=None, rows=None):
    T, H, D, R, V = h.shape[0], m["heads"], m["dim"], m["rot_dim"], m["vdim"]
    if rows is None:
        d = h @ w["dkv"].T
        rows = _rms(d[:, :m["kv_rank"]], eps) * w["dkv.norm"], _rotate(d[:, m["kv_rank"]:], m["rot"], halves)
    c, k_rot = rows
    q = ((_rms(h @ w["dq"].T, eps) * w["dq.norm"]) @ w["uq"].T).reshape(T, H, D + R)
    q = torch.cat([q[..., :D], _rotate(q[..., D:], m["rot"], halves)], -1)
    k = torch.cat([(c @ w["uk"].T).reshape(T, H, D), k_rot[:, None].expand(T, H, R)], -1)
    o = _attend(q, k, (c @ w["uv"].T).reshape(T, H, V), m["scale"], _seen(T), sink=sink)
    if gated:
        o = o * torch.sigmoid(h @ w["g"].T)[..., None]
    return o.reshape(T, H * V) @ w["o"].T, rows


def _experts(h, w, chosen, weights, n_experts, one):
    """sum over the chosen: weight * expert; numbers from n_experts on hand the row itself back."""
    out = torch.zeros_like(h)
    for e in range(n_experts):
        rows, place = (chosen == e).nonzero(as_tuple=True)
        if len(rows):
            out.index_add_(0, rows, weights[rows, place, None] * one(h[rows], w[f"e{e}.gate"], w[f"e{e}.up"], w[f"e{e}.down"]))
    return out + (weights * (chosen >= n_experts)).sum(-1, keepdim=True) * h


def _swiglu(h, gate, up, down):
    return (_silu(h @ gate.T) * (h @ up.T)) @ down.T


def _clamped(limit):
    def one(h, gate, up, down):
        g, u = torch.clamp(h @ gate.T, max=limit), torch.clamp(h @ up.T, -limit, limit)
        return (g * torch.sigmoid(1.702 * g) * (u + 1.0)) @ down.T
    return one


class _Tensors(dict):
    """A layer's tensors in 64 bits by their names below a prefix, made when they are first read."""

    def __init__(self, source, prefix):
        super().__init__()
        self.source, self.prefix = source, prefix

    def __missing__(self, name):
        self[name] = self.source.get(self.prefix + name).to(F)
        return self[name]

    def __contains__(self, name):
        return self.prefix + name in self.source.entries

    def below(self, prefix):
        return _Tensors(self.source, self.prefix + prefix)


def _qwen3_layer(x, w, raw, i, kept):
    T, H, G, D, eps = x.shape[0], raw["num_attention_heads"], raw["num_key_value_heads"], raw["head_dim"], raw["rms_norm_eps"]
    h = _rms(x, eps) * w["input_layernorm.weight"]
    rot = {"dims": D, "base": raw["rope_theta"]}
    q = _rms((h @ w["self_attn.q_proj.weight"].T).reshape(T, H, D), eps) * w["self_attn.q_norm.weight"]
    k = _rms((h @ w["self_attn.k_proj.weight"].T).reshape(T, G, D), eps) * w["self_attn.k_norm.weight"]
    v = (h @ w["self_attn.v_proj.weight"].T).reshape(T, G, D)
    o = _attend(_rotate(q, rot, True), _rotate(k, rot, True), v, D ** -0.5, _seen(T))
    x = x + o.reshape(T, H * D) @ w["self_attn.o_proj.weight"].T
    h = _rms(x, eps) * w["post_attention_layernorm.weight"]
    return x + _swiglu(h, w["mlp.gate_proj.weight"], w["mlp.up_proj.weight"], w["mlp.down_proj.weight"])


def _kudazen_layer(x, w, raw, i, kept):
    entry, eps, T = raw["layers"][i], raw["norm"]["eps"], x.shape[0]
    m, mix = entry["mixer"], w.below("mix.")
    h = _rms(x.reshape(T, raw["norm"]["groups"], -1), eps).reshape(T, -1) * w["norm1"]
    if entry["type"] == "latent_attention":
        y = _latent(h, mix, m, eps, False, sink=mix["sink"])[0]
    elif entry["type"] == "wkv":
        H, D = m["heads"], m["dim"]
        before = torch.cat([torch.zeros_like(h[:1]), h[:-1]])

        def of(name):
            return (h + (before - h) * mix["mu." + name]) @ mix["w1" if name == "w" else name].T
        r, k, v = (of(n).reshape(T, H, D) for n in "rkv")
        decay = torch.exp(-torch.exp(torch.tanh(of("w")) @ mix["w2"].T + mix["w0"])).reshape(T, H, D)
        o = _memory(r, k, v, decay, bonus=mix["u"].reshape(H, D))
        y = (_rms(o, eps).reshape(T, H * D) * mix["norm"] * _silu(of("g"))) @ mix["o"].T
    else:
        H, G, D, V = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
        pos = torch.arange(T, dtype=F, device=DEVICE)

        def bias(head, s):
            return s * mix["temp"][head] - 2.0 ** (-8.0 * (head + 1) / H) * (pos[:, None] - pos[None])
        o = _attend((h @ mix["q"].T).reshape(T, H, D), (h @ mix["k"].T).reshape(T, G, D), _rms((h @ mix["v"].T).reshape(T, G, V), eps),
                    m["scale"], _seen(T, chunk=m["mask"]["size"]), bias=bias)
        y = o.reshape(T, H * V) @ mix["o"].T
    return x + y + _clamped(entry["mlp"]["limit"])(h, w["mlp.gate"], w["mlp.up"], w["mlp.down"])


def _nazulorn_layer(X, w, raw, i, kept):
    entry, eps, S, mult = raw["layers"][i], raw["norm"]["eps"], raw["streams"], raw["residual_mult"]
    m, T, W = entry["mixer"], X.shape[0], raw["width"]
    X = X.reshape(T, S, W)
    for which in ("1", "2"):
        h = _rms(torch.einsum("s,tsw->tw", w[f"hc{which}.in"], X), eps) * w["norm" + which]
        if which == "2":
            f, r = w.below("mlp."), entry["mlp"]["router"]
            s = torch.softmax(h @ f["router"].T, -1)
            chosen = torch.topk(s + f["correction"], r["top"], -1).indices
            picked = s.gather(1, chosen)
            one = _clamped(entry["mlp"]["expert"]["limit"])
            y = _experts(h, f, chosen, picked / picked.sum(-1, keepdim=True) * r["scale"], r["experts"], one)
            y = y + one(h, f["shared.gate"], f["shared.up"], f["shared.down"])
        else:
            mix = w.below("mix.")
            if entry["type"] == "attention":
                y = _two_maps(h, mix, m, eps, True, window=m["mask"]["size"])
            else:
                H, D, V = m["heads"], m["dim"], m["vdim"]
                alpha = torch.sigmoid((h @ mix["a1"].T) @ mix["a2"].T + mix["a2.b"]) ** (1.0 / m["tau"])
                o = _memory((h @ mix["q"].T).reshape(T, H, D) * D ** -0.5, (h @ mix["k"].T).reshape(T, H, D),
                            (h @ mix["v"].T).reshape(T, H, V), alpha.reshape(T, H, D))
                y = (_rms(o, eps) * mix["norm"]).reshape(T, H * V) * _silu(h @ mix["g"].T)
            y = y @ mix["o"].T
        X = torch.einsum("st,jsw->jtw", w[f"hc{which}.mix"], X) + mult * w[f"hc{which}.out"][None, :, None] * y[:, None]
    return X.reshape(T, S * W)


def _gulazen_layer(x, w, raw, i, kept):
    entry, eps, T = raw["layers"][i], raw["norm"]["eps"], x.shape[0]
    m, mix = entry["mixer"], w.below("mix.")
    H, G, D, V = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
    h = x + _conv(x, w["canon1"])
    q = (_rms(h @ mix["q"].T, eps) * mix["q.norm"]).reshape(T, H, D)
    k = (_rms(h @ mix["k"].T, eps) * mix["k.norm"]).reshape(T, G, D)
    v = (h @ mix["v"].T).reshape(T, G, V)
    seen, o = _seen(T, window=m["mask"]["size"], keep=m["mask"]["keep_first"]), torch.empty(T, H, V, dtype=F, device=DEVICE)
    for t in range(0, T, 256):      # every head's scores at once, for some of the queries
        s = torch.stack([q[t:t + 256, a] @ k[:, a * G // H].T for a in range(H)]) * m["scale"]
        s = torch.einsum("hg,gij->hij", mix["talk"], m["softcap"] * torch.tanh(s / m["softcap"]))
        for a in range(H):
            o[t:t + 256, a] = _weights(s[a], seen[t:t + 256], mix["sink"][a]) @ v[:, a * G // H]
    x = x + _rms(o.reshape(T, H * V) @ mix["o"].T, eps) * (1.0 + w["norm1"]) * w["ls1"]
    f = w.below("mlp.")
    if entry["mlp"]["kind"] == "dense":
        z, (p, n) = x @ f["up"].T, torch.nn.functional.softplus(f["act"])
        y = torch.where(z > 0, p * z * z + 0.5 * z, (0.5 + n) * (torch.expm1(torch.clamp(z, max=0.0)) - z) + 0.5 * z) @ f["down"].T
    else:
        r = entry["mlp"]["router"]
        best = torch.topk(x @ f["router"].T + f["router.b"], r["top"], -1)
        y = _experts(x, f, best.indices, torch.softmax(best.values, -1), r["experts"], _swiglu)
        y = y + _swiglu(x, f["shared.gate"], f["shared.up"], f["shared.down"])
    return x + _rms(y, eps) * (1.0 + w["norm2"]) * w["ls2"]


def _paditar_layer(x, w, raw, i, kept):
    entry, eps, T = raw["layers"][i], raw["norm"]["eps"], x.shape[0]
    m, mix = entry["mixer"], w.below("mix.")
    h = _rms(x, eps) * (1.0 + w["norm1"])
    if entry["type"] == "attention":
        y = (_two_maps(h, mix, m, eps, True) * torch.sigmoid(h @ mix["g"].T)) @ mix["o"].T
    else:
        a, l = m["left"], mix.below("left.")
        H, G, D = a["heads"], a["kv_heads"], a["dim"]
        q, k = _conv(h @ l["q"].T + l["q.b"], l["q.conv"]).reshape(T, H, D), _conv(h @ l["k"].T + l["k.b"], l["k.conv"]).reshape(T, G, D)
        warm = torch.floor((torch.arange(T, dtype=F, device=DEVICE) + 1) / a["q_temp"]["every"])
        q = _rms(q, eps) * l["q.norm"] * (1.0 + a["q_temp"]["coef"] * torch.log(warm + 1.0))[:, None, None]
        o = _attend(q, _rms(k, eps) * l["k.norm"], k, a["scale"], _seen(T), sink=torch.zeros(H, dtype=F, device=DEVICE))
        y = m["left_scale"] * ((o * torch.sigmoid(h @ l["g"].T)[..., None]).reshape(T, H * D) @ l["o"].T + l["o.b"])
        b, r = m["right"], mix.below("right.")
        H, D, V, cap = b["heads"], b["dim"], b["vdim"], b["gate_cap"]
        log_i = cap * torch.tanh((h @ r["i"].T + r["i.b"]) / cap)
        log_f = torch.nn.functional.logsigmoid(cap * torch.tanh((h @ r["f"].T + r["f.b"]) / cap))
        tops, top = [], torch.zeros(H, dtype=F, device=DEVICE)
        for t in range(T):
            tops.append(torch.maximum(log_f[t] + top, log_i[t]))
            top = tops[-1]
        top = torch.stack(tops)
        keep = torch.exp(log_f + torch.cat([torch.zeros_like(top[:1]), top[:-1]]) - top)
        v = torch.cat([(h @ r["v"].T).reshape(T, H, V), torch.ones(T, H, 1, dtype=F, device=DEVICE)], -1)   # the last column is the sum of keys
        o = _memory((h @ r["q"].T).reshape(T, H, D) * D ** -0.5, (h @ r["k"].T).reshape(T, H, D), v, keep[..., None], add=torch.exp(log_i - top))
        o = o[..., :V] / (torch.maximum(o[..., V:].abs(), torch.exp(-top)[..., None]) + 1e-6)
        y = y + m["right_scale"] * ((_rms(o, eps).reshape(T, H * V) * r["norm"] * torch.sigmoid(h @ r["g"].T)) @ r["o"].T)
    x = x + _rms(y, eps) * (1.0 + w["norm1b"])
    h = _rms(x, eps) * (1.0 + w["norm2"])
    return x + _rms(torch.relu(h @ w["mlp.up"].T) ** 2 @ w["mlp.down"].T, eps) * (1.0 + w["norm2b"])


def _siparax_layer(x, w, raw, i, kept):
    entry, eps, T = raw["layers"][i], raw["norm"]["eps"], x.shape[0]
    m, mix = entry["mixer"], w.below("mix.")
    h = _layer_norm(x, w["norm1"], w["norm1.b"], eps)
    if entry["type"] == "channel_delta":
        H, G, D, V = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
        q, k, v = (_silu(_conv(h @ mix[n].T, mix[n + ".conv"])).reshape(T, a, b) for n, a, b in (("q", G, D), ("k", G, D), ("v", H, V)))
        q, k = (t / torch.sqrt((t * t).sum(-1, keepdim=True) + 1e-6) for t in (q, k))
        q, k = (t.repeat_interleave(H // G, 1) for t in (q * D ** -0.5, k))
        beta = torch.sigmoid(h @ mix["b"].T)
        pre = torch.nn.functional.softplus(h @ mix["a1"].T @ mix["a2"].T + mix["dt_bias"]).reshape(T, H, D)
        decay = torch.exp(-torch.exp(mix["A_log"])[None, :, None] * pre)
        S, o = torch.zeros(H, D, V, dtype=F, device=DEVICE), torch.empty(T, H, V, dtype=F, device=DEVICE)
        for t in range(T):
            S = decay[t, :, :, None] * S
            S = S + k[t, :, :, None] * (beta[t, :, None, None] * (v[t, :, None] - k[t, :, None] @ S))
            o[t] = (q[t, :, None] @ S)[:, 0]
        gate = torch.sigmoid(h @ mix["g1"].T @ mix["g2"].T).reshape(T, H, V)
        y = (_rms(o, eps) * mix["norm"] * gate).reshape(T, H * V) @ mix["o"].T
    else:
        second = entry["type"] == "latent_attention_2"
        y, kept[i] = _latent(h, mix, m, eps, second, gated=second, rows=kept.get(m.get("kv_from")))
    x = x + y
    h = _layer_norm(x, w["norm2"], w["norm2.b"], eps)
    return x + (torch.nn.functional.gelu(h @ w["mlp.gate"].T, approximate="tanh") * (h @ w["mlp.up"].T)) @ w["mlp.down"].T


def _nifalorn_layer(x, w, raw, i, kept):
    entry, eps, T = raw["layers"][i], raw["norm"]["eps"], x.shape[0]
    m, mix = entry["mixer"], w.below("mix.")
    h = _rms(x, eps) * (1.0 + w["norm1"])
    if entry["type"] == "attention":
        y = _two_maps(h, mix, m, eps, False, chunk=m["mask"]["size"]) @ mix["o"].T
    elif entry["type"] == "lightning":
        H, D, V = m["heads"], m["dim"], m["vdim"]
        q, k, v = (_silu(h @ mix[n].T).reshape(T, H, d) for n, d in (("q", D), ("k", D), ("v", V)))
        o = _memory(q, k, v, torch.tensor(m["decay"], dtype=F, device=DEVICE)[None, :, None].expand(T, H, 1))
        y = (_rms(o.reshape(T, H * V), eps) * mix["norm"] * torch.sigmoid(h @ mix["g"].T)) @ mix["o"].T
    else:
        H, V, N, G = m["heads"], m["vdim"], m["state"], m["groups"]
        z, u, dt = (h @ mix["in"].T).split([H * V, H * V + 2 * G * N, H], -1)
        v, k, q = _silu(_conv(u, mix["conv"], mix["conv.b"])).split([H * V, G * N, G * N], -1)
        v, k, q = v.reshape(T, H, V), k.reshape(T, G, N).repeat_interleave(H // G, 1), q.reshape(T, G, N).repeat_interleave(H // G, 1)
        dt = torch.nn.functional.softplus(dt + mix["dt_bias"])
        o = _memory(q, k, v, torch.exp(-torch.exp(mix["A_log"]) * dt)[..., None], add=dt) + mix["D"][:, None] * v
        o = o.reshape(T, H * V) * _silu(z)
        y = (_rms(o.reshape(T, m["norm_groups"], -1), eps).reshape(T, -1) * mix["norm"]) @ mix["o"].T
    x = x + y
    h, f, r = _rms(x, eps) * (1.0 + w["norm2"]), w.below("mlp."), entry["mlp"]["router"]
    s = torch.sigmoid(h @ f["router"].T)
    pick = (s + f["correction"]).reshape(T, r["groups"]["count"], -1)
    kept_groups = torch.topk(torch.topk(pick, 2, -1).values.sum(-1), r["groups"]["keep"], -1).indices
    allowed = torch.zeros(pick.shape[:2], dtype=torch.bool, device=DEVICE).scatter_(1, kept_groups, True)
    chosen = torch.topk(pick.masked_fill(~allowed[..., None], -math.inf).reshape(T, -1), r["top"], -1).indices
    picked = s.gather(1, chosen)
    y = _experts(h, f, chosen, picked / picked.sum(-1, keepdim=True) * r["scale"], r["experts"], _swiglu)
    return x + y + torch.sigmoid(h @ f["shared.sg"].T) * _swiglu(h, f["shared.gate"], f["shared.up"], f["shared.down"])


LAYERS = {"Qwen3": _qwen3_layer, "Kudazen": _kudazen_layer, "Nazulorn": _nazulorn_layer, "Gulazen": _gulazen_layer,
          "Paditar": _paditar_layer, "Siparax": _siparax_layer, "Nifalorn": _nifalorn_layer}


@torch.no_grad()
def exact(case, seed):
    raw = MODELS[case["model"]]
    arch = raw.get("architecture", "Qwen3")
    sequences, tokens = _tokens(case, seed)
    if case["kind"] == "decode":
        sequences = [s + [t] for s, t in zip(sequences, tokens)]
    whole = dict(case, kind="prompt")
    if work(whole)["flops"] > EXACT_FLOPS:
        return None
    source = _Weights(case, DEVICE)
    names = _Tensors(source, "")
    if arch == "Qwen3":
        embed, eps, prefix, order = names["model.embed_tokens.weight"], raw["rms_norm_eps"], "model.layers.%d.", list(range(raw["num_hidden_layers"]))
    else:
        embed, eps, prefix, order = names["embed"], raw["norm"]["eps"], "l%d.", list(range(len(raw["layers"])))
    xs = [embed[torch.tensor(s, device=DEVICE)] for s in sequences]
    if arch in ("Nazulorn", "Nifalorn"):
        xs = [x * raw["embedding"]["scale"] for x in xs]
    if arch == "Nazulorn":
        xs = [x.repeat(1, raw["streams"]) for x in xs]
    if arch == "Siparax":
        xs = [_layer_norm(x, names["embed.norm"], names["embed.norm.b"], eps) for x in xs]
    if arch == "Gulazen":
        angle = 10000.0 ** (-torch.arange(0, raw["width"], 2, dtype=F, device=DEVICE) / raw["width"])
        xs = [x + torch.stack([torch.sin(a), torch.cos(a)], -1).reshape(x.shape)
              for x, a in ((x, torch.arange(len(x), dtype=F, device=DEVICE)[:, None] * angle) for x in xs)]
    starts = {}
    if raw.get("loop"):
        first, last, times = raw["loop"]["start"], raw["loop"]["stop"], raw["loop"]["times"]
        starts = {first + t * (last - first): t for t in range(times)}
        order = order[:first] + order[first:last] * times + order[last:]
        embedded = xs
    kept = [{} for _ in xs]
    for pos, i in enumerate(order):
        if pos in starts:
            xs = [x + (e if starts[pos] else 0.0) + names["loop.step"][starts[pos]] for x, e in zip(xs, embedded)]
        w = _Tensors(source, prefix % i)
        xs = [LAYERS[arch](x, w, raw, i, k) for x, k in zip(xs, kept)]
    x = torch.stack([x[-1] for x in xs])
    if arch == "Qwen3":
        logits = (_rms(x, eps) * names["model.norm.weight"]) @ embed.T
    elif arch == "Kudazen":
        logits = (_rms(x.reshape(len(x), raw["norm"]["groups"], -1), eps).reshape(x.shape) * names["final.norm"]) @ embed.T
    elif arch == "Nazulorn":
        x = x.reshape(len(x), raw["streams"], -1).sum(1)
        logits = (_rms(x, eps) * names["final.norm"]) @ names["head"].T * raw["logit_scale"]
    elif arch == "Siparax":
        cap = raw["logit_softcap"]
        logits = cap * torch.tanh(_layer_norm(x, names["final.norm"], names["final.norm.b"], eps) @ names["head"].T / cap)
    else:
        head = names["head"] * raw["logit_scale"] if arch == "Nifalorn" else embed
        logits = (_rms(x, eps) * (1.0 + names["final.norm"])) @ head.T
    out = {"logits": logits}
    if case["kind"] == "decode":
        out["score"] = None
    return out
