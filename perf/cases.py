"""What a user has this library do, as cases that can be timed and compared.

A pass serves one batch of sequences through the public entry points: the prompts in one step, then one token of
every sequence a step (`Model.step`), the logits kept; or, on the 32-bit engine, `Model.generate` and then one step
that scores what it produced.  The tokens that are fed are given (a recorded continuation, as in a replay or when
scoring), so that two implementations are compared on the same inputs.  Slots are taken at a pass's begin and given
back at its end, so a pass can be run again.

Weights are random (a function of a fixed seed and of the tensor's name), four layers of each architecture at the
sizes of the benchmark; the model is what a program keeps, the prompts are the inputs.  Where experts are chosen, a
token's embedding carries the directions of two of them and the router reads those, as trained routers specialise:
with routers of noise alone, a choice now and then rests on the last bit of a sum, and a token's logits with it.
"""
import gc
import json
import math
import re

import numpy as np
import torch

import janus_b200
from janus_b200.config import resolve_architecture
from janus_b200.engine import StepEntry
from janus_b200.weights import RandomCheckpoint

WEIGHT_SEED = 5
NORM_STD = 0.1
ROUTED = ("mugedra", "buludra", "forisun", "mibezen")     # architectures with experts

# ---------------------------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------------------------
SIZE_1B = dict(width=2048, ff=8192, heads=32, kv_heads=8, dim=64)
SIZE_2K = dict(width=2048, ff=8192, heads=16, kv_heads=4, dim=128)
SIZE_4K = dict(width=4096, ff=14336, heads=32, kv_heads=8, dim=128)


def _case(name, model, size, sequences, shortest, longest, new, vocab=32000, window=512, dtype="bfloat16", score=False,
          temperature=0.0, std=0.02, tied=False):
    return dict(name=name, model=model, **size, vocab=vocab, window=window, sequences=sequences, shortest=shortest,
                longest=longest, new=new, dtype=dtype, score=score, temperature=temperature, std=std, tied=tied)


def listed():
    return [
        # a chat turn of one user on the 1B layers: a short prompt, then token after token; latency
        _case("llama_1b_one_sequence", "llama", SIZE_1B, 1, 23, 23, 16, vocab=128256, tied=True),
        # a full batch of short requests on the 1B layers: 64 sequences of unequal lengths
        _case("llama_1b_64_sequences", "llama", SIZE_1B, 64, 5, 130, 12, vocab=128256, tied=True),
        # the headline: eight sequences on the 8B layers, prompts of unequal lengths
        _case("llama_8b_8_sequences", "llama", SIZE_4K, 8, 150, 701, 16, vocab=128256),
        # a long document on the 8B layers: one prompt, a few tokens of answer
        _case("llama_8b_long_prompt", "llama", SIZE_4K, 1, 8190, 8190, 4, vocab=128256),
        # scoring whole texts: the logits of every token of a batch of prompts
        _case("llama_2k_score", "llama", SIZE_2K, 6, 65, 400, 0, score=True),
        # the true 32-bit engine through `generate`, greedy, then the scores of what it said
        _case("llama_float32_generate", "llama", SIZE_2K, 4, 17, 90, 16, dtype="float32"),
        # the other architectures, prompts of unequal lengths and single tokens: lightning and differential attention ...
        _case("zivitar_2k_4_sequences", "zivitar", SIZE_2K, 4, 211, 1100, 12),
        # ... state-space mixers, window attention and latents, eight sequences on the larger size ...
        _case("ramolix_4k_8_sequences", "ramolix", SIZE_4K, 8, 33, 600, 12),
        # ... chunked attention beside the delta rule with experts: one long prompt and its answer ...
        _case("mugedra_2k_one_sequence", "mugedra", SIZE_2K, 1, 1500, 1500, 12, std=0.006),
        # ... gated linear attention, matrix memories, sinks, shared and chosen experts ...
        _case("buludra_2k_8_sequences", "buludra", SIZE_2K, 8, 40, 511, 12, std=0.006),
        # ... latent attention with dynamic tanh around every sublayer, many sequences ...
        _case("forisun_2k_16_sequences", "forisun", SIZE_2K, 16, 9, 257, 12, std=0.006),
        # ... latent queries, distance bias, learned sinks; long prompts of two sequences on the larger size
        _case("mibezen_4k_2_sequences", "mibezen", SIZE_4K, 2, 1023, 2049, 8, std=0.006),
    ]


def draw(rng):
    """A model, a width and a batch from the ranges above: widths of 1,024 to 4,096, one to 64 sequences of one to
    4,000 tokens, at most 6,000 tokens a prompt step (3,000 of the architectures with more work a token)."""
    model = rng.choice(["llama", "llama", "llama", "zivitar", "ramolix", "mugedra", "buludra", "forisun", "mibezen"])
    heads = rng.choice([8, 12, 16, 20, 24, 32])
    width = 128 * heads
    kv_heads = rng.choice([g for g in (2, 4, 8) if heads % g == 0])
    ff = 64 * int(width * rng.uniform(2.5, 4.0) / 64)
    sequences = int(round(2 ** rng.uniform(0, 6)))
    most = min(4000, (6000 if model == "llama" else 3000) // sequences)
    longest = int(round(math.exp(rng.uniform(math.log(4), math.log(most)))))
    shortest = max(1, int(longest * rng.uniform(0.1, 1.0)))
    dtype, temperature, new = "bfloat16", 0.0, rng.randint(1, 16)
    if model == "llama" and rng.random() < 0.25:
        dtype, temperature = "float32", rng.choice([0.0, 0.8])
        longest, sequences, heads, width, kv_heads, ff = min(longest, 200), min(sequences, 8), 12, 1536, 4, 4096
        shortest = min(shortest, longest)
    score = dtype == "bfloat16" and rng.random() < 0.2 and sequences * longest <= 2500
    return dict(model=model, width=width, ff=ff, heads=heads, kv_heads=kv_heads, dim=128,
                vocab=rng.choice([8000, 32000, 50257, 128256]) if not score else 32000, window=rng.choice([130, 512, 1024]),
                sequences=sequences, shortest=shortest, longest=longest, new=new, dtype=dtype, score=score,
                temperature=temperature, std=0.006 if model in ROUTED else 0.02, tied=model == "llama" and rng.random() < 0.3)


def _config(case):
    """config.json of a case: four layer runs, laid out as the benchmark lays them out."""
    W, F, H, G, d, V, window = (case[k] for k in ("width", "ff", "heads", "kv_heads", "dim", "vocab", "window"))
    m, dense = case["model"], dict(kind="dense", ff=F)
    ramp = dict(factor=4.0, original=4096, fast=32.0, slow=1.0)
    if m == "llama":
        return dict(architectures=["LlamaForCausalLM"], hidden_size=W, num_hidden_layers=4, num_attention_heads=H,
                    num_key_value_heads=G, head_dim=d, intermediate_size=F, vocab_size=V, max_position_embeddings=16384,
                    rms_norm_eps=1e-5, rope_theta=500000.0, tie_word_embeddings=case["tied"],
                    rope_scaling=dict(rope_type="llama3", factor=8.0, low_freq_factor=1.0, high_freq_factor=4.0,
                                      original_max_position_embeddings=8192))
    if m == "zivitar":
        mlp = dict(dense, limit=7.0)
        attention = dict(type="attention", mlp=mlp,
                         mixer=dict(heads=H, kv_heads=G, dim=64, vdim=128, scale=0.125, diff=0.5, conv=4,
                                    mask=dict(size=window, keep_first=4), rot=dict(dims=32, base=10000.0, scaling=ramp)))
        lightning = dict(type="lightning", mlp=mlp, mixer=dict(heads=H, dim=128, vdim=128,
                                                               decay=[1.0 - 2.0 ** (-5 - 3 * h / H) for h in range(H)]))
        return dict(architecture="Zivitar", vocab=V, width=W, norm=dict(eps=1e-5), streams=2, logit_scale=1.0,
                    logit_softcap=30.0, layers=[lightning, attention, attention, attention])
    if m == "ramolix":
        mamba = dict(type="mamba2", mlp=dense, mixer=dict(heads=2 * W // 64, vdim=64, state=128, groups=1, conv=4, norm_groups=1))
        attention = dict(type="attention", mlp=dense,
                         mixer=dict(heads=H, kv_heads=G, dim=128, vdim=128, scale=128 ** -0.5, mask=dict(size=window),
                                    rot=dict(dims=64, base=10000.0, scaling=dict(factor=4.0, low=1.0, high=4.0, original=4096))))
        latent = dict(type="latent_attention", mlp=dense, mixer=dict(heads=H, dim=128, vdim=128, kv_rank=256, scale=128 ** -0.5))
        return dict(architecture="Ramolix", vocab=V, width=W, norm=dict(eps=1e-5), embedding=dict(scale=W ** 0.5),
                    residual_mult=0.7, layers=[mamba, attention, mamba, latent])
    if m == "mugedra":
        layer = dict(type="parallel",
                     mixer=dict(left=dict(heads=H, kv_heads=G, dim=128, vdim=128, scale=128 ** -0.5, softcap=50.0,
                                          mask=dict(size=window), rot=dict(dims=64, base=10000.0, scaling=ramp)),
                                right=dict(heads=H, kv_heads=G, dim=128, vdim=128, conv=4)),
                     mlp=dict(kind="moe", expert=dict(ff=F // 2), router=dict(experts=8, top=2)))
        return dict(architecture="Mugedra", vocab=V, width=W, norm=dict(eps=1e-5), loop=dict(start=1, stop=2, times=2),
                    layers=[layer, layer, layer])
    if m == "buludra":
        side = dict(left=dict(heads=H, kv_heads=G, dim=128, vdim=128, scale=0.5 * 128 ** -0.5, rot=dict(dims=64, base=10000.0)),
                    right=dict(heads=H, dim=128, vdim=128, gate_cap=15.0), left_scale=0.8, right_scale=0.9)
        experts = dict(kind="moe", expert=dict(ff=F // 2), router=dict(experts=8, top=2, groups=dict(count=4, keep=2)),
                       shared=dict(ff=F // 4))
        return dict(architecture="Buludra", vocab=V, width=W, norm=dict(eps=1e-5), logit_softcap=30.0,
                    layers=[dict(type="parallel", mixer=side, mlp=dense),
                            dict(type="attention", mlp=experts, mixer=dict(heads=H, kv_heads=G, dim=128, vdim=128, scale=128 ** -0.5,
                                                                           q_temp=dict(coef=0.1, every=1024))),
                            dict(type="gla", mlp=dense, mixer=dict(heads=H, dim=128, vdim=128, tau=16.0, rank=64)),
                            dict(type="parallel", mixer=side, mlp=experts)])
    latent = dict(heads=H, dim=128, rot_dim=64, vdim=128, kv_rank=512, scale=192 ** -0.5,
                  rot=dict(dims=64, base=10000.0, scaling=ramp))
    experts, kind = dict(kind="moe", expert=dict(ff=F // 2), router=dict(experts=8, top=2)), "latent_attention"
    if m == "forisun":
        experts["router"]["scale"] = 1.5
        return dict(architecture="Forisun", vocab=V, width=W, norm=dict(eps=1e-5), embedding=dict(scale=W ** 0.5),
                    layers=[dict(type=kind, mixer=latent, mlp=dense), dict(type=kind, mixer=latent, mlp=experts),
                            dict(type=kind, mixer=latent, mlp=experts), dict(type=kind, mixer=dict(latent, kv_from=2), mlp=experts)])
    latent["q_rank"] = W * 3 // 4
    chunked = dict(heads=H, kv_heads=G, dim=128, vdim=128, scale=128 ** -0.5, mask=dict(size=4 * window), v_mix=True)
    return dict(architecture="Mibezen", vocab=V, width=W, norm=dict(eps=1e-6), logit_softcap=15.0,
                layers=[dict(type=kind, mixer=latent, mlp=dense), dict(type="attention", mixer=chunked, mlp=experts),
                        dict(type="attention", mixer=chunked, mlp=dense), dict(type=kind, mixer=latent, mlp=experts)])


class _Weights(RandomCheckpoint):
    """Seeded random tensors; with experts, embeddings that name two experts each and routers that look for them."""

    SHARE, GAIN = 3.0, 3.0

    def __init__(self, case):
        config = _config(case)
        arch = resolve_architecture(config)
        super().__init__(arch.weight_specs(arch.config_class.from_dict(config)), WEIGHT_SEED, dtype=case["dtype"],
                         std=case["std"], norm_std=NORM_STD, device="cuda")
        self.routed = case["model"] in ROUTED

    def tensor(self, name):
        t = super().tensor(name)
        if not self.routed or not (name == "embed" or name.endswith(".router")):
            return t
        i, e = torch.arange(t.shape[1], device=t.device), torch.arange(1, 9, device=t.device)[:, None]
        bits = i[None, :] & e
        walsh = 1.0 - 2.0 * ((bits ^ (bits >> 1) ^ (bits >> 2) ^ (bits >> 3)) & 1)        # eight orthogonal rows of +1, -1
        if name != "embed":
            return (walsh * (self.GAIN / t.shape[1])).to(t.dtype)
        v = torch.arange(t.shape[0], device=t.device)
        first, second = v % 8, (v + 1 + (v // 8) % 7) % 8
        return (t.float() + self.std * self.SHARE * (1.3 * walsh[first] + walsh[second])).to(t.dtype)


# ---------------------------------------------------------------------------------------------
# a pass
# ---------------------------------------------------------------------------------------------
_kept = {}       # the model of the case at hand: a program loads it once and serves many batches with it


def _model(case):
    key = json.dumps({k: v for k, v in case.items() if k != "name"}, sort_keys=True)
    if key not in _kept:
        _kept.clear()
        gc.collect()
        torch.cuda.empty_cache()
        room = sum(64 * (n + case["new"] + 64) // 64 for n in _lengths(case)) + 64 * case["sequences"]
        model = janus_b200.load_random(_config(case), seed=WEIGHT_SEED, dtype=case["dtype"], std=case["std"],
                                       norm_std=NORM_STD, max_tokens=room, max_seq_len=case["longest"] + case["new"] + 1,
                                       max_slots=case["sequences"])
        if case["model"] in ROUTED:
            model.engine.model.load(_Weights(case))
        _kept[key] = model
    return _kept[key]


def _lengths(case):
    n, a, b = case["sequences"], case["shortest"], case["longest"]
    return [b if n == 1 else b - (b - a) * i // (n - 1) for i in range(n)]


def _tokens(case, seed):
    """(prompts, for every later step one token per sequence)"""
    g = np.random.default_rng(seed)
    prompts = [g.integers(0, case["vocab"], n) for n in _lengths(case)]
    return prompts, g.integers(0, case["vocab"], (case["new"], case["sequences"]))


def prepare(case, seed):
    prompts, later = _tokens(case, seed)
    return dict(case=case, seed=seed, model=_model(case), prompts=[p.tolist() for p in prompts], later=later.tolist())


def _want(case, n):
    return range(n) if case["score"] else (n - 1,)


def run(state):
    case, model, prompts = state["case"], state["model"], state["prompts"]
    if case["dtype"] == "float32":
        said, _ = model.generate(prompts, max_tokens=case["new"], ignore_eos=True, seed=state["seed"],
                                 temperature=case["temperature"], top_p=0.95 if case["temperature"] > 0 else 1.0)
        prompts = [p + s for p, s in zip(prompts, said)]
    slots = [model.alloc_slot() for _ in prompts]
    if case["dtype"] == "float32":
        n = case["new"]
        scores = model.step([StepEntry(s, p, range(len(p) - n, len(p))) for s, p in zip(slots, prompts)])
        out = dict(tokens=torch.tensor(said), scores=scores)
    else:
        out = dict(prompt=model.step([StepEntry(s, p, _want(case, len(p))) for s, p in zip(slots, prompts)]))
        out["later"] = [model.step([StepEntry(s, (t,), (0,)) for s, t in zip(slots, step)]) for step in state["later"]]
    for s in slots:
        model.free_slot(s)
    return out


# ---------------------------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------------------------
def _mixers(config):
    """Per layer run: (kind of the mixer, its sizes), two entries for two mixers side by side."""
    if "architectures" in config:
        one = dict(heads=config["num_attention_heads"], kv_heads=config["num_key_value_heads"], dim=config["head_dim"],
                   vdim=config["head_dim"])
        return [("attention", one)] * config["num_hidden_layers"]
    runs = list(config["layers"])
    if config.get("loop"):
        runs.insert(1, runs[1])
    out = []
    for layer in runs:
        if layer["type"] == "parallel":
            out += [("attention", layer["mixer"]["left"]), ("state", layer["mixer"]["right"])]
        else:
            out.append((layer["type"], layer["mixer"]))
    return out


def work(case):
    config = _config(case)
    arch = resolve_architecture(config)
    size, B, new, lens = 2 if case["dtype"] == "bfloat16" else 4, case["sequences"], case["new"], _lengths(case)
    T = sum(lens)
    loops = config["loop"]["times"] if config.get("loop") else 1
    dense = expert = n_experts = top = 0.0
    for spec in arch.weight_specs(arch.config_class.from_dict(config)):
        n = math.prod(spec.shape) * (loops if spec.name.startswith("l1.") else 1)
        if re.search(r"\.e\d+\.", spec.name):
            expert, n_experts, top = expert + n, 8, 2
        elif "embed" not in spec.name:
            dense += n
    head = case["vocab"] * case["width"]
    if case["tied"] or case["model"] == "ramolix":
        dense += head
    prompt_rows = T if case["score"] else B
    later_rows = new * B + (new * B if case["dtype"] == "float32" else 0)
    share = lambda tokens: 1.0 - (1.0 - top / n_experts) ** tokens if n_experts else 0.0     # noqa: E731  experts that are read
    steps_bytes = (dense + expert * share(T)) + new * (dense + expert * share(B))
    passes = 2 if case["dtype"] == "float32" else 1                # generate, then the scores in one step
    if passes == 2:
        steps_bytes += dense
    tokens = T * passes + new * B * (passes if passes == 2 else 1)
    active = dense - head + (expert * top / n_experts if n_experts else 0.0)
    flops, numbers = 2.0 * active * tokens + 2.0 * head * (prompt_rows + later_rows), steps_bytes
    for kind, m in _mixers(config):
        H, d, e = m["heads"], m.get("dim", m.get("state", 0)), m["vdim"]
        if kind in ("state", "lightning", "gla", "mamba2"):
            flops += 4.0 * H * d * e * tokens
            numbers += 2 * 4 / size * H * d * e * B * (1 + new)
            continue
        window = (m.get("mask") or {}).get("size") or 1 << 30
        cached = m["kv_rank"] + m.get("rot_dim", 0) if "kv_rank" in m else m["kv_heads"] * (2 * d + e if "diff" in m else d + e)
        pair = 2.0 * H * (d + m.get("rot_dim", 0) + e) * (2 if "diff" in m else 1)
        seen = sum(min(i + 1, window) for n in lens for i in range(n))
        later = sum(min(n + i + 1, window) for n in lens for i in range(new))
        flops += pair * (seen + later) * passes
        numbers += cached * (later + 2 * tokens)
    numbers += (prompt_rows + later_rows) * case["vocab"] * 4 / size
    return dict(bytes=size * numbers, flops=flops)


def tolerance(case):
    """Other orders of 32-bit sums, bfloat16 where the engine rounds to it: measured against `exact`."""
    if case["dtype"] == "float32":
        return dict(rel=2e-5, max=1e-3, differ=0.01)
    return dict(rel=0.03, max=0.2)


# ---------------------------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------------------------
def exact(case, seed):
    if case["temperature"] > 0.0:
        return None                          # drawn tokens depend on the library's random numbers
    prompts, later = _tokens(case, seed)
    plain = _Plain(_config(case), case, "cuda")
    if case["dtype"] != "float32":
        rows = plain([list(p) + later[:, i].tolist() for i, p in enumerate(prompts)])
        out = dict(prompt=torch.cat([r[list(_want(case, len(p)))] for r, p in zip(rows, prompts)]))
        out["later"] = [torch.stack([r[len(p) + j] for r, p in zip(rows, prompts)]) for j in range(case["new"])]
        return out
    texts = [list(p) for p in prompts]
    for _ in range(case["new"]):
        for t, r in zip(texts, plain(texts)):
            t.append(int(r[-1].argmax()))
    rows = plain(texts)
    n = case["new"]
    return dict(tokens=torch.tensor([t[len(t) - n:] for t in texts]), scores=torch.cat([r[len(r) - n:] for r in rows]))


def _rms(x, eps):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps)


def _silu(z):
    return z * torch.sigmoid(z)


class _Plain:
    """Every architecture of the cases on whole sequences in float64, a layer at a time for all sequences."""

    def __init__(self, config, case, device):
        self.c, self.case, self.device = config, case, device
        self.ck = _Weights(case)
        self.eps = config.get("rms_norm_eps") or config["norm"]["eps"]

    def w(self, name):
        return self.ck.tensor(name).double()

    def __call__(self, texts):
        self.lens = [len(t) for t in texts]
        self.pos = torch.cat([torch.arange(n, device=self.device) for n in self.lens]).double()
        ids = torch.tensor([t for text in texts for t in text], device=self.device)
        x = getattr(self, self.case["model"])(ids)
        return list(torch.split(x, self.lens))

    # -- pieces --------------------------------------------------------------------------------
    def lin(self, name, h):
        return h @ self.w(name).T

    def gated(self, p, h, act=_silu, names=("gate", "up", "down")):
        return self.lin(p + names[2], act(self.lin(p + names[0], h)) * self.lin(p + names[1], h))

    def rotate(self, x, dims, f, amplitude=1.0, neighbours=False):
        angle = self.pos[:, None] * torch.tensor(f, dtype=torch.float64, device=self.device)
        c, s = (torch.cos(angle) * amplitude)[:, None], (torch.sin(angle) * amplitude)[:, None]
        out = x.clone()
        a = slice(0, dims, 2) if neighbours else slice(0, dims // 2)
        b = slice(1, dims, 2) if neighbours else slice(dims // 2, dims)
        out[..., a], out[..., b] = x[..., a] * c - x[..., b] * s, x[..., b] * c + x[..., a] * s
        return out

    def ramped(self, x, rot, neighbours=False):
        """Rotation whose frequencies go over to 1/factor of themselves along a ramp."""
        dims, base, s = rot["dims"], rot["base"], rot.get("scaling")
        f = [base ** (-2.0 * i / dims) for i in range(dims // 2)]
        if s is None:
            return self.rotate(x, dims, f, 1.0, neighbours)
        pair = lambda turns: dims * math.log(s["original"] / (2 * math.pi * turns)) / (2 * math.log(base))     # noqa: E731
        lo, hi = max(math.floor(pair(s["fast"])), 0), min(math.ceil(pair(s["slow"])), dims - 1)
        ramp = [min(max((i - lo) / max(hi - lo, 0.001), 0.0), 1.0) for i in range(dims // 2)]
        f = [v / s["factor"] * r + v * (1.0 - r) for v, r in zip(f, ramp)]
        return self.rotate(x, dims, f, 0.1 * math.log(s["factor"]) + 1.0, neighbours)

    def banded(self, x, dims, base, factor, low, high, original):
        """Rotation whose frequencies are scaled by bands of wavelength."""
        f = []
        for i in range(dims // 2):
            v = base ** (-2.0 * i / dims)
            wave = 2.0 * math.pi / v
            s = min(max((original / wave - low) / (high - low), 0.0), 1.0)
            f.append((1.0 - s) * v / factor + s * v)
        return self.rotate(x, dims, f)

    def attend(self, q, k, v, scale, window=0, keep_first=0, chunk=0, cap=0.0, sink=None, slopes=None):
        """q [T, H, d], k [T, G, d], v [T, G, e] of all sequences -> [T, H, e]; every key at or before the query, of
        its window (or among the kept first), of its chunk."""
        out, at = [], 0
        for n in self.lens:
            i = torch.arange(n, device=self.device)
            back = i[:, None] - i[None, :]
            seen = back >= 0
            if window:
                seen = seen & ((back < window) | (i < keep_first)[None, :])
            if chunk:
                seen = seen & ((i // chunk)[:, None] == (i // chunk)[None, :])
            heads = []
            for h in range(q.shape[1]):
                g = h // (q.shape[1] // k.shape[1])
                s = (q[at:at + n, h] @ k[at:at + n, g].T) * scale
                if cap:
                    s = cap * torch.tanh(s / cap)
                if slopes is not None:
                    s = s - slopes[h] * back
                s = s.masked_fill(~seen, -math.inf)
                if sink is not None:
                    s = torch.cat([s, sink[h].expand(n, 1)], dim=1)
                heads.append(torch.softmax(s, -1)[:, :n] @ v[at:at + n, g])
            out.append(torch.stack(heads, 1))
            at += n
        return torch.cat(out)

    def walk(self, step, state, *inputs):
        """A recurrence over the sequences side by side: step(state, *a token's inputs) -> (state, output)."""
        B, L = len(self.lens), max(self.lens)
        inside = torch.arange(L, device=self.device)[None, :] < torch.tensor(self.lens, device=self.device)[:, None]

        def padded(x):
            out = x.new_zeros((B, L) + x.shape[1:])
            out[inside] = x
            return out
        inputs = [padded(x) for x in inputs]
        outs = []
        for t in range(L):
            state, o = step(state, *(x[:, t] for x in inputs))
            outs.append(o)
        return torch.stack(outs, 1)[inside]

    def zeros(self, *shape):
        return torch.zeros((len(self.lens),) + shape, dtype=torch.float64, device=self.device)

    def conv(self, u, w):
        """Short causal convolution, the last column of w [C, taps] meets the current token."""
        out = []
        for x in torch.split(u, self.lens):
            full = torch.cat([x.new_zeros(w.shape[1] - 1, x.shape[1]), x])
            out.append(sum(full[j:j + len(x)] * w[:, j] for j in range(w.shape[1])))
        return torch.cat(out)

    def chosen(self, p, h, picks, weights, on_input=False):
        out = torch.zeros_like(h)
        for x in range(8):
            t, j = (picks == x).nonzero(as_tuple=True)
            if len(t):
                s = weights[t, j][:, None]
                y = self.gated(f"{p}e{x}.", h[t] * s if on_input else h[t])
                out[t] += y if on_input else y * s
        return out

    # -- architectures -------------------------------------------------------------------------
    def llama(self, ids):
        c, eps = self.c, self.eps
        T, H, G, d, s = len(ids), c["num_attention_heads"], c["num_key_value_heads"], c["head_dim"], c["rope_scaling"]
        turn = lambda x: self.banded(x, d, c["rope_theta"], s["factor"], s["low_freq_factor"], s["high_freq_factor"],    # noqa: E731
                                     s["original_max_position_embeddings"])
        x = self.w("model.embed_tokens.weight")[ids]
        for i in range(c["num_hidden_layers"]):
            p = f"model.layers.{i}."
            h = _rms(x, eps) * self.w(p + "input_layernorm.weight")
            q, k, v = (self.lin(p + f"self_attn.{n}_proj.weight", h).view(T, -1, d) for n in "qkv")
            x = x + self.lin(p + "self_attn.o_proj.weight", self.attend(turn(q), turn(k), v, d ** -0.5).reshape(T, H * d))
            h = _rms(x, eps) * self.w(p + "post_attention_layernorm.weight")
            x = x + self.gated(p + "mlp.", h, names=("gate_proj.weight", "up_proj.weight", "down_proj.weight"))
        h = _rms(x, eps) * self.w("model.norm.weight")
        return self.lin("model.embed_tokens.weight" if c["tie_word_embeddings"] else "lm_head.weight", h)

    def zivitar(self, ids):
        eps, T = self.eps, len(ids)
        x = self.w("embed")[ids]
        streams = [x] * self.c["streams"]
        for i, layer in enumerate(self.c["layers"]):
            p, m = f"l{i}.", layer["mixer"]
            for q in (1, 2):
                into, out, mix = self.w(p + f"hc{q}.in"), self.w(p + f"hc{q}.out"), self.w(p + f"hc{q}.mix")
                h = _rms(sum(a * s for a, s in zip(into, streams)), eps) * self.w(p + f"norm{q}")
                if q == 2:
                    limit = layer["mlp"]["limit"]
                    g = torch.clamp(self.lin(p + "mlp.gate", h), max=limit)
                    u = torch.clamp(self.lin(p + "mlp.up", h), -limit, limit)
                    y = self.lin(p + "mlp.down", g * torch.sigmoid(1.702 * g) * (u + 1.0))
                elif layer["type"] == "lightning":
                    y = self._lightning(h, p + "mix.", m)
                else:
                    y = self._differential(h, p + "mix.", m, T)
                streams = [sum(mix[s, t] * streams[s] for s in range(len(streams))) + out[t] * y for t in range(len(streams))]
        logits = self.lin("head", _rms(sum(streams), eps) * self.w("final.norm")) * self.c["logit_scale"]
        return self.c["logit_softcap"] * torch.tanh(logits / self.c["logit_softcap"])

    def _lightning(self, h, p, m):
        T, H, d, e = len(h), m["heads"], m["dim"], m["vdim"]
        q, k, v = (_silu(self.lin(p + n, h)).view(T, H, -1) for n in "qkv")
        decay = torch.tensor(m["decay"], dtype=torch.float64, device=self.device)[:, None, None]

        def step(S, q, k, v):
            S = decay * S + k[..., :, None] * v[..., None, :]
            return S, torch.einsum("bhde,bhd->bhe", S, q)
        o = self.walk(step, self.zeros(H, d, e), q, k, v).reshape(T, H * e)
        return self.lin(p + "o", _rms(o, self.eps) * self.w(p + "norm") * torch.sigmoid(self.lin(p + "g", h)))

    def _differential(self, h, p, m, T):
        H, G, d, e, diff = m["heads"], m["kv_heads"], m["dim"], m["vdim"], m["diff"]
        q, k, v = (self.conv(self.lin(p + n, h), self.w(p + n + ".conv")) for n in "qkv")
        q, k = (self.ramped(t.view(T, -1, d), m["rot"]).view(T, -1, 2, d) for t in (q, k))
        v = v.view(T, G, e)
        lam = (torch.exp((self.w(p + "lq1") * self.w(p + "lk1")).sum()) - torch.exp((self.w(p + "lq2") * self.w(p + "lk2")).sum()) + diff)
        maps = [self.attend(q[:, :, j], k[:, :, j], v, m["scale"], m["mask"]["size"], m["mask"]["keep_first"]) for j in (0, 1)]
        o = _rms(maps[0] - lam * maps[1], self.eps) * (1.0 - diff)
        return self.lin(p + "o", o.reshape(T, H * e))

    def ramolix(self, ids):
        eps, T, mult = self.eps, len(ids), self.c["residual_mult"]
        x = self.w("embed")[ids] * self.c["embedding"]["scale"]
        gelu = lambda z: 0.5 * z * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (z + 0.044715 * z ** 3)))       # noqa: E731
        for i, layer in enumerate(self.c["layers"]):
            p, m = f"l{i}.", layer["mixer"]
            a = p + "mix."
            if layer["type"] == "mamba2":
                y = self._mamba(x, a, m)
            elif layer["type"] == "attention":
                H, G, d, r = m["heads"], m["kv_heads"], m["dim"], m["rot"]
                q, k = (self.lin(a + n, x) + self.w(a + n + ".b") for n in "qk")
                v = k.view(T, G, d)
                turn = lambda t: self.banded(t, r["dims"], r["base"], **r["scaling"])                       # noqa: E731
                q, k = (turn((_rms(t, eps) * self.w(a + n + ".norm")).view(T, -1, d)) for t, n in ((q, "q"), (k, "k")))
                y = self.lin(a + "o", self.attend(q, k, v, m["scale"], m["mask"]["size"]).reshape(T, H * d))
            else:
                H, d, e = m["heads"], m["dim"], m["vdim"]
                c = _rms(self.lin(a + "dkv", x), eps) * self.w(a + "dkv.norm")
                o = self.attend(self.lin(a + "q", x).view(T, H, d), self.lin(a + "uk", c).view(T, H, d),
                                self.lin(a + "uv", c).view(T, H, e), m["scale"])
                y = self.lin(a + "o", o.reshape(T, H * e))
            x = x + mult * _rms(y, eps) * self.w(p + "norm1")
            x = x + mult * _rms(self.gated(p + "mlp.", x, gelu), eps) * self.w(p + "norm2")
        return self.lin("embed", _rms(x, eps) * self.w("final.norm"))

    def _mamba(self, x, p, m):
        T, H, P, N = len(x), m["heads"], m["vdim"], m["state"]
        z, u, dt = torch.split(self.lin(p + "in", x), [H * P, H * P + 2 * N, H], dim=1)
        u = _silu(self.conv(u, self.w(p + "conv")) + self.w(p + "conv.b"))
        v, b, c = u[:, :H * P].view(T, H, P), u[:, H * P:H * P + N], u[:, H * P + N:]
        dt = torch.logaddexp(dt + self.w(p + "dt_bias"), torch.zeros_like(dt))
        A = -torch.exp(self.w(p + "A_log"))

        def step(S, v, b, c, dt):
            S = torch.exp(A * dt)[..., None, None] * S + (dt[..., None] * b[:, None, :])[..., None] * v[:, :, None, :]
            return S, torch.einsum("bhnp,bn->bhp", S, c)
        y = self.walk(step, self.zeros(H, N, P), v, b, c, dt) + self.w(p + "D")[:, None] * v
        y = _rms(y.reshape(T, H * P) * _silu(z), self.eps) * self.w(p + "norm")
        return self.lin(p + "o", y)

    def mugedra(self, ids):
        eps, loop = self.eps, self.c["loop"]

        def norm(x, name):
            x = x - x.mean(-1, keepdim=True)
            return _rms(x, eps) * self.w(name)
        x = start = self.w("embed")[ids]
        order = list(range(loop["start"]))
        for n in range(loop["times"]):
            order += [i if n == 0 else -i for i in range(loop["start"], loop["stop"])]
        for i in order + list(range(loop["stop"], len(self.c["layers"]))):
            if i < 0:
                x, i = x + start, -i
            layer, p = self.c["layers"][i], f"l{i}."
            h, a = norm(x, p + "norm1"), p + "mix."
            left = self._capped(h, a + "left.", layer["mixer"]["left"])
            right = self._delta(h, a + "right.", layer["mixer"]["right"])
            y = 0.5 * (_rms(left, eps) * self.w(a + "left.out") + _rms(right, eps) * self.w(a + "right.out"))
            x = x + y * self.w(p + "ls1")
            h = norm(x, p + "norm2")
            weights, picks = torch.sigmoid(self.lin(p + "mlp.router", h)).topk(2, dim=-1)
            x = x + self.chosen(p + "mlp.", h, picks, weights, on_input=True) * self.w(p + "ls2")
        return self.lin("head", norm(x, "final.norm"))

    def _capped(self, h, p, m):
        T, H, d, e = len(h), m["heads"], m["dim"], m["vdim"]
        q, k = (self.ramped(_rms(self.lin(p + n, h).view(T, -1, d), self.eps) * self.w(p + n + ".norm"), m["rot"]) for n in "qk")
        o = self.attend(q, k, self.lin(p + "v", h).view(T, -1, e), m["scale"], chunk=m["mask"]["size"], cap=m["softcap"])
        return self.lin(p + "o", o.reshape(T, H * e) * torch.sigmoid(self.lin(p + "g", h)))

    def _delta(self, h, p, m):
        T, H, G, d, e = len(h), m["heads"], m["kv_heads"], m["dim"], m["vdim"]
        q, k, v = (_silu(self.conv(self.lin(p + n, h), self.w(p + n + ".conv"))) for n in "qkv")
        unit = lambda t: (t / torch.sqrt((t * t).sum(-1, keepdim=True) + 1e-6)).repeat_interleave(H // G, dim=1)   # noqa: E731
        q, k, v = unit(q.view(T, G, d)) * d ** -0.5, unit(k.view(T, G, d)), v.view(T, H, e)
        beta = torch.sigmoid(self.lin(p + "b", h))
        z = self.lin(p + "a", h) + self.w(p + "dt_bias")
        decay = torch.exp(-torch.exp(self.w(p + "A_log")) * torch.logaddexp(z, torch.zeros_like(z)))

        def step(S, q, k, v, beta, decay):
            S = decay[..., None, None] * S
            u = beta[..., None] * (v - torch.einsum("bhde,bhd->bhe", S, k))
            S = S + k[..., :, None] * u[..., None, :]
            return S, torch.einsum("bhde,bhd->bhe", S, q)
        o = _rms(self.walk(step, self.zeros(H, d, e), q, k, v, beta, decay), self.eps) * self.w(p + "norm")
        return self.lin(p + "o", o.reshape(T, H * e) * _silu(self.lin(p + "g", h)))

    def buludra(self, ids):
        eps, cap = self.eps, self.c["logit_softcap"]
        x = self.w("embed")[ids]
        for i, layer in enumerate(self.c["layers"]):
            p, m = f"l{i}.", layer["mixer"]
            h, a = _rms(x, eps) * self.w(p + "norm1"), p + "mix."
            if layer["type"] == "attention":
                y = self._tempered(h, a, m)
            elif layer["type"] == "gla":
                y = self._gated_linear(h, a, m)
            else:
                y = (m["left_scale"] * self._sink(h, a + "left.", m["left"])
                     + m["right_scale"] * self._memory(h, a + "right.", m["right"]))
            x = x + y
            h, f = _rms(x, eps) * self.w(p + "norm2"), p + "mlp."
            if layer["mlp"]["kind"] == "dense":
                x = x + self.gated(f, h)
                continue
            s = torch.softmax(self.lin(f + "router", h), -1)
            groups = layer["mlp"]["router"]["groups"]
            best = s.view(len(h), groups["count"], -1).amax(-1).topk(groups["keep"], dim=-1).indices
            kept = torch.zeros(len(h), groups["count"], dtype=torch.bool, device=self.device).scatter_(1, best, True)
            weights, picks = s.masked_fill(~kept.repeat_interleave(8 // groups["count"], dim=1), -1.0).topk(2, dim=-1)
            x = x + (self.chosen(f, h, picks, weights)
                     + self.gated(f + "shared.", h) * torch.sigmoid(self.lin(f + "shared.sg", h)))
        return cap * torch.tanh(self.lin("head", _rms(x, eps) * self.w("final.norm")) / cap)

    def _tempered(self, h, p, m):
        T, d = len(h), m["dim"]
        q, k = (_rms(self.lin(p + n, h).view(T, -1, d), self.eps) * self.w(p + n + ".norm") for n in "qk")
        t = m["q_temp"]
        q = q * (1.0 + t["coef"] * torch.log(torch.floor((self.pos + 1.0) / t["every"]) + 1.0))[:, None, None]
        o = self.attend(q, k, self.lin(p + "v", h).view(T, -1, m["vdim"]), m["scale"])
        return self.lin(p + "o", o.reshape(T, -1))

    def _sink(self, h, p, m):
        T, d, r = len(h), m["dim"], m["rot"]
        q, k = (_rms(self.ramped(self.lin(p + n, h).view(T, -1, d), r), self.eps) for n in "qk")
        o = self.attend(q, k, self.lin(p + "v", h).view(T, -1, m["vdim"]), m["scale"], sink=self.zeros(0).new_zeros(m["heads"], 1))
        return self.lin(p + "o", o.reshape(T, -1))

    def _gated_linear(self, h, p, m):
        T, H, d, e = len(h), m["heads"], m["dim"], m["vdim"]
        q, k, v = (self.lin(p + n, h).view(T, H, -1) for n in "qkv")
        z = self.lin(p + "a2", self.lin(p + "a1", h)) + self.w(p + "a2.b")
        alpha = torch.exp(-torch.logaddexp(-z, torch.zeros_like(z)) / m["tau"]).view(T, H, d)

        def step(S, q, k, v, alpha):
            S = alpha[..., None] * S + k[..., :, None] * v[..., None, :]
            return S, torch.einsum("bhde,bhd->bhe", S, q)
        o = _rms(self.walk(step, self.zeros(H, d, e), q * d ** -0.5, k, v, alpha), self.eps) * self.w(p + "norm")
        return self.lin(p + "o", o.reshape(T, H * e) * _silu(self.lin(p + "g", h)))

    def _memory(self, h, p, m):
        T, H, d, e, cap = len(h), m["heads"], m["dim"], m["vdim"], m["gate_cap"]
        q, k, v = (self.lin(p + n, h).view(T, H, -1) for n in "qkv")
        gi, gf = (cap * torch.tanh((self.lin(p + n, h) + self.w(p + n + ".b")) / cap) for n in "if")
        gf = -torch.logaddexp(-gf, torch.zeros_like(gf))

        def step(state, q, k, v, gi, gf):
            S, n, top = state
            new = torch.maximum(gf + top, gi)
            keep, take = torch.exp(gf + top - new), torch.exp(gi - new)
            S = keep[..., None, None] * S + take[..., None, None] * k[..., :, None] * v[..., None, :]
            n = keep[..., None] * n + take[..., None] * k
            below = torch.maximum((n * q).sum(-1).abs(), torch.exp(-new)) + 1e-6
            return (S, n, new), torch.einsum("bhde,bhd->bhe", S, q) / below[..., None]
        o = self.walk(step, (self.zeros(H, d, e), self.zeros(H, d), self.zeros(H)), q * d ** -0.5, k, v, gi, gf)
        y = _rms(o, self.eps).reshape(T, H * e) * self.w(p + "norm") * torch.sigmoid(self.lin(p + "g", h))
        return self.lin(p + "o", y)

    def forisun(self, ids):
        norm = lambda name, x: torch.tanh(self.w(name + ".alpha") * x) * self.w(name) + self.w(name + ".b")      # noqa: E731
        x = norm("embed.norm", self.w("embed")[ids] * self.c["embedding"]["scale"])
        rows = {}
        for i, layer in enumerate(self.c["layers"]):
            p, m = f"l{i}.", layer["mixer"]
            h = norm(p + "norm1", x)
            if m.get("kv_from") is None:
                rows[i] = self._rows(h, p + "mix.", m)
            q = self.lin(p + "mix.q", h).view(len(h), m["heads"], -1)
            o = self._latent(q, rows[m.get("kv_from", i)], p + "mix.", m)
            x = x + norm(p + "norm1b", self.lin(p + "mix.o", o.reshape(len(h), -1) * torch.sigmoid(self.lin(p + "mix.g", h))))
            h, f = norm(p + "norm2", x), p + "mlp."
            if layer["mlp"]["kind"] == "dense":
                u = self.lin(f + "up", h)
                y = self.lin(f + "down", 0.5 * u * (1.0 + torch.erf(u / math.sqrt(2.0))))
            else:
                s = torch.sigmoid(self.lin(f + "router", h))
                picks = (s + self.w(f + "correction")).topk(2, dim=-1).indices
                y = self.chosen(f, h, picks, s.gather(1, picks) * layer["mlp"]["router"]["scale"])
            x = x + norm(p + "norm2b", y)
        return self.lin("head", norm("final.norm", x))

    def _rows(self, h, p, m, neighbours=False):
        both = self.lin(p + "dkv", h)
        c = _rms(both[:, :m["kv_rank"]], self.eps) * self.w(p + "dkv.norm")
        return c, self.ramped(both[:, None, m["kv_rank"]:], m["rot"], neighbours)

    def _latent(self, q, rows, p, m, neighbours=False):
        T, H, d = len(q), m["heads"], m["dim"]
        q = torch.cat([q[..., :d], self.ramped(q[..., d:], m["rot"], neighbours)], -1)
        k = torch.cat([self.lin(p + "uk", rows[0]).view(T, H, d), rows[1].expand(T, H, -1)], -1)
        return self.attend(q, k, self.lin(p + "uv", rows[0]).view(T, H, -1), m["scale"])

    def mibezen(self, ids):
        eps, cap, T = self.eps, self.c["logit_softcap"], len(ids)
        norm = lambda name, x: _rms(x, eps) * (1.0 + self.w(name))                                               # noqa: E731
        x, first = self.w("embed")[ids], None
        for i, layer in enumerate(self.c["layers"]):
            p, m = f"l{i}.", layer["mixer"]
            h, a, H = norm(p + "norm1", x), p + "mix.", m["heads"]
            if layer["type"] == "latent_attention":
                q = self.lin(a + "uq", _rms(self.lin(a + "dq", h), eps) * self.w(a + "dq.norm")).view(T, H, -1)
                o = self._latent(q, self._rows(h, a, m, True), a, m, True)
            else:
                q, k, v = (self.lin(a + n, h).view(T, -1, m["dim"]) for n in "qkv")
                if first is None:
                    first = v
                else:
                    share = self.w(a + "vmix")
                    v = (1.0 - share) * v + share * first
                slopes = [2.0 ** (-8.0 * (j + 1) / H) for j in range(H)]
                o = self.attend(q, k, v, m["scale"], chunk=m["mask"]["size"], sink=self.w(a + "sink")[:, None], slopes=slopes)
            x = x + self.lin(a + "o", (o * torch.sigmoid(self.lin(a + "g", h))[:, :, None]).reshape(T, -1))
            h, f = norm(p + "norm2", x), p + "mlp."
            if layer["mlp"]["kind"] == "dense":
                x = x + self.lin(f + "down", torch.clamp(self.lin(f + "up", h), min=0.0) ** 2)
            else:
                best, picks = torch.softmax(self.lin(f + "router", h), -1).topk(2, dim=-1)
                x = x + self.chosen(f, h, picks, best / (best.sum(-1, keepdim=True) + 1e-20))
        return cap * torch.tanh(self.lin("head", norm("final.norm", x)) / cap)
