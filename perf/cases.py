"""What a user has this framework do, as cases whose time is compared between versions of it.

A case is a model (a benchmark shape with fewer layers, so that the weights of a tick are still larger than the L2) and a piece of
serving work through the public entry points: a whole engine run (prompts, then greedy tokens), ticks of one-token lanes over
sessions that already hold a history, or ticks that carry both.  The GGUF families run as Q4_K_M (and Q8_0) checkpoints with f16
pages, the mixer-built designs in bfloat16.

Weights are random, but the embedding of the GGUF models has unit scale and is tied to the output head, as it is in trained models
that the residual stream keeps the token's own direction: the greedy choice is then far from a tie, and comparisons do not
hang on one.  Mixer-built models are fed given tokens instead.

`exact` states the models again in 64-bit torch, without the 8-bit blocks that the reference's matmuls make of activations; these
are most of the distance that the GGUF cases have from it.
"""
import importlib
import json
import math
import struct
import tempfile
from pathlib import Path

import numpy as np
import torch

import __graft_entry__ as entry

entry.load_package()
capi = importlib.import_module(entry.PKG_NAME + "._capi")
engine = importlib.import_module(entry.PKG_NAME + ".engine")
mixer_bench = importlib.import_module(entry.PKG_NAME + ".mixer_bench")
seed_gguf = importlib.import_module(entry.PKG_NAME + ".seed_gguf")

VOCAB = 32000

# name -> (shape, layers, KV tokens, most tokens and lanes of a tick, prefix-cache tokens).  Layers keep the share that the
# output head has in the whole model at a vocabulary of 32000.  The pool holds several states' sessions.
GGUF_MODELS = {
    "tinyllama": ("tinyllama-1.1b", 8, 260000, 512, 64, 0),
    "tinyllama-q8_0": ("tinyllama-1.1b", 8, 260000, 512, 64, 0),
    "smollm3": ("smollm3-3b", 8, 300000, 2048, 64, 0),
    "qwen3": ("qwen3-8b", 4, 400000, 1024, 64, 65536),
    "gemma2": ("gemma2-9b", 2, 1000000, 2048, 64, 0),
    "qwen3moe": ("qwen3-30b-a3b", 2, 600000, 4096, 256, 0),
}
# mixer-built designs, at the width 2048 of their benchmark
MIXERS = {
    "sizilorn": mixer_bench.SHAPES[0],
    "kunonex": mixer_bench.BESIDE_SHAPES[0],
    "tevanex": mixer_bench.EXPERT_SHAPES[0],
    "mamivik": mixer_bench.CONV_SHAPES[0],
}
MIXER_TICK, MIXER_LANES = 2048, 32


def listed():
    return [
        # one user's chat: a single sequence decodes; launches and latency are everything
        dict(name="chat-1-lane", model="smollm3", kind="decode", lanes=1, low=200, high=200, ticks=16, mix=1),
        # the small continuous batch of the first benchmark workload (prompts of 17, 64, 128 and 301 tokens), engine and all
        dict(name="batch-of-4", model="tinyllama", kind="engine", lanes=4, low=17, high=301, spread="log", new=32, quantum=128, budget=256, mix=0),
        # prompts of the second benchmark workload on their way in: 512-token chunks, 2048 tokens a tick, up to the first token
        dict(name="ragged-prompts", model="smollm3", kind="engine", lanes=64, low=32, high=1024, spread="even", new=1, quantum=512, budget=2048, mix=2),
        # the same sequences while they generate: 64 one-token lanes at ragged histories
        dict(name="ragged-decode", model="smollm3", kind="decode", lanes=64, low=32, high=1152, ticks=8, mix=2),
        # requests that share a cached 2048-token prefix: suffixes, then a few tokens each
        dict(name="shared-prefix", model="qwen3", kind="engine", lanes=32, low=16, high=256, spread="even", prefix=2048, new=6, quantum=512, budget=1024, mix=3),
        # long documents with sliding-window and global layers, head size 256
        dict(name="long-prompts", model="gemma2", kind="engine", lanes=6, low=256, high=8192, spread="lognormal", new=1, quantum=512, budget=2048, mix=4),
        # generation over such histories: the K/V pages are most of what is read
        dict(name="long-decode", model="gemma2", kind="decode", lanes=64, low=256, high=8192, spread="lognormal", ticks=4, mix=5),
        # a busy server of sparse experts: prompt chunks beside many decoding lanes in every tick
        dict(name="experts-mixed", model="qwen3moe", kind="mixed", lanes=96, low=64, high=1024, prompts=4, chunk=331, ticks=3, mix=6),
        # the mixer-built designs: ragged prompts, then generation
        dict(name="sizilorn-turn", model="sizilorn", kind="turn", lanes=16, low=48, high=1024, ticks=12, mix=7),
        dict(name="kunonex-turn", model="kunonex", kind="turn", lanes=16, low=48, high=1024, ticks=12, mix=8),
        dict(name="tevanex-turn", model="tevanex", kind="turn", lanes=16, low=48, high=1024, ticks=12, mix=9),
        dict(name="mamivik-turn", model="mamivik", kind="turn", lanes=16, low=48, high=1024, ticks=12, mix=10),
    ]


def draw(rng):
    def log(lo, hi):
        return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49))))))

    mix = rng.randrange(100, 1 << 20)
    kind = rng.choice(["decode", "decode", "engine", "engine", "mixed", "turn", "turn"])
    if kind == "decode":
        model = rng.choice(["tinyllama", "tinyllama-q8_0", "smollm3", "smollm3", "qwen3", "gemma2", "qwen3moe"])
        if model == "gemma2":
            return dict(model=model, kind=kind, lanes=log(1, 48), low=256, high=log(512, 8192), spread="lognormal", ticks=log(2, 4), mix=mix)
        high = log(40, 1900 if model.startswith("tinyllama") else 4000)
        lanes = log(1, min(64, max(2, 60000 // high)))
        return dict(model=model, kind=kind, lanes=lanes, low=log(1, high), high=high, ticks=log(2, 12), mix=mix)
    if kind == "engine":
        model = rng.choice(["tinyllama", "tinyllama-q8_0", "smollm3", "smollm3", "qwen3", "gemma2", "qwen3moe"])
        if model == "gemma2":
            return dict(model=model, kind=kind, lanes=log(1, 5), low=256, high=log(600, 8000), spread="lognormal", new=1, quantum=512, budget=2048, mix=mix)
        high = log(24, 1500)
        lanes = log(1, min(48, max(2, 24000 // high)))
        quantum = rng.choice([128, 256, 512])
        case = dict(model=model, kind=kind, lanes=lanes, low=log(3, high), high=high, spread=rng.choice(["even", "log"]), new=log(1, 12),
                    quantum=quantum, budget=min(GGUF_MODELS[model][3], quantum * rng.choice([1, 2, 4])), mix=mix)
        if model == "qwen3" and rng.random() < 0.5:
            case.update(prefix=16 * log(8, 160))
        return case
    if kind == "mixed":
        model = rng.choice(["qwen3moe", "qwen3moe", "smollm3"])
        prompts = log(1, 4)
        return dict(model=model, kind=kind, lanes=log(1, 60), low=log(16, 512), high=log(512, 900), prompts=prompts, chunk=log(9, 480), ticks=log(1, 3), mix=mix)
    high = log(24, 1500)
    lanes = log(1, min(MIXER_LANES, max(2, 9000 // high)))
    return dict(model=rng.choice(list(MIXERS)), kind="turn", lanes=lanes, low=log(2, high), high=high, ticks=log(2, 12), mix=mix)


def lengths(case):
    """History or prompt length of every lane: part of the case, not of its inputs."""
    n, lo, hi = case["lanes"], case["low"], case["high"]
    if case["mix"] == 0:
        return [17, 64, 128, 301]
    r = np.random.default_rng(case["mix"])
    spread = case.get("spread", "even")
    if spread == "lognormal":
        x = r.lognormal(math.log(3000.0), 0.6, n)
    elif spread == "log":
        x = np.exp(r.uniform(math.log(lo), math.log(hi + 1), n))
    else:
        x = r.integers(min(lo, hi), hi + 1, n)
    return [int(min(hi, max(min(lo, hi), round(float(v))))) for v in x]


# ------------------------------------------------------------------------------------------------------------ models

_models = {}


def gguf_spec(name):
    shape, layers = GGUF_MODELS[name][:2]
    kind = dict(matrix_type=capi.TYPE_Q8_0, high_type=capi.TYPE_Q8_0) if name.endswith("q8_0") else {}
    return seed_gguf.scaled(shape, layers=layers, vocab=VOCAB, tied=True, **kind)


def checkpoint(name, folder):
    if name in MIXERS:
        return mixer_bench.write_checkpoint(Path(folder) / name, MIXERS[name])
    spec = gguf_spec(name)
    plan = [(n, dims, kind, 1.0 if n == "token_embd.weight" and spec.arch != "gemma2" else std) for n, dims, kind, std in seed_gguf.tensor_plan(spec)]
    return seed_gguf._write_file(Path(folder) / (name + ".gguf"), seed_gguf._meta(spec), plan, spec, 0)


def loaded(name):
    """The model as a server keeps it: loaded once, used for every request."""
    if name not in _models:
        with tempfile.TemporaryDirectory() as tmp:
            path = checkpoint(name, tmp)
            if name in MIXERS:
                _models[name] = engine.Model.load(path, kv_capacity_tokens=65536, max_batch_tokens=MIXER_TICK, max_batch_lanes=MIXER_LANES, state_slots=MIXER_LANES)
            else:
                _, _, kv, tokens, lanes, prefix = GGUF_MODELS[name]
                _models[name] = engine.Model.load_gguf(path, kv_capacity_tokens=kv, max_batch_tokens=tokens, max_batch_lanes=lanes, prefix_capacity_tokens=prefix)
    return _models[name]


def ids(rng, n):
    return rng.integers(3, VOCAB, size=n).astype(np.uint32)


def inputs(case, seed):
    """The token ids of every part of a case."""
    rng = np.random.default_rng([int(seed) & 0xFFFFFFFF, case["mix"]])
    prefix = ids(rng, case.get("prefix", 0))
    texts = [np.concatenate([prefix, ids(rng, n)]) for n in lengths(case)]
    chunks = [ids(rng, case["chunk"] * case["ticks"]) for _ in range(case.get("prompts", 0))]
    given = ids(rng, (case.get("ticks", 0), case["lanes"]))
    return prefix, texts, chunks, given


def feed(model, sessions, texts, most):
    """Whole texts into sessions that hold nothing, in packed ticks of up to `most` tokens."""
    at, todo = [0] * len(texts), list(range(len(texts)))
    lanes_most = 32
    while todo:
        lanes, room = [], most
        for i in todo[:lanes_most]:
            n = min(room, len(texts[i]) - at[i])
            if n == 0:
                break
            lanes.append((sessions[i], texts[i][at[i]:at[i] + n], at[i]))
            at[i] += n
            room -= n
        model.forward_batch(lanes, want_logits=False)
        todo = [i for i in todo if at[i] < len(texts[i])]


def prepare(case, seed):
    model = loaded(case["model"])
    prefix, texts, chunks, given = inputs(case, seed)
    state = dict(case=case, model=model, texts=texts, chunks=chunks, given=given)
    if case["kind"] == "engine":
        state["engine"] = engine.Engine(model, max_active_sequences=case["lanes"], scheduler_token_budget=case["budget"], prefill_token_quantum=case["quantum"],
                                        queue_capacity=case["lanes"], record_logits=True)
        state["engine"].keep_trace(False)
        if len(prefix):  # the prefix is in the cache before its users arrive
            session = model.new_session()
            model.reset_session_for_prompt(session, prefix)
            at = len(session)
            while at < len(prefix):
                n = min(len(prefix) - at, GGUF_MODELS[case["model"]][3])
                model.forward_batch([(session, prefix[at:at + n], at)], want_logits=False)
                at += n
            model.publish_prompt_prefix(session, prefix)
            session.close()
    elif case["kind"] in ("decode", "mixed"):
        state["sessions"] = [model.new_session() for _ in texts]
        feed(model, state["sessions"], texts, GGUF_MODELS[case["model"]][3])
    return state


# ------------------------------------------------------------------------------------------------------------ one pass

def run_engine(state):
    case, eng = state["case"], state["engine"]
    requests = [engine.Request(t, case["new"], publish_prompt_prefix=False) for t in state["texts"]]
    numbers = eng.submit(requests, atomic_batch=True)
    eng.run()
    tokens = np.stack([eng.result(n)["tokens"] for n in numbers])
    logits = np.stack([eng.logits(n) for n in numbers])
    for n in numbers:
        eng.release(n)
    return dict(tokens=tokens, logits=logits)


def run_decode(state):
    """Every history continues greedily in a fork of its session, so that the history itself stays."""
    model, ticks = state["model"], state["case"]["ticks"]
    forks = [s.fork_prefix(len(t)) for s, t in zip(state["sessions"], state["texts"])]
    at = [len(t) for t in state["texts"]]
    tokens = state["given"][0]
    out = []
    for k in range(ticks):
        logits, tokens = model.forward_batch([(f, tokens[i:i + 1], at[i] + k) for i, f in enumerate(forks)], want_logits=k == ticks - 1)
        out.append(tokens)
    for f in forks:
        f.close()
    return dict(tokens=np.stack(out), logits=logits)


def run_mixed(state):
    """Ticks that carry a chunk of every new prompt beside one token of every running sequence."""
    model, case = state["model"], state["case"]
    n = case["chunk"]
    forks = [s.fork_prefix(len(t)) for s, t in zip(state["sessions"], state["texts"])]
    fresh = [model.new_session() for _ in state["chunks"]]
    tokens = state["given"][0]
    for k in range(case["ticks"]):
        lanes = [(f, tokens[i:i + 1], len(t) + k) for i, (f, t) in enumerate(zip(forks, state["texts"]))]
        lanes += [(s, c[k * n:(k + 1) * n], k * n) for s, c in zip(fresh, state["chunks"])]
        logits, tokens = model.forward_batch(lanes, want_logits=k == case["ticks"] - 1)
    for s in forks + fresh:
        s.close()
    return dict(tokens=tokens, logits=logits)


def run_turn(state):
    """Prompts into new sessions, then the given tokens one by one."""
    model, case, texts, given = state["model"], state["case"], state["texts"], state["given"]
    sessions = [model.new_session() for _ in texts]
    feed(model, sessions, texts, MIXER_TICK)
    for k in range(case["ticks"]):
        logits, _ = model.forward_batch([(s, given[k, i:i + 1], len(texts[i]) + k) for i, s in enumerate(sessions)], want_logits=k == case["ticks"] - 1)
    for s in sessions:
        s.close()
    return dict(logits=logits)


RUN = {"engine": run_engine, "decode": run_decode, "mixed": run_mixed, "turn": run_turn}


def run(state):
    return RUN[state["case"]["kind"]](state)


# ------------------------------------------------------------------------------------------------------------ work

def work(case):
    """Weights once per tick, cached keys and values once per tick and query tile at most (counted once per tick), logits out."""
    lens, kind = lengths(case), case["kind"]
    prefix = case.get("prefix", 0)
    if kind == "engine":
        prompt, steps = sum(lens), case["new"] - 1
        prompt_ticks = -(-prompt // case["budget"])
        spans = [(prefix, prefix + n) for n in lens]
    elif kind == "turn":
        prompt, steps = sum(lens), case["ticks"]
        prompt_ticks = -(-prompt // MIXER_TICK)
        spans = [(0, n) for n in lens]
    else:
        prompt, steps, prompt_ticks, spans = case["ticks"] * case.get("chunk", 0) * case.get("prompts", 0), case["ticks"], 0, []
        if prompt:
            spans = [(0, case["chunk"] * case["ticks"])] * case["prompts"]
    decode = steps * len(lens)
    pairs = sum((a + 1 + b) * (b - a) / 2 for a, b in spans)                     # (query, key) pairs of prompts
    steps_keys = sum(prefix + n + k + 1 for n in lens for k in range(steps))     # and of one-token lanes
    keys = steps_keys + sum(b for _, b in spans)
    if case["model"] in MIXERS:
        s = MIXERS[case["model"]]
        per_token, shared, banks = 0, 0, 0
        for name, (shape, _, _) in mixer_bench.tensor_shapes(s).items():
            if len(shape) < 2 or "embed" in name or name.endswith("conv") or "canon" in name:
                continue
            n = math.prod(shape)
            if ".mlp.e" in name:
                banks += n
                per_token += n * s.top / s.experts
            else:
                shared += n
                per_token += n
        runs = s.runs if hasattr(s, "runs") else 2 * s.pairs
        if hasattr(s, "loop"):
            f = runs / (2 * s.pairs)
            per_token, shared = per_token * f, shared * f
        attending = {"sizilorn": 0.5, "kunonex": 0.5, "tevanex": 0.5, "mamivik": 1.0}[case["model"]] * runs
        tick = 2 * (shared + banks)
        flops_pair = 4 * s.heads * s.dim * attending
        bytes_key = 4 * (s.kv_heads * s.dim if case["model"] != "kunonex" else s.kv_rank / 2) * attending
        head = VOCAB * s.width
        per_token -= head
    else:
        spec = gguf_spec(case["model"])
        h = spec.hidden
        attn = h * spec.head_dim * (2 * spec.q_heads + 2 * spec.kv_heads)
        ffn = 3 * h * (spec.expert_ffn * spec.experts_used if spec.experts else spec.ffn)
        per_token = spec.layers * (attn + ffn)
        sizes = seed_gguf.weight_bytes(spec)
        routed = max(len(lens), (prompt + decode) / max(1, prompt_ticks + steps))     # rows of a tick, on average
        touched = 1 - (1 - spec.experts_used / spec.experts) ** routed if spec.experts else 0
        tick = sizes["all_experts"] - sizes["experts_only"] * (1 - touched)
        flops_pair = 4 * spec.q_heads * spec.head_dim * spec.layers
        bytes_key = 4 * spec.kv_heads * spec.head_dim * spec.layers
        head = VOCAB * h
    rows = len(lens) * (steps + (1 if kind in ("engine", "turn") else 0)) + (case["ticks"] * case["prompts"] if kind == "mixed" else 0)
    ticks = prompt_ticks + steps
    out = 4 * VOCAB * (len(lens) * (case["new"] if kind == "engine" else 1))
    return {"bytes": ticks * tick + bytes_key * keys + out,
            "flops": 2 * per_token * (prompt + decode) + 2 * head * rows + flops_pair * (pairs + steps_keys)}


def tolerance(case):
    # GGUF models make 8-bit blocks of every matmul's input, as the reference does: a sum in another order moves single blocks by
    # a step, and each such step changes what comes behind it.  They are 0.9 to 2.3 percent from the 64-bit statement, which
    # makes no blocks.  Mixer-built models round matmul inputs to bfloat16 and are 0.2 to 0.5 percent from it.
    return {"rel": 0.02, "max": 0.2} if case["model"] in MIXERS else {"rel": 0.03, "max": 0.3, "differ": 0.01}


# ------------------------------------------------------------------------------------------------------------ 64 bits

F64 = torch.float64


def unpack_blocks(raw, kind, rows, cols):
    """The published GGML block formats as 64-bit numbers on the GPU."""
    def half(a):
        return a.contiguous().view(torch.float16).to(F64)

    if kind == capi.TYPE_F32:
        return torch.from_numpy(np.frombuffer(raw, np.float32).copy()).cuda().to(F64).reshape(rows, cols)
    b = torch.from_numpy(np.frombuffer(raw, np.uint8).copy()).cuda()
    if kind == capi.TYPE_Q8_0:
        b = b.reshape(-1, 34)
        return (half(b[:, :2]) * b[:, 2:].contiguous().view(torch.int8).to(F64)).reshape(rows, cols)
    if kind == capi.TYPE_Q4_K:
        b = b.reshape(-1, 144)
        d, dmin, s = half(b[:, 0:2]), half(b[:, 2:4]), b[:, 4:16].to(torch.int32)
        scale = torch.cat([s[:, 0:4] & 63, (s[:, 8:12] & 15) | ((s[:, 0:4] >> 6) << 4)], 1)
        least = torch.cat([s[:, 4:8] & 63, (s[:, 8:12] >> 4) | ((s[:, 4:8] >> 6) << 4)], 1)
        q = b[:, 16:].reshape(-1, 4, 1, 32)
        q = torch.cat([q & 15, q >> 4], 2).reshape(-1, 8, 32)
        return ((d * scale)[:, :, None] * q - (dmin * least)[:, :, None]).reshape(rows, cols)
    if kind != capi.TYPE_Q6_K:
        raise ValueError("block format %d" % kind)
    b = b.reshape(-1, 210)
    low, high = b[:, :128].reshape(-1, 2, 2, 32), b[:, 128:192].reshape(-1, 2, 1, 32)
    low = torch.cat([low & 15, low >> 4], 2)                                   # quarters 0 .. 3 of each half of 128
    high = torch.cat([(high >> (2 * k)) & 3 for k in range(4)], 2)
    q = (low.to(torch.int32) | (high.to(torch.int32) << 4)) - 32
    scale = b[:, 192:208].contiguous().view(torch.int8).to(F64) * half(b[:, 208:210])
    return (q.reshape(-1, 16, 16) * scale[:, :, None]).reshape(rows, cols)


def rms(x, eps):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps)


def turn_half(x, pos, dims, freq, times=1.0):
    """x [T, heads, dim]: pairs (i, i + dims / 2) turn."""
    a = pos[:, None, None].to(F64) * freq
    c, s, n = torch.cos(a) * times, torch.sin(a) * times, dims // 2
    u, v = x[..., :n], x[..., n:dims]
    return torch.cat([u * c - v * s, v * c + u * s, x[..., dims:]], -1)


def turn_pairs(x, pos, dims, freq, times=1.0):
    """x [T, heads, dim]: pairs (2i, 2i + 1) turn."""
    a = pos[:, None, None].to(F64) * freq
    c, s = torch.cos(a) * times, torch.sin(a) * times
    u, v = x[..., 0:dims:2], x[..., 1:dims:2]
    return torch.cat([torch.stack([u * c - v * s, v * c + u * s], -1).flatten(-2), x[..., dims:]], -1)


def attend(q, k, v, scale, first, softcap=0.0, window=0, sink=None):
    """q [n, H, d] at positions first ..; k, v [m, G, *] from position 0.  Returns [n, H, e]."""
    n, H, _ = q.shape
    k, v = (x.repeat_interleave(H // x.shape[1], 1).transpose(0, 1) for x in (k, v))
    out = torch.empty(H, n, v.shape[2], dtype=F64, device=q.device)
    for a in range(0, n, 512):
        b, end = min(n, a + 512), first + min(n, a + 512)
        lo = max(0, first + a - window + 1) if window else 0
        s = torch.matmul(q[a:b].transpose(0, 1), k[:, lo:end].transpose(1, 2)) * scale
        if softcap:
            s = softcap * torch.tanh(s / softcap)
        p = torch.arange(first + a, end, device=q.device)[:, None] - torch.arange(lo, end, device=q.device)[None]
        s = s.masked_fill((p < 0) | ((p >= window) if window else (p < 0)), -math.inf)
        if sink is not None:
            s = torch.cat([s, sink[:, None, None].expand(H, b - a, 1)], 2)
        w = torch.softmax(s, -1)
        out[:, a:b] = torch.matmul(w[:, :, :end - lo], v[:, lo:end])
    return out.transpose(0, 1)


class ExactGguf:
    """The decoder families over packed lanes with 64-bit keys and values per lane."""

    def __init__(self, name):
        self.s = s = gguf_spec(name)
        with tempfile.TemporaryDirectory() as tmp:
            data = np.memmap(checkpoint(name, tmp), np.uint8, "r")
            plan = seed_gguf.tensor_plan(s)
            size = [seed_gguf._tensor_bytes(dims, kind) for _, dims, kind, _ in plan]
            padded = [(n + 31) // 32 * 32 for n in size]
            at = len(data) - sum(padded)
            self.w = {}
            for (n, dims, kind, _), take, step in zip(plan, size, padded):
                self.w[n] = unpack_blocks(data[at:at + take].tobytes(), kind, math.prod(dims[:-1]) if len(dims) > 1 else 1, dims[-1])
                if len(dims) == 3:
                    self.w[n] = self.w[n].reshape(dims).to(torch.float32)  # block formats hold few bits: exact, and half the room
                at += step
            del data
        if s.arch in ("llama", "smollm3"):  # these files keep the rotated pairs of q and k side by side
            for l in range(s.layers):
                for x, heads in (("attn_q", s.q_heads), ("attn_k", s.kv_heads)):
                    n = "blk.%d.%s.weight" % (l, x)
                    self.w[n] = self.w[n].reshape(heads, -1, 2, s.hidden).transpose(1, 2).reshape(-1, s.hidden)
        self.freq = s.theta ** (-2.0 * torch.arange(s.head_dim // 2, dtype=F64, device="cuda") / s.head_dim)

    def experts(self, x, p):
        s = self.s
        best, chosen = torch.topk(x @ self.w[p + "ffn_gate_inp.weight"].T, s.experts_used, 1)
        weight, out = torch.softmax(best, 1), torch.zeros_like(x)
        for e in range(s.experts):
            t, j = torch.nonzero(chosen == e, as_tuple=True)
            if len(t):
                gate, up, down = (self.w[p + "ffn_%s_exps.weight" % n][e].to(F64) for n in ("gate", "up", "down"))
                out[t] += weight[t, j][:, None] * ((torch.nn.functional.silu(x[t] @ gate.T) * (x[t] @ up.T)) @ down.T)
        return out

    def __call__(self, lanes, caches):
        """lanes: (token ids, start) each; caches: a dict per lane.  Logits of every lane's last token."""
        s, w = self.s, self.w
        lens = [len(t) for t, _ in lanes]
        tokens = torch.from_numpy(np.concatenate([t for t, _ in lanes]).astype(np.int64)).cuda()
        pos = torch.cat([torch.arange(a, a + n) for n, (_, a) in zip(lens, lanes)]).cuda()
        h = w["token_embd.weight"][tokens] * (math.sqrt(s.hidden) if s.arch == "gemma2" else 1.0)
        cuts = np.cumsum([0] + lens)
        for l in range(s.layers):
            p = "blk.%d." % l
            x = rms(h, s.eps) * w[p + "attn_norm.weight"]
            q, k, v = ((x @ w[p + "attn_%s.weight" % n].T).reshape(len(x), -1, s.head_dim) for n in "qkv")
            if s.arch.startswith("qwen3"):
                q, k = rms(q, s.eps) * w[p + "attn_q_norm.weight"], rms(k, s.eps) * w[p + "attn_k_norm.weight"]
            if s.arch != "smollm3" or (l + 1) % 4:
                q, k = turn_half(q, pos, s.head_dim, self.freq), turn_half(k, pos, s.head_dim, self.freq)
            o = []
            for i, (_, a) in enumerate(lanes):
                c, r = caches[i], slice(int(cuts[i]), int(cuts[i + 1]))
                c[l] = [torch.cat([old[:a], new[r]]) for old, new in zip(c[l], (k, v))] if l in c else [k[r], v[r]]
                o.append(attend(q[r], *c[l], s.head_dim ** -0.5, a, s.attn_softcap if s.arch == "gemma2" else 0.0, s.window if s.arch == "gemma2" and l % 2 == 0 else 0))
            o = torch.cat(o).reshape(len(x), -1) @ w[p + "attn_output.weight"].T
            if s.arch == "gemma2":
                o = rms(o, s.eps) * w[p + "post_attention_norm.weight"]
            h = h + o
            x = rms(h, s.eps) * w[p + "ffn_norm.weight"]
            if s.experts:
                o = self.experts(x, p)
            else:
                gate = x @ w[p + "ffn_gate.weight"].T
                gate = torch.nn.functional.gelu(gate, approximate="tanh") if s.arch == "gemma2" else torch.nn.functional.silu(gate)
                o = (gate * (x @ w[p + "ffn_up.weight"].T)) @ w[p + "ffn_down.weight"].T
            if s.arch == "gemma2":
                o = rms(o, s.eps) * w[p + "post_ffw_norm.weight"]
            h = h + o
        z = (rms(h[torch.from_numpy(cuts[1:] - 1).cuda()], s.eps) * w["output_norm.weight"]) @ w["token_embd.weight"].T
        return s.final_softcap * torch.tanh(z / s.final_softcap) if s.arch == "gemma2" else z

    def feed(self, texts, caches):
        out = []
        for t, c in zip(texts, caches):
            for a in range(0, len(t), 4096):
                z = self([(t[a:a + 4096], a)], [c])
            out.append(z)
        return torch.cat(out)


def exact_gguf(case, seed):
    model = ExactGguf(case["model"])
    prefix, texts, chunks, given = inputs(case, seed)
    caches = [{} for _ in texts]
    if case["kind"] == "engine":
        if len(prefix):
            model.feed([prefix], caches[:1])
            for c in caches[1:]:
                c.update(caches[0])
            shared = [dict(c) for c in caches]
            z = torch.cat([model([(t[len(prefix):], len(prefix))], [c]) for t, c in zip(texts, shared)])
            caches = shared
        else:
            z = model.feed(texts, caches)
        rows, tokens = [z], [z.argmax(1)]
        for k in range(case["new"] - 1):
            t = tokens[-1].cpu().numpy()
            z = model([(t[i:i + 1], len(x) + k) for i, x in enumerate(texts)], caches)
            rows.append(z)
            tokens.append(z.argmax(1))
        return dict(tokens=torch.stack(tokens, 1), logits=torch.stack(rows, 1))
    model.feed(texts, caches)
    fresh, n, tokens, out = [{} for _ in chunks], case.get("chunk", 0), given[0], []
    for k in range(case["ticks"]):
        z = model([(tokens[i:i + 1], len(t) + k) for i, t in enumerate(texts)], caches)
        if chunks:
            z = torch.cat([z, model([(c[k * n:(k + 1) * n], k * n) for c in chunks], fresh)])
        tokens = z.argmax(1).cpu().numpy()
        out.append(tokens)
    return dict(tokens=np.stack(out) if case["kind"] == "decode" else tokens, logits=z)


def bend(dims, base, factor, original, fast, slow):
    """YaRN: frequencies stretched where a pair turns seldom, kept where it turns often; and the factor of cosine and sine."""
    i = torch.arange(dims // 2, dtype=F64, device="cuda")
    f = base ** (-2.0 * i / dims)
    lo, hi = (dims * math.log(original / (2 * math.pi * t)) / (2 * math.log(base)) for t in (fast, slow))
    lo, hi = max(math.floor(lo), 0.0), min(math.ceil(hi), dims - 1.0)
    r = ((i - lo) / max(hi - lo, 0.001)).clamp(0, 1)
    return f / factor * r + f * (1 - r), 0.1 * math.log(factor) + 1.0


def stretch(dims, base, factor, low, high, original):
    """Long wavelengths divided by `factor`, short ones kept, a blend in between."""
    f = base ** (-2.0 * torch.arange(dims // 2, dtype=F64, device="cuda") / dims)
    turns = original * f / (2 * math.pi)
    s = ((turns - low) / (high - low)).clamp(0, 1)
    return (1 - s) * f / factor + s * f


class ExactMixer:
    """The mixer-built designs over whole sequences, padded to one length: x [lanes, T, width]; recurrences row by row."""

    def __init__(self, name):
        self.s = s = MIXERS[name]
        self.cfg = mixer_bench.config_of(s)
        self.w = {}
        with tempfile.TemporaryDirectory() as tmp:
            raw = (checkpoint(name, tmp) / "model.safetensors").read_bytes()
        (n,) = struct.unpack("<Q", raw[:8])
        for key, t in json.loads(raw[8:8 + n]).items():
            lo, hi = t["data_offsets"]
            self.w[key] = torch.from_numpy(np.frombuffer(raw, np.int16, (hi - lo) // 2, 8 + n + lo).copy()).cuda().view(torch.bfloat16).reshape(t["shape"])
        self.eps = self.cfg["norm"]["eps"]

    def t(self, name):
        return self.w[name].to(F64)

    def mat(self, x, name):
        return x @ self.t(name).T

    def heads(self, x, name, n):
        y = self.mat(x, name)
        return y.reshape(*y.shape[:2], n, -1)

    def each(self, f, *a):
        return torch.stack([f(*x) for x in zip(*a)])

    def conv(self, x, taps):
        K = taps.shape[1]
        padded = torch.nn.functional.pad(x, (0, 0, K - 1, 0))
        return sum(padded[:, j:j + x.shape[1]] * taps[:, j] for j in range(K))

    def shift(self, h, mu):
        prev = torch.nn.functional.pad(h, (0, 0, 1, 0))[:, :-1]
        return h + (prev - h) * mu

    def gated(self, x, p, act):
        return self.mat(act(self.mat(x, p + "gate")) * self.mat(x, p + "up"), p + "down")

    # ---- Sizilorn

    def wkv(self, h, p, m):
        H, d = m["heads"], m["dim"]
        mix = {x: self.shift(h, self.t(p + "mu." + x)) for x in "rkvgw"}
        r, k, v = (self.heads(mix[x], p + x, H) for x in "rkv")
        w = torch.exp(-torch.exp(self.mat(torch.tanh(self.mat(mix["w"], p + "w1")), p + "w2") + self.t(p + "w0"))).reshape(r.shape)
        u, S, o = self.t(p + "u")[:, :, None], torch.zeros(len(h), H, d, d, dtype=F64, device="cuda"), torch.empty_like(v)
        for i in range(h.shape[1]):
            kv = k[:, i, :, :, None] * v[:, i, :, None, :]
            o[:, i] = (r[:, i, :, None, :] @ (S + u * kv))[..., 0, :]
            S = w[:, i, :, :, None] * S + kv
        return self.mat(rms(o, self.eps).flatten(2) * self.t(p + "norm") * torch.nn.functional.silu(self.mat(mix["g"], p + "g")), p + "o")

    def parallel(self, h, p, m):
        a, b = m["left"], m["right"]
        L, R, pos = p + "left.", p + "right.", torch.arange(h.shape[1], device="cuda")
        q, k, v = self.heads(h, L + "q", a["heads"]), self.heads(h, L + "k", a["kv_heads"]), self.heads(h, L + "v", a["kv_heads"])
        f = stretch(a["rot"]["dims"], a["rot"]["base"], **a["rot"]["scaling"])
        q, k = (torch.stack([turn_pairs(y, pos, a["rot"]["dims"], f) for y in rms(x, self.eps) * self.t(L + n)]) for x, n in ((q, "q.norm"), (k, "k.norm")))
        o = self.each(lambda q, k, v: attend(q, k, v, a["scale"], 0), q, k, v) * torch.sigmoid(self.mat(h, L + "g"))[..., None]
        left = self.mat(o.flatten(2), L + "o")
        act = torch.nn.functional.silu
        q, k, v = (act(self.conv(self.mat(h, R + x), self.t(R + x + ".conv"))).reshape(*h.shape[:2], n, -1) for x, n in (("q", b["kv_heads"]), ("k", b["kv_heads"]), ("v", b["heads"])))
        unit = lambda x: x * torch.rsqrt((x * x).sum(-1, keepdim=True) + 1e-6)  # noqa: E731
        group = b["heads"] // b["kv_heads"]
        q, k = (unit(q) / math.sqrt(b["dim"])).repeat_interleave(group, 2), unit(k).repeat_interleave(group, 2)
        beta = torch.sigmoid(self.mat(h, R + "b"))
        g = torch.exp(-torch.exp(self.t(R + "A_log")) * torch.nn.functional.softplus(self.mat(h, R + "a") + self.t(R + "dt_bias")))
        S, o = torch.zeros(len(h), b["heads"], b["dim"], b["vdim"], dtype=F64, device="cuda"), torch.empty_like(v)
        for i in range(h.shape[1]):
            S = S * g[:, i, :, None, None]
            u = beta[:, i, :, None] * (v[:, i] - (k[:, i, :, None, :] @ S)[..., 0, :])
            S = S + k[:, i, :, :, None] * u[:, :, None, :]
            o[:, i] = (q[:, i, :, None, :] @ S)[..., 0, :]
        o = rms(o, self.eps) * self.t(R + "norm") * act(self.heads(h, R + "g", b["heads"]))
        right = self.mat(o.flatten(2), R + "o")
        return 0.5 * (rms(left, self.eps) * self.t(L + "out") + rms(right, self.eps) * self.t(R + "out"))

    def sizilorn(self, tokens):
        norm = lambda n, x: torch.tanh(self.t(n + ".alpha") * x) * self.t(n) + self.t(n + ".b")  # noqa: E731
        x, dim = self.t("embed")[tokens], self.cfg["token_side"]["dim"]
        for i, layer in enumerate(self.cfg["layers"]):
            p = "l%d." % i
            x = x + (self.wkv if layer["type"] == "wkv" else self.parallel)(norm(p + "norm1", x), p + "mix.", layer["mixer"])
            x = x + self.gated(norm(p + "norm2", x), p + "mlp.", torch.nn.functional.silu)
            e = self.w["side.embed"][tokens][..., i * dim:(i + 1) * dim].to(F64)
            y = self.mat(torch.nn.functional.gelu(self.mat(x, p + "side.gate"), approximate="tanh") * e, p + "side.proj")
            x = x + rms(y, self.eps) * self.t(p + "side.norm")
        return lambda rows: norm("final.norm", x[rows])

    # ---- Kunonex

    def latent(self, h, p, m):
        H = m["heads"]
        q = self.heads(rms(self.mat(h, p + "dq"), self.eps) * self.t(p + "dq.norm"), p + "uq", H)
        c = rms(self.mat(h, p + "dkv"), self.eps) * self.t(p + "dkv.norm")
        o = self.each(lambda q, k, v: attend(q, k, v, m["scale"], 0), q, self.heads(c, p + "uk", H), self.heads(c, p + "uv", H))
        return self.mat((o * torch.sigmoid(self.mat(h, p + "g"))[..., None]).flatten(2), p + "o")

    def mingru(self, h, p, m):
        z, u = torch.sigmoid(self.mat(h, p + "z") + self.t(p + "z.b")), self.mat(h, p + "x") + self.t(p + "x.b")
        new, S, out = z * torch.where(u >= 0, u + 0.5, torch.sigmoid(u)), torch.zeros_like(z[:, 0]), torch.empty_like(z)
        for i in range(h.shape[1]):
            S = (1 - z[:, i]) * S + new[:, i]
            out[:, i] = S
        return self.mat(out * torch.nn.functional.silu(self.mat(h, p + "g")), p + "o")

    def kunonex(self, tokens):
        width = self.cfg["width"]

        def norm(n, x):
            c = x - x.mean(-1, keepdim=True)
            return rms(c, self.eps) * self.t(n)

        a = torch.arange(tokens.shape[1], device="cuda")[:, None] * 10000.0 ** (-2.0 * (torch.arange(width, dtype=F64, device="cuda") // 2) / width)
        x0 = x = norm("embed.norm", self.t("embed")[tokens] + torch.where(torch.arange(width, device="cuda") % 2 == 1, torch.cos(a), torch.sin(a)))
        loop = self.cfg["loop"]
        lo, hi = loop["start"], loop["stop"]
        order = [(i, None) for i in range(lo)] + [(i, t) for t in range(loop["times"]) for i in range(lo, hi)] + [(i, None) for i in range(hi, len(self.cfg["layers"]))]
        for i, t in order:
            if t is not None and i == lo:
                x = self.mat(torch.cat([x, x0], -1), "loop.in") + self.t("loop.step")[t]
            p, layer = "l%d." % i, self.cfg["layers"][i]
            h = norm(p + "norm1", x)
            y = (self.mingru if layer["type"] == "mingru" else self.latent)(self.shift(h, self.t(p + "shift")), p + "mix.", layer["mixer"])
            z, c = self.mat(h, p + "mlp.up") + self.t(p + "mlp.up.b"), self.t(p + "mlp.act")
            z = c[0] * rms(z, self.eps) + c[1] * rms(z ** 2, self.eps) + c[2] * rms(z ** 3, self.eps) + c[3]
            x = x + y + self.mat(z, p + "mlp.down") + self.t(p + "mlp.down.b")
        return lambda rows: norm("final.norm", x[rows])

    # ---- Tevanex

    def capped(self, h, p, m, sink):
        pos, rot = torch.arange(h.shape[1], device="cuda"), m["rot"]
        q, k, v = (self.mat(h, p + x) + self.t(p + x + ".b") for x in "qkv")
        q, k = rms(q, self.eps) * self.t(p + "q.norm"), rms(k, self.eps) * self.t(p + "k.norm")
        q, k, v = (x.reshape(*h.shape[:2], n, -1) for x, n in ((q, m["heads"]), (k, m["kv_heads"]), (v, m["kv_heads"])))
        if sink:
            f = rot["base"] ** (-2.0 * torch.arange(rot["dims"] // 2, dtype=F64, device="cuda") / rot["dims"])
            q, k = (torch.stack([turn_half(y, pos, rot["dims"], f) for y in x]) for x in (q, k))
        else:
            f, times = bend(rot["dims"], rot["base"], **rot["scaling"])
            q, k = (torch.stack([turn_pairs(y, pos, rot["dims"], f, times) for y in x]) for x in (q, k))
        # every length here is within the first chunk
        o = self.each(lambda q, k, v: attend(q, k, v, m["scale"], 0, 0.0 if sink else m["softcap"], 0, self.t(p + "sink") if sink else None), q, k, v).flatten(2)
        return self.mat(o if sink else o * torch.sigmoid(self.mat(h, p + "g")), p + "o") + self.t(p + "o.b")

    def mlstm(self, h, p, m):
        H, d, e, cap = m["heads"], m["dim"], m["vdim"], m["gate_cap"]
        q, k, v = self.heads(h, p + "q", H) / math.sqrt(d), self.heads(h, p + "k", H), self.heads(h, p + "v", H)
        i, f = (cap * torch.tanh((self.mat(h, p + x) + self.t(p + x + ".b")) / cap) for x in "if")
        f = torch.nn.functional.logsigmoid(f)
        S, n, top = torch.zeros(len(h), H, d, e, dtype=F64, device="cuda"), torch.zeros(len(h), H, d, dtype=F64, device="cuda"), torch.zeros(len(h), H, dtype=F64, device="cuda")
        o = torch.empty_like(v)
        for t in range(h.shape[1]):
            new = torch.maximum(f[:, t] + top, i[:, t])
            keep, write = torch.exp(f[:, t] + top - new)[..., None], torch.exp(i[:, t] - new)[..., None]
            S = keep[..., None] * S + (write * k[:, t])[..., None] * v[:, t, :, None, :]
            n, top = keep * n + write * k[:, t], new
            den = torch.maximum((n * q[:, t]).sum(-1).abs(), torch.exp(-top)) + 1e-6
            o[:, t] = (q[:, t, :, None, :] @ S)[..., 0, :] / den[..., None]
        return self.mat(rms(o, self.eps).flatten(2) * self.t(p + "norm") * torch.sigmoid(self.mat(h, p + "g")), p + "o")

    def clamped(self, x, p, limit):
        g, u = self.mat(x, p + "gate").clamp(max=limit), self.mat(x, p + "up").clamp(-limit, limit)
        return self.mat(g * torch.sigmoid(1.702 * g) * (u + 1), p + "down")

    def moe(self, h, p, m):
        x = h.flatten(0, 1)
        weight, chosen = torch.topk(torch.sigmoid(self.mat(x, p + "router")), m["router"]["top"], 1)
        out = torch.sigmoid(self.mat(x, p + "shared.sg")) * self.clamped(x, p + "shared.", m["shared"]["limit"])
        for e in range(m["router"]["experts"]):
            t, j = torch.nonzero(chosen == e, as_tuple=True)
            if len(t):
                out[t] += self.clamped(weight[t, j][:, None] * x[t], p + "e%d." % e, m["expert"]["limit"])
        return out.reshape(h.shape)

    def tevanex(self, tokens):
        norm = lambda n, x: rms(x, self.eps) * self.t(n)  # noqa: E731
        x, m = self.t("embed")[tokens] * self.cfg["embedding"]["scale"], self.cfg["residual_mult"]
        for i, layer in enumerate(self.cfg["layers"]):
            p = "l%d." % i
            y = self.mlstm(x, p + "mix.", layer["mixer"]) if layer["type"] == "mlstm" else self.capped(x, p + "mix.", layer["mixer"], layer["type"] == "attention")
            x = x + m * norm(p + "norm1", y)
            x = x + m * norm(p + "norm2", self.moe(x, p + "mlp.", layer["mlp"]))
        return lambda rows: norm("final.norm", x[rows])

    # ---- Mamivik

    def scaled(self, h, p, m):
        a, b = m["left"], m["right"]
        L, R, pos = p + "left.", p + "right.", torch.arange(h.shape[1], device="cuda")
        q, k = ((self.mat(h, L + x) + self.t(L + x + ".b")).reshape(*h.shape[:2], n, -1) for x, n in (("q", a["heads"]), ("k", a["kv_heads"])))
        f = a["rot"]["base"] ** (-2.0 * torch.arange(a["rot"]["dims"] // 2, dtype=F64, device="cuda") / a["rot"]["dims"])
        turn = lambda x: turn_half(x, pos, a["rot"]["dims"], f)  # noqa: E731
        left = self.mat(self.each(lambda q, k: attend(turn(q), turn(k), k, a["scale"], 0, 0.0, a["mask"]["size"]), q, k).flatten(2), L + "o")
        H = b["heads"]
        r, k, v = (self.heads(h, R + x, H) for x in "rkv")
        w = torch.exp(-math.exp(-0.5) * torch.sigmoid(self.mat(torch.tanh(self.mat(h, R + "w1")), R + "w2") + self.t(R + "w0"))).reshape(r.shape)
        c = torch.sigmoid(self.mat(h, R + "a") + self.t(R + "a.b")).reshape(r.shape)
        u = k * torch.rsqrt((k * k).sum(-1, keepdim=True) + 1e-6)
        S, o = torch.zeros(len(h), H, b["dim"], b["dim"], dtype=F64, device="cuda"), torch.empty_like(v)
        for i in range(h.shape[1]):
            seen = u[:, i, :, None, :] @ S
            S = w[:, i, :, :, None] * S - (c[:, i] * u[:, i])[..., None] * seen + k[:, i, :, :, None] * v[:, i, :, None, :]
            o[:, i] = (r[:, i, :, None, :] @ S)[..., 0, :]
        right = self.mat(rms(o, self.eps).flatten(2) * self.t(R + "norm") * torch.sigmoid(self.mat(h, R + "g")), R + "o")
        return m["left_scale"] * left + m["right_scale"] * right

    def turned_latent(self, h, p, m):
        H, d, r, rank = m["heads"], m["dim"], m["rot_dim"], m["kv_rank"]
        pos = torch.arange(h.shape[1], device="cuda")
        f, times = bend(r, m["rot"]["base"], **m["rot"]["scaling"])
        turn = lambda x: turn_half(x, pos, r, f, times)  # noqa: E731
        q = self.heads(rms(self.mat(h, p + "dq"), self.eps) * self.t(p + "dq.norm"), p + "uq", H)
        down = self.mat(h, p + "dkv")
        c = rms(down[..., :rank], self.eps) * self.t(p + "dkv.norm")
        k, v = self.heads(c, p + "uk", H), self.heads(c, p + "uv", H)

        def one(q, k, v, part):
            k = torch.cat([k, turn(part[:, None]).expand(-1, H, -1)], -1)
            return attend(torch.cat([q[..., :d], turn(q[..., d:])], -1), k, v, m["scale"], 0, 0.0, m["mask"]["size"], self.t(p + "sink"))

        return self.mat(self.each(one, q, k, v, down[..., rank:]).flatten(2) * torch.sigmoid(self.mat(h, p + "g")), p + "o")

    def mamivik(self, tokens):
        norm = lambda n, x: rms(x, self.eps) * self.t(n)  # noqa: E731
        x = self.t("embed")[tokens]
        for i, layer in enumerate(self.cfg["layers"]):
            p = "l%d." % i
            h = norm(p + "norm1", x)
            h = h + self.conv(h, self.t(p + "canon1"))
            x = x + (self.scaled if layer["type"] == "parallel" else self.turned_latent)(h, p + "mix.", layer["mixer"])
            x = x + self.gated(norm(p + "norm2", x), p + "mlp.", lambda z: torch.nn.functional.gelu(z, approximate="tanh"))
        return lambda rows: norm("final.norm", x[rows])

    def logits(self, texts):
        """Of every text's last token; shorter texts are padded behind their end, which no earlier row sees."""
        T = max(len(t) for t in texts)
        tokens = torch.from_numpy(np.stack([np.pad(t.astype(np.int64), (0, T - len(t))) for t in texts])).cuda()
        name = self.cfg["architecture"].lower()
        rows = (torch.arange(len(texts), device="cuda"), torch.tensor([len(t) - 1 for t in texts], device="cuda"))
        z = self.mat(getattr(self, name)(tokens)(rows), "head") * self.cfg.get("logit_scale", 1.0)
        cap = self.cfg.get("logit_softcap")
        return cap * torch.tanh(z / cap) if cap else z


@torch.no_grad()
def exact(case, seed):
    if case["model"] not in MIXERS:
        return exact_gguf(case, seed)
    _, texts, _, given = inputs(case, seed)
    model = ExactMixer(case["model"])
    return dict(logits=model.logits([np.concatenate([t, given[:, i]]) for i, t in enumerate(texts)]))
