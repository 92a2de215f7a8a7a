"""The work that users have this library do, as cases that can be prepared, run, timed and compared with a computation in 64 bits.

Twelve cases over seven entry points: the Stella-1.5B encoder, the int4 decoder, the hybrid decoder, the latent-attention decoder, the
int4 linear, the paged attention of decode steps and the sampling chain. Sizes are those of the benchmark and of its configurations.
``draw`` spreads the same kinds of case over their ranges.

A model is loaded once per process, as a server does; a case's state holds what a request brings: token ids, the sequences' cache blocks and
state slots with their history already computed by real prompt steps, activations, logits. Shapes follow from the case alone, values from the seed.
The decoders' vocabulary is the decoder benchmarks' (32768); their greedy tokens are the largest of the returned logits, which are compared
instead: between nearly equal logits the larger one is no stable output."""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from logismos_b200 import ops
from logismos_b200.cache import BlockAllocator, SlotAllocator
from logismos_b200.decoder import DecoderModel
from logismos_b200.embed import StellaModel
from logismos_b200.hybrid import HYBRID_SERVING, HybridModel, is_full_attention
from logismos_b200.latent import GLU_ALPHA, GLU_SHIFT, LatentModel
from logismos_b200.sampling import DecodeChain, MinP, MultinomialSampler, TemperatureScale, TopK, TopP
from logismos_b200.synthetic import STELLA_1_5B

VOCAB = 32768
STELLA = STELLA_1_5B
DECODER = dict(STELLA_1_5B, vocab=VOCAB)
HYBRID = dict(HYBRID_SERVING, vocab=VOCAB)
LATENT_LAYER = {"heads": 16, "dim": 128, "vdim": 128, "q_rank": 1024, "kv_rank": 512, "ff": 8192, "scale": 128 ** -0.5, "glu_limit": 7.0}
LATENT = {"vocab": VOCAB, "hidden": 2048, "n_layers": 16, "conv_taps": 4, "rms_eps": 1e-6, "logit_softcap": 15.0, "layers": [LATENT_LAYER] * 16}
PROMPT_TOKENS = 4096  # prompt tokens of one step
EXACT_FLOPS = 4e14    # what 64-bit arithmetic does in less than 20 seconds
INT4_SHAPES = ((1536, 1536), (8960, 1536), (1536, 8960), (151936, 1536))


def listed():
    return [
        # a search query: one short text, where launches and weights count
        {"name": "embed_query", "kind": "embed", "seqs": 1, "lo": 17, "hi": 17},
        # the benchmark's headline batch: eight texts of 32 to 512 tokens
        {"name": "embed_batch", "kind": "embed", "seqs": 8, "lo": 32, "hi": 512},
        # indexing a corpus: many long passages in one call
        {"name": "embed_documents", "kind": "embed", "seqs": 64, "lo": 128, "hi": 512},
        # one chat: a token for a single sequence
        {"name": "chat_token", "kind": "decoder", "decode": 1, "lo": 1200, "hi": 1200, "prompts": 0, "prompt": 0, "prefix": 0},
        # continuous batching: 64 sequences decode while four prompts of 512 tokens continue cached prefixes
        {"name": "ragged_step", "kind": "decoder", "decode": 64, "lo": 256, "hi": 8192, "prompts": 4, "prompt": 512, "prefix": 1024},
        # serving the hybrid decoder: a token for each of 64 sequences
        {"name": "hybrid_decode", "kind": "hybrid", "decode": 64, "lo": 512, "hi": 512, "prompts": 0, "prompt": 0},
        # and the prompts of four new requests
        {"name": "hybrid_prompts", "kind": "hybrid", "decode": 0, "lo": 0, "hi": 0, "prompts": 4, "prompt": 1024},
        # the vocabulary projection of a small batch from int4 weights
        {"name": "int4_vocabulary", "kind": "int4", "n": 151936, "k": 1536, "batch": 4},
        # the attention of one decode step over long and short contexts, with the append of the new token
        {"name": "paged_decode", "kind": "paged", "seqs": 256, "lo": 128, "hi": 32768},
        # serving the latent-attention decoder: a token for each of 64 sequences, and the prompts of four
        {"name": "latent_decode", "kind": "latent", "decode": 64, "lo": 2048, "hi": 2048, "prompts": 0, "prompt": 0},
        {"name": "latent_prompts", "kind": "latent", "decode": 0, "lo": 0, "hi": 0, "prompts": 4, "prompt": 1024},
        # choosing the next tokens of 64 sequences from their logits
        {"name": "sample_tokens", "kind": "sample", "rows": 64, "vocab": 151936, "temperature": 0.8, "top_k": 50, "top_p": 0.95, "min_p": 0.0},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["embed", "embed", "decoder", "decoder", "hybrid", "latent", "int4", "int4", "paged", "sample"])
    if kind == "embed":
        seqs = _log_int(rng, 1, 64)
        lo = rng.randint(4, 256)
        return {"kind": kind, "seqs": seqs, "lo": lo, "hi": rng.randint(lo, 512)}
    if kind in ("decoder", "hybrid", "latent"):
        mode = rng.choice(["decode", "prompts"] + (["both"] if kind == "decoder" else []))
        case = {"kind": kind, "decode": 0, "lo": 0, "hi": 0, "prompts": 0, "prompt": 0}
        if mode != "prompts":
            case["decode"] = _log_int(rng, 1, 64)
            case["lo"] = rng.randint(16, 1024)
            case["hi"] = rng.randint(case["lo"], 2048)
        if mode != "decode":
            case["prompts"] = rng.randint(1, 4)
            case["prompt"] = _log_int(rng, 16, 1024)
        if kind == "decoder":
            case["prefix"] = rng.choice([0, rng.randint(1, 1500)]) if mode != "decode" else 0
        return case
    if kind == "int4":
        n, k = rng.choice(INT4_SHAPES)
        return {"kind": kind, "n": n, "k": k, "batch": _log_int(rng, 1, 64)}
    if kind == "paged":
        lo = rng.randint(1, 256)
        return {"kind": kind, "seqs": _log_int(rng, 1, 256), "lo": lo, "hi": _log_int(rng, lo + 1, 32768)}
    return {"kind": kind, "rows": _log_int(rng, 1, 64), "vocab": _log_int(rng, 4000, 151936), "temperature": round(rng.uniform(0.5, 1.5), 2), "top_k": rng.randint(2, 100),
            "top_p": round(rng.uniform(0.5, 0.99), 2), "min_p": rng.choice([0.0, 0.02])}


# ---- shapes and work ---------------------------------------------------------------------------------

def _lengths(n, lo, hi, log=False):
    """n lengths between lo and hi, the same for every seed."""
    r = np.random.default_rng([n, lo, hi])
    if log:
        return np.exp(r.uniform(math.log(lo), math.log(hi), n)).round().astype(np.int64)
    return r.integers(lo, hi + 1, n)


def _step(case):
    """(cached, new) tokens of every sequence of a step; the first prompt starts its sequence."""
    cached = list(_lengths(case["decode"], case["lo"], case["hi"])) if case["decode"] else []
    new = [1] * len(cached) + [case["prompt"]] * case["prompts"]
    cached += [i * case.get("prefix", 0) * 2 // 3 for i in range(case["prompts"])]
    return np.asarray(cached, np.int32), np.asarray(new, np.int32)


def _pairs(cached, new):
    """Query-key pairs of causal attention."""
    c, n = np.asarray(cached, np.float64), np.asarray(new, np.float64)
    return float((n * c + n * (n + 1) / 2).sum())


def _qwen_params(c):
    kv = c["n_kv_heads"] * 128
    return c["hidden"] * (2 * c["hidden"] + 2 * kv + 3 * c["intermediate"]) * c["n_layers"]


def work(case):
    kind = case["kind"]
    if kind == "embed":
        lens = _lengths(case["seqs"], case["lo"], case["hi"]).astype(np.float64)
        p, T = _qwen_params(STELLA), float(lens.sum())
        return {"bytes": 2 * p + T * 4 + 2 * T * 1536 + case["seqs"] * 4096 + 1024 * 1536 * 2,
                "flops": 2 * p * T + 4 * 1536 * float((lens ** 2).sum()) * STELLA["n_layers"] + 2 * 1024 * 1536 * case["seqs"]}
    if kind == "int4":
        n, k, b = case["n"], case["k"], case["batch"]
        return {"bytes": n * k * 0.5625 + 2 * b * (n + k), "flops": 2 * b * n * k}
    if kind == "paged":
        ctx = float(_lengths(case["seqs"], case["lo"], case["hi"], log=True).sum())
        return {"bytes": 1024 * ctx + case["seqs"] * (2 * 4096 + 1024), "flops": 8192 * ctx}
    if kind == "sample":
        return {"bytes": 2 * 4 * case["rows"] * case["vocab"], "flops": 0}
    cached, new = _step(case)
    T, rows, pairs, seen = float(new.sum()), len(new), _pairs(cached, new), float((cached + new).sum())
    if kind == "decoder":
        p, n = _qwen_params(DECODER), DECODER["n_layers"]
        return {"bytes": 0.5625 * (p + VOCAB * 1536) + 1024 * seen * n + 4 * rows * VOCAB + 2 * T * 1536,
                "flops": 2 * p * T + 4 * 1536 * pairs * n + 2 * rows * VOCAB * 1536}
    if kind == "hybrid":
        H, I, full = 2048, 6144, HYBRID["n_layers"] // 4
        lin = HYBRID["n_layers"] - full
        p = HYBRID["n_layers"] * 3 * H * I + full * H * (3 * 4096 + 2 * 512) + lin * H * (5 * 2048 + 32)
        states = rows * 16 * 128 * 128 * 4 * lin * (2 if case["decode"] else 1)
        return {"bytes": 0.5625 * (p + VOCAB * H) + 2048 * seen * full + states + 4 * rows * VOCAB + 2 * T * H,
                "flops": 2 * p * T + 4 * 4096 * pairs * full + 6 * 16 * 128 * 128 * T * lin + 2 * rows * VOCAB * H}
    y, H, n = LATENT_LAYER, LATENT["hidden"], LATENT["n_layers"]
    HD, Q, R = y["heads"] * y["dim"], y["q_rank"], y["kv_rank"]
    p = (H * (Q + R + 3 * y["ff"] + HD) + HD * (Q + 2 * R)) * n
    pair = 4 * HD if case["prompts"] else 4 * y["heads"] * R
    return {"bytes": 2 * (p + VOCAB * H) + 2 * R * seen * n + 4 * rows * VOCAB + 2 * T * H, "flops": 2 * p * T + pair * pairs * n + 2 * rows * VOCAB * H}


# About four times the error against 64 bits that each path shows: int4 and paged round their result to bfloat16 once, the models carry
# bfloat16 activations through 16 to 48 layers. The decoders' residual streams are dominated by the embedding, so less of it reaches their logits.
REL = {"embed": 2.5e-2, "decoder": 4e-3, "hybrid": 4e-3, "latent": 1e-2, "int4": 1.1e-2, "paged": 8e-3, "sample": 1e-6}


def tolerance(case):
    return {"rel": REL[case["kind"]], "max": 10 * REL[case["kind"]], "differ": 0.0}


# ---- models ------------------------------------------------------------------------------------------

def _gen(*seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(np.random.SeedSequence(list(seed)).generate_state(1)[0]))
    return g


def _mat(g, n, k, std):
    """A matrix whose values are representable in bfloat16."""
    return (torch.randn((n, k), generator=g, device="cuda") * std).to(torch.bfloat16).float()


def _int4(g, n, k, std):
    """Uniform codes and half-normal scales of a group-32 matrix."""
    codes = torch.randint(0, 256, (n, k // 2), generator=g, device="cuda", dtype=torch.uint8)
    return codes, (torch.randn((n, k // 32), generator=g, device="cuda") * std).abs().to(torch.float16)


def _expand(codes, scales):
    """int4 group-32 weights in 64 bits: value k of a row is a nibble of byte k / 2, the even one the low nibble, in two's complement."""
    q = torch.stack([codes & 15, codes >> 4], dim=-1).reshape(codes.shape[0], -1).to(torch.int16)
    q = torch.where(q > 7, q - 16, q).double()
    return (q.reshape(codes.shape[0], -1, 32) * scales.double()[:, :, None]).reshape(codes.shape[0], -1)


def _ones(n):
    return torch.ones(n, device="cuda")


def _zeros(n):
    return torch.zeros(n, device="cuda")


def _stella_layer(i):
    g, H, I, kv, s = _gen(1, i), 1536, STELLA["intermediate"], 256, 0.02
    vec = lambda n: _mat(g, 1, n, s)[0]
    return {"norm1": _ones(H), "norm2": _ones(H), "wq": _mat(g, H, H, s), "bq": vec(H), "wk": _mat(g, kv, H, s), "bk": vec(kv), "wv": _mat(g, kv, H, s), "bv": vec(kv),
            "wo": _mat(g, H, H, s), "w_gate": _mat(g, I, H, s), "w_up": _mat(g, I, H, s), "w_down": _mat(g, H, I, s)}


def _stella_ends():
    g = _gen(1, 1000)
    return {"tok_embed": _mat(g, STELLA["vocab"], 1536, 0.02), "final_norm": _ones(1536), "head_w": _mat(g, 1024, 1536, 0.02), "head_b": _mat(g, 1, 1024, 0.02)[0]}


def _decoder_layer(i):
    g, H, I, kv = _gen(2, i), 1536, DECODER["intermediate"], 256
    q = lambda n, k: _int4(g, n, k, 0.25 / math.sqrt(k))
    return {"norm1": _ones(H), "norm2": _ones(H), "bq": _zeros(H), "bk": _zeros(kv), "bv": _zeros(kv), "wq": q(H, H), "wk": q(kv, H), "wv": q(kv, H), "wo": q(H, H),
            "w_gate": q(I, H), "w_up": q(I, H), "w_down": q(H, I)}


def _hybrid_layer(i):
    g, H, I = _gen(3, i), HYBRID["hidden"], HYBRID["intermediate"]
    q = lambda n, k: _int4(g, n, k, 0.25 / math.sqrt(k))
    out = {"w_gate": q(I, H), "w_up": q(I, H), "w_down": q(H, I), "norm1": _ones(H), "norm2": _ones(H)}
    if is_full_attention(i, HYBRID["full_attn_interval"]):
        return dict(out, wq=q(4096, H), wgate=q(4096, H), wk=q(512, H), wv=q(512, H), wo=q(H, 4096))
    u = lambda lo, hi: torch.rand(16, generator=g, device="cuda") * (hi - lo) + lo
    return dict(out, wq=q(2048, H), wk=q(2048, H), wv=q(2048, H), wgate=q(2048, H), wo=q(H, 2048), wa=q(16, H), wb=q(16, H), A_log=torch.log(u(0.5, 4.0)), dt_bias=u(-3.0, 0.0))


def _int4_ends(seed, H, std):
    g = _gen(seed, 1000)
    return {"tok_embed": _mat(g, VOCAB, H, std), "final_norm": _ones(H), "lm_head": _int4(g, VOCAB, H, 0.25 / math.sqrt(H))}


def _latent_layer(i):
    g, y, H = _gen(4, i), LATENT_LAYER, LATENT["hidden"]
    HD, Q, R, F = y["heads"] * y["dim"], y["q_rank"], y["kv_rank"], y["ff"]
    m = lambda n, k, gain=1.0: _mat(g, n, k, gain / math.sqrt(k))
    return dict(norm1=_zeros(H), dq=m(Q, H), dq_norm=_ones(Q), uq=m(HD, Q), dkv=m(R, H), dkv_norm=_ones(R), uk=m(HD, R), uv=m(HD, R), o=m(H, HD, 0.3), gate=m(F, H),
                gate_b=_zeros(F), up=m(F, H), up_b=_zeros(F), down=m(H, F, 0.3), down_b=_zeros(H), conv1=m(H, 4, 0.3), conv2=m(H, 4, 0.3),
                dwa=torch.cat([0.02 * _ones(i + 1), _ones(1)]).to(torch.bfloat16).float())


def _latent_ends():
    g, H = _gen(4, 1000), LATENT["hidden"]
    return {"embed": _mat(g, VOCAB, H, 1.0), "final_norm": _zeros(H), "head": _mat(g, VOCAB, H, 1.0 / math.sqrt(H))}


def _host(t):
    if isinstance(t, tuple):
        return tuple(_host(x) for x in t)
    return np.ascontiguousarray(t.cpu().numpy())


def _bits(t):
    return np.ascontiguousarray(t.to(torch.bfloat16).view(torch.int16).cpu().numpy().view(np.uint16))


def _weights(ends, layer, n, put):
    each = lambda d: {k: put(v) for k, v in d.items()}
    return dict(each(ends), layers=[each(layer(i)) for i in range(n)])


class Server:
    """A loaded decoder with the blocks and slots that its live sequences hold."""

    def __init__(self, model, blocks, per_seq, slots):
        self.model, self.takes_slots = model, slots > 0
        self.blocks, self.slots, self.requests = BlockAllocator(blocks, per_seq, seed=1), SlotAllocator(max(slots, 1)), 0


@functools.lru_cache(maxsize=None)
def _stella():
    return StellaModel(STELLA, _weights(_stella_ends(), _stella_layer, STELLA["n_layers"], _host), max_batch_tokens=32768, max_batch_seqs=256)


@functools.lru_cache(maxsize=None)
def _server(kind):
    if kind == "decoder":
        w = _weights(_int4_ends(2, 1536, 1.0), _decoder_layer, DECODER["n_layers"], _host)
        return Server(DecoderModel(DECODER, w, 72000, 520, PROMPT_TOKENS + 64, 68), 72000, 520, 0)
    if kind == "hybrid":
        w = _weights(_int4_ends(3, HYBRID["hidden"], 0.5), _hybrid_layer, HYBRID["n_layers"], _host)
        return Server(HybridModel(HYBRID, w, 36000, 260, PROMPT_TOKENS, 64, 272), 36000, 260, 272)
    w = _weights(_latent_ends(), _latent_layer, LATENT["n_layers"], _bits)
    return Server(LatentModel(LATENT, w, 36000, 260, PROMPT_TOKENS, 64, 272), 36000, 260, 272)


def _tokens(case, seed):
    cached, new = _step(case)
    rng = np.random.default_rng([seed, 7])
    return [rng.integers(0, VOCAB, int(c + n), dtype=np.uint32) for c, n in zip(cached, new)]


class Sequences:
    """Sequences of one server with their cached history; what they hold goes back when they are dropped."""

    def __init__(self, kind, case, seed):
        self.kind, self.server = kind, _server(kind)
        self.cached, self.new = _step(case)
        tokens, n_seqs = _tokens(case, seed), len(self.new)
        self.names = [(self.server.requests, i) for i in range(n_seqs)]
        self.server.requests += 1
        self.tables = np.stack([self.server.blocks.ensure(s, int(c + n)) for s, c, n in zip(self.names, self.cached, self.new)])
        self.slots = np.asarray([self.server.slots.get(s) if self.server.takes_slots else 0 for s in self.names], np.int32)
        self.ids = np.concatenate([t[c:] for t, c in zip(tokens, self.cached)])
        done = np.zeros(n_seqs, np.int64)
        while (done < self.cached).any():  # the history, in prompt steps
            idx, new, room = [], [], PROMPT_TOKENS
            for i in range(n_seqs):
                n = int(min(self.cached[i] - done[i], room))
                if n > 0:
                    idx.append(i)
                    new.append(n)
                    room -= n
            self._step(np.concatenate([tokens[i][done[i]:done[i] + n] for i, n in zip(idx, new)]), done[idx], new, idx)
            done[idx] += new

    def _step(self, ids, cached, new, idx=slice(None)):
        args = [ids, cached, new, self.tables[idx]]
        if self.server.takes_slots:
            args.append(self.slots[idx])
        return self.server.model.step(*args)

    def step(self):
        self._step(self.ids, self.cached, self.new)
        return self.server.model.logits_tensor() if self.kind == "latent" else self.server.model.last_logits()

    def __del__(self):
        for s in getattr(self, "names", ()):
            self.server.blocks.release(s)
            self.server.slots.release(s)


# ---- prepare, run ------------------------------------------------------------------------------------

def _embed_inputs(case, seed):
    lens = _lengths(case["seqs"], case["lo"], case["hi"])
    cu = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    return np.random.default_rng([seed, 3]).integers(0, STELLA["vocab"], int(cu[-1]), dtype=np.uint32), cu


def _int4_inputs(case, seed):
    g, n, k = _gen(seed, 5), case["n"], case["k"]
    codes, scales = _int4(g, n, k, 0.02)
    return codes, scales, torch.randn((case["batch"], k), generator=g, device="cuda").to(torch.bfloat16)


def _paged_inputs(case, seed):
    """16 query and 2 key heads of 128; block tables are a permutation of a shared pool."""
    g, n = _gen(seed, 6), case["seqs"]
    ctx = _lengths(n, case["lo"], case["hi"], log=True)
    nb = (ctx + 15) // 16
    perm = np.random.default_rng([seed, 6]).permutation(int(nb.sum())).astype(np.int32)
    tables, at = np.zeros((n, int(nb.max())), np.int32), 0
    for i in range(n):
        tables[i, :nb[i]] = perm[at:at + nb[i]]
        at += nb[i]
    r = lambda *shape: torch.randn(shape, generator=g, device="cuda", dtype=torch.bfloat16)
    return {"ctx": ctx.astype(np.int32), "tables": torch.from_numpy(tables).cuda(), "k": r(int(nb.sum()), 16, 256), "v": r(int(nb.sum()), 16, 256), "q": r(n, 2048),
            "new_k": r(n, 256), "new_v": r(n, 256)}


def _sample_inputs(case, seed):
    return torch.randn((case["rows"], case["vocab"]), generator=_gen(seed, 8), device="cuda") * 3.0


def prepare(case, seed):
    kind = case["kind"]
    if kind == "embed":
        ids, cu = _embed_inputs(case, seed)
        return {"kind": kind, "model": _stella(), "ids": ids, "cu": cu}
    if kind == "int4":
        codes, scales, x = _int4_inputs(case, seed)
        return {"kind": kind, "codes": codes, "scales": scales, "x": x, "workspace": _zeros(case["batch"] * case["n"]),
                "status": torch.zeros(1, dtype=torch.int32, device="cuda")}
    if kind == "paged":
        s = _paged_inputs(case, seed)
        chunk = ops.pick_decode_chunk(s["ctx"], 2, 128)
        offsets, total = ops.build_decode_chunks(s["ctx"], chunk)
        return {"kind": kind, **s, "ctx": torch.from_numpy(s["ctx"]).cuda(), "offsets": offsets.cuda(), "total": total, "chunk": chunk,
                "scratch": torch.empty(int(ops.lib.logismos_paged_decode_scratch_bytes(total, 16, 128)), dtype=torch.uint8, device="cuda")}
    if kind == "sample":
        chain = DecodeChain(MultinomialSampler(seed=seed % (1 << 31)))
        chain.push(TemperatureScale(case["temperature"])).push(TopK(case["top_k"])).push(TopP(case["top_p"]))
        if case["min_p"]:
            chain.push(MinP(case["min_p"]))
        return {"kind": kind, "logits": _sample_inputs(case, seed), "chain": chain}
    return {"kind": kind, "sequences": Sequences(kind, case, seed)}


def run(state):
    kind, s = state["kind"], state
    if kind == "embed":
        return s["model"].encode_ids_batch(s["ids"], s["cu"])
    if kind == "int4":
        return ops.skinny_int4(s["codes"], s["scales"], s["x"], s["workspace"], status=s["status"], sync=False)
    if kind == "paged":
        return ops.paged_attention_decode(s["q"], s["k"], s["v"], s["new_k"], s["new_v"], s["tables"], s["ctx"], s["offsets"], s["total"], s["chunk"], 16, 2, 128,
                                          scratch=s["scratch"], sync=False)
    if kind == "sample":
        logits = s["logits"].clone()  # the chain works in place on what a step left
        return {"tokens": s["chain"].step(logits), "logits": logits}
    # a decode step repeated at one position; recurrent states go on from step to step
    return s["sequences"].step()


# ---- the same in 64 bits -----------------------------------------------------------------------------

def _rms(x, w, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * w


def _silu(x):
    return x * torch.sigmoid(x)


def _rope(x, base):
    """x [B, L, heads, d], pairs (i, i + d / 2)."""
    half = x.shape[-1] // 2
    f = base ** (-2.0 * torch.arange(half, device=x.device, dtype=torch.float64) / x.shape[-1])
    a = torch.arange(x.shape[1], device=x.device, dtype=torch.float64)[:, None] * f
    c, s, u, v = a.cos()[:, None], a.sin()[:, None], x[..., :half], x[..., half:]
    return torch.cat([u * c - v * s, v * c + u * s], dim=-1)


def _attend(q, k, v, lens, scale, causal, rows=1024):
    """q [B, L, H, d], k [B, L, G, d], v [B, L, G, e] -> [B, L, H e]."""
    B, L, H, _ = q.shape
    G = k.shape[2]
    out = torch.zeros((B, L, H, v.shape[3]), device=q.device, dtype=q.dtype)
    for b in range(B):
        n = int(lens[b])
        kb, vb = (t[b, :n].permute(1, 0, 2).repeat_interleave(H // G, dim=0) for t in (k, v))
        for i in range(0, n, rows):
            qb = q[b, i:min(i + rows, n)].permute(1, 0, 2)
            s = qb @ kb.transpose(1, 2) * scale
            if causal:
                at = torch.arange(i, i + qb.shape[1], device=q.device)
                s = s.masked_fill(torch.arange(n, device=q.device)[None, :] > at[:, None], -math.inf)
            out[b, i:i + qb.shape[1]] = (torch.softmax(s, dim=-1) @ vb).permute(1, 0, 2)
    return out.reshape(B, L, -1)


def _padded(tokens):
    lens = [len(t) for t in tokens]
    ids = np.zeros((len(tokens), max(lens)), np.int64)
    for i, t in enumerate(tokens):
        ids[i, :lens[i]] = t
    return torch.from_numpy(ids).cuda(), lens


def _layers64(layer, n):
    """One layer's tensors at a time, int4 matrices expanded."""
    for i in range(n):
        yield {k: _expand(*v) if isinstance(v, tuple) else v.double() for k, v in layer(i).items()}


def _gated_ff(x, w):
    h = _rms(x, w["norm2"], 1e-6)
    return x + (_silu(h @ w["w_gate"].T) * (h @ w["w_up"].T)) @ w["w_down"].T


def _qwen64(x, layers, lens, base, causal):
    B, L, _ = x.shape
    for w in layers:
        h = _rms(x, w["norm1"], 1e-6)
        q, k, v = ((h @ w["w" + n].T + w["b" + n]).reshape(B, L, -1, 128) for n in "qkv")
        x = _gated_ff(x + _attend(_rope(q, base), _rope(k, base), v, lens, 128 ** -0.5, causal) @ w["wo"].T, w)
    return x


def _delta_rule(h, w):
    B, L, _ = h.shape
    heads = lambda n: (h @ w[n].T).reshape(B, L, 16, 128)
    unit = lambda t: t / t.norm(dim=-1, keepdim=True).clamp_min(1e-12)
    q, k, v, z = unit(heads("wq")) * 128 ** -0.5, unit(heads("wk")), heads("wv"), heads("wgate")
    decay = torch.exp(-torch.exp(w["A_log"]) * torch.nn.functional.softplus(h @ w["wa"].T + w["dt_bias"]))
    beta, S, o = torch.sigmoid(h @ w["wb"].T), torch.zeros((B, 16, 128, 128), device=h.device, dtype=h.dtype), torch.empty_like(v)
    for t in range(L):
        S.mul_(decay[:, t, :, None, None])
        d = beta[:, t, :, None] * (v[:, t] - (k[:, t, :, None] @ S)[:, :, 0])
        S += k[:, t, :, :, None] * d[:, :, None]
        o[:, t] = (q[:, t, :, None] @ S)[:, :, 0]
    return (o * _silu(z)).reshape(B, L, -1)


def _hybrid64(x, lens):
    B, L, _ = x.shape
    base = HYBRID["rope_theta"]
    for i, w in enumerate(_layers64(_hybrid_layer, HYBRID["n_layers"])):
        h = _rms(x, w["norm1"], 1e-6)
        if is_full_attention(i, HYBRID["full_attn_interval"]):
            q, k, v = ((h @ w[n].T).reshape(B, L, -1, 256) for n in ("wq", "wk", "wv"))
            m = _attend(_rope(q, base), _rope(k, base), v, lens, 256 ** -0.5, True) * torch.sigmoid(h @ w["wgate"].T)
        else:
            m = _delta_rule(h, w)
        x = _gated_ff(x + m @ w["wo"].T, w)
    return x


def _latent64(x, lens):
    B, L, _ = x.shape
    y, eps, history = LATENT_LAYER, LATENT["rms_eps"], [x]

    def conv(h, w):
        p = torch.nn.functional.pad(h, (0, 0, w.shape[1] - 1, 0))
        return sum(p[:, j:j + L] * w[:, j] for j in range(w.shape[1]))

    for w in _layers64(_latent_layer, LATENT["n_layers"]):
        h = _rms(x, 1.0 + w["norm1"], eps)
        a, f = h + conv(h, w["conv1"]), h + conv(h, w["conv2"])
        c = _rms(a @ w["dkv"].T, w["dkv_norm"], eps)
        q = (_rms(a @ w["dq"].T, w["dq_norm"], eps) @ w["uq"].T).reshape(B, L, -1, 128)
        k, v = ((c @ w[n].T).reshape(B, L, -1, 128) for n in ("uk", "uv"))
        g, u = (f @ w["gate"].T + w["gate_b"]).clamp(max=y["glu_limit"]), (f @ w["up"].T + w["up_b"]).clamp(-y["glu_limit"], y["glu_limit"])
        ff = (g * torch.sigmoid(GLU_ALPHA * g) * (u + GLU_SHIFT)) @ w["down"].T + w["down_b"]
        history.append(x + _attend(q, k, v, lens, y["scale"], True) @ w["o"].T + ff)
        x = sum(m * t for m, t in zip(w["dwa"], history))
    return x


def _decode64(kind, case, seed):
    """Logits after the last token of every sequence, each computed from its first token on."""
    tokens, rows, at = _tokens(case, seed), [], 0
    if kind == "latent":
        e = _latent_ends()
        table, head = e["embed"], e["head"].double()
    else:
        e = _int4_ends(2, 1536, 1.0) if kind == "decoder" else _int4_ends(3, HYBRID["hidden"], 0.5)
        table, head = e["tok_embed"], _expand(*e["lm_head"])
    while at < len(tokens):  # some sequences at a time
        to = at + 1
        while to < len(tokens) and (to + 1 - at) * max(len(t) for t in tokens[at:to + 1]) <= 40000:
            to += 1
        ids, lens = _padded(tokens[at:to])
        x = table[ids].double()
        if kind == "decoder":
            x = _qwen64(x, _layers64(_decoder_layer, DECODER["n_layers"]), lens, DECODER["rope_theta"], True)
        else:
            x = _hybrid64(x, lens) if kind == "hybrid" else _latent64(x, lens)
        z = _rms(torch.stack([x[i, n - 1] for i, n in enumerate(lens)]), 1.0, 1e-6) @ head.T
        rows.append(LATENT["logit_softcap"] * torch.tanh(z / LATENT["logit_softcap"]) if kind == "latent" else z)
        at = to
    return torch.cat(rows)


def _decode64_flops(kind, case):
    cached, new = _step(case)
    p = {"decoder": _qwen_params(DECODER), "hybrid": 5.8e9, "latent": 1.2e9}[kind]  # the hybrid's recurrence takes as long again
    return 2 * p * float((cached + new).sum())


def _embed64(case, seed):
    ids, cu = _embed_inputs(case, seed)
    e, out = _stella_ends(), []
    tokens = [ids[a:b] for a, b in zip(cu[:-1], cu[1:])]
    for at in range(0, len(tokens), 32):
        t, lens = _padded(tokens[at:at + 32])
        x = _qwen64(e["tok_embed"][t].double(), _layers64(_stella_layer, STELLA["n_layers"]), lens, STELLA["rope_theta"], False)
        x = _rms(x, 1.0, STELLA["rms_eps"])
        p = torch.stack([x[i, :n].mean(0) for i, n in enumerate(lens)])
        p = p / p.norm(dim=-1, keepdim=True) @ e["head_w"].double().T + e["head_b"].double()
        out.append(p / p.norm(dim=-1, keepdim=True))
    return torch.cat(out)


def _paged64(case, seed):
    s, out = _paged_inputs(case, seed), []
    for i, n in enumerate(s["ctx"].tolist()):
        t = s["tables"][i, :(n + 15) // 16].long()
        k, v = (s[p][t].reshape(-1, 256)[:n].double() for p in "kv")
        k[n - 1], v[n - 1] = s["new_k"][i].double(), s["new_v"][i].double()
        k, v = (p.reshape(n, 2, 128).permute(1, 0, 2) for p in (k, v))
        out.append((torch.softmax(s["q"][i].double().reshape(2, 8, 128) @ k.transpose(1, 2) * 128 ** -0.5, dim=-1) @ v).reshape(-1))
    return torch.stack(out)


def _sample64(case, seed):
    x = _sample_inputs(case, seed).double() / case["temperature"]
    order = x.argsort(dim=-1, descending=True)[:, :case["top_k"]]
    kept = x.gather(1, order)
    p = torch.softmax(kept, dim=-1)
    keep = p.cumsum(-1) - p < case["top_p"]  # up to and with the value that reaches the mass
    if case["min_p"]:
        keep &= p >= case["min_p"] * p[:, :1]
    none = torch.full_like(kept, -math.inf)
    return {"tokens": None, "logits": torch.full_like(x, -math.inf).scatter_(1, order, torch.where(keep, kept, none))}


def exact(case, seed):
    kind = case["kind"]
    if kind == "embed":
        return _embed64(case, seed)
    if kind == "int4":
        codes, scales, x = _int4_inputs(case, seed)
        return torch.cat([x.double() @ _expand(codes[i:i + 16384], scales[i:i + 16384]).T for i in range(0, case["n"], 16384)], dim=1)
    if kind == "paged":
        return _paged64(case, seed)
    if kind == "sample":
        return _sample64(case, seed)
    return _decode64(kind, case, seed) if _decode64_flops(kind, case) <= EXACT_FLOPS else None
