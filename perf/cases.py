"""The calls a program that serves RWKV models makes of this library, as cases that can be timed.

A serving program loads a model once (quantizing its matrices), keeps one bundle of recurrent states for its sequences,
and from then on does two things: it reads prompts (`RnnInput` of many tokens, cut into jobs by `token_chunk_size`) and it
decodes (one token per sequence and step), both through `Bundle.infer` with host tokens in and host logits out.  Models are
kept for the life of the process, as such a program keeps them; a case's bundle, tokens and states are its own and come
from the seed.  Shapes are the configurations of `synth.CONFIGS`; the 7B- and 3B-shaped models have eight of their 32 layers
here (all layers are alike), the smaller ones are whole.
"""
import ctypes
import importlib
import math

import numpy as np
import torch

wrk = importlib.import_module("web-rwkv_b200")
rt = importlib.import_module("web-rwkv_b200.runtime")
synth = importlib.import_module("web-rwkv_b200.synth")

LAYERS = {"v6-3b": 8, "v6-7b": 8, "v7-7b": 8}
# an unquantized v5 model of the 1.6B-shaped configuration's widths, twelve layers
V5_WIDE = (5, 2048, 12, 7168, 65536)
QUANT = {"fp16": wrk.QUANT_NONE, "int8": wrk.QUANT_INT8, "nf4": wrk.QUANT_NF4, "sf4": wrk.QUANT_SF4}
SERVED = [("v6-0.1b", "int8"), ("v6-1.6b", "int8"), ("v6-7b", "int8"), ("v6-3b", "nf4"), ("v7-7b", "int8"), ("v5-2048", "fp16")]
WEIGHT_SEED = 1000
PROMPT = 16  # tokens that every decoding sequence has read before the timed step


def listed():
    return [
        # one user, one token: the smallest call there is, bound by launches and latency
        dict(name="decode v6 0.1b int8, 1 seq", kind="decode", model="v6-0.1b", quant="int8", batch=1),
        # one user on a model of ordinary size
        dict(name="decode v6 1.6b int8, 1 seq", kind="decode", model="v6-1.6b", quant="int8", batch=1),
        # one user on a large model: weight streaming
        dict(name="decode v6 7b int8, 1 seq", kind="decode", model="v6-7b", quant="int8", batch=1),
        # the same for the current model family
        dict(name="decode v7 7b int8, 1 seq", kind="decode", model="v7-7b", quant="int8", batch=1),
        # a few users on 4-bit weights
        dict(name="decode v6 3b nf4, 4 seq", kind="decode", model="v6-3b", quant="nf4", batch=4),
        # a small server on unquantized weights
        dict(name="decode v5 2048 fp16, 16 seq", kind="decode", model="v5-2048", quant="fp16", batch=16),
        # a busy server: 64 sequences in step, states and weights both count
        dict(name="decode v7 7b int8, 64 seq", kind="decode", model="v7-7b", quant="int8", batch=64),
        # a prompt in small chunks (little memory, other work interleaved) on a small model
        dict(name="prefill v6 0.1b int8, 256 / 32", kind="prefill", model="v6-0.1b", quant="int8", batch=1, tokens=256, mixed=False, chunk=32),
        # one long prompt whose length is no multiple of the chunk
        dict(name="prefill v6 7b int8, 1000 / 256", kind="prefill", model="v6-7b", quant="int8", batch=1, tokens=1000, mixed=False, chunk=256),
        # several prompts of one length read together, 4-bit weights
        dict(name="prefill v6 3b nf4, 4x512 / 256", kind="prefill", model="v6-3b", quant="nf4", batch=4, tokens=512, mixed=False, chunk=256),
        # prompts of mixed lengths (16 to 700 tokens) read together
        dict(name="prefill v7 7b int8, 8 mixed", kind="prefill", model="v7-7b", quant="int8", batch=8, tokens=700, mixed=True, chunk=256),
        # loading: one FFN matrix of the 7B shape quantized on the device
        dict(name="quantize int8 14336 x 4096", kind="quantize", k=4096, m=14336, quant="int8"),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["decode", "decode", "decode", "prefill", "prefill", "prefill", "quantize"])
    if kind == "quantize":
        # rows of whole quantization blocks; row counts as they come
        return dict(kind=kind, k=128 * _log_uniform(rng, 4, 56), m=_log_uniform(rng, 500, 14336), quant=rng.choice(["int8", "nf4", "sf4"]))
    model, quant = rng.choice(SERVED)
    if kind == "decode":
        return dict(kind=kind, model=model, quant=quant, batch=_log_uniform(rng, 1, 64))
    batch = _log_uniform(rng, 1, 8)
    chunk = rng.choice([32, 64, 128, 256, 256])
    tokens = min(_log_uniform(rng, 9, 700), 8 * chunk // batch)
    return dict(kind=kind, model=model, quant=quant, batch=batch, tokens=tokens, mixed=rng.random() < 0.5, chunk=chunk)


def _config(model):
    version, C, L, F, V = V5_WIDE if model == "v5-2048" else synth.CONFIGS[model]
    return version, C, LAYERS.get(model, L), F, V


def _lengths(case):
    """Prompt lengths of a prefill case: all equal, or from `tokens` down to 16 in equal ratios."""
    n, longest = case["batch"], case["tokens"]
    if not case["mixed"] or n == 1:
        return [longest] * n
    shortest = min(16, longest)
    return [int(round(longest * (shortest / longest) ** (i / (n - 1)))) for i in range(n)]


# ---- models: seeded weights of synth's distributions, made on the GPU ---------------------------------------------------

NORMAL, NEAR_ONE, UNIT, DECAY, BONUS, WIDE = range(6)


def _tensors(version, C, L, F, V):
    """(name, shape, distribution) of every tensor of a model file."""
    H = C // synth.HEAD_SIZE
    for name in ("emb.weight", "head.weight"):
        yield name, (V, C), NORMAL
    yield from ((n, (C,), d) for n, d in (("ln_out.weight", NEAR_ONE), ("ln_out.bias", NORMAL), ("blocks.0.ln0.weight", NEAR_ONE), ("blocks.0.ln0.bias", NORMAL)))
    for i in range(L):
        b, att, ffn = f"blocks.{i}", f"blocks.{i}.att", f"blocks.{i}.ffn"
        for ln in (f"{b}.ln1", f"{b}.ln2", f"{att}.ln_x"):
            yield f"{ln}.weight", (C,), NEAR_ONE
            yield f"{ln}.bias", (C,), NORMAL
        for n in ("key", "value", "receptance", "output"):
            yield f"{att}.{n}.weight", (C, C), NORMAL
        yield f"{ffn}.key.weight", (F, C), NORMAL
        yield f"{ffn}.value.weight", (C, F), NORMAL
        if version in (5, 6):
            yield f"{att}.gate.weight", (C, C), NORMAL
            yield f"{ffn}.receptance.weight", (C, C), NORMAL
            yield f"{att}.time_decay", (H, synth.HEAD_SIZE), DECAY
            yield f"{att}.time_first", (H, synth.HEAD_SIZE), BONUS
            for n in ("att.time_mix_k", "att.time_mix_v", "att.time_mix_r", "att.time_mix_g", "ffn.time_mix_k", "ffn.time_mix_r"):
                yield f"{b}.{n}", (1, 1, C), UNIT
        if version == 6:
            D, W = synth.V6_TIME_MIX, synth.V6_TIME_DECAY
            yield f"{att}.time_mix_x", (1, 1, C), UNIT
            yield f"{att}.time_mix_w", (1, 1, C), UNIT
            yield f"{att}.time_mix_w1", (5 * D, C), NORMAL
            yield f"{att}.time_mix_w2", (5, C, D), NORMAL
            yield f"{att}.time_decay_w1", (W, C), NORMAL
            yield f"{att}.time_decay_w2", (C, W), NORMAL
        if version == 7:
            for n in ("att.x_r", "att.x_w", "att.x_k", "att.x_v", "att.x_a", "att.x_g", "ffn.x_k", "att.k_k", "att.k_a"):
                yield f"{b}.{n}", (1, 1, C), UNIT
            yield f"{att}.w0", (1, 1, C), DECAY
            yield f"{att}.r_k", (H, synth.HEAD_SIZE), UNIT
            for n, rank in (("a", synth.V7_A), ("w", synth.V7_W), ("g", synth.V7_G), ("v", synth.V7_V)):
                if n == "v" and i == 0:
                    continue
                if n in "av":
                    yield f"{att}.{n}0", (1, 1, C), WIDE
                yield f"{att}.{n}1", (rank, C), NORMAL
                yield f"{att}.{n}2", (C, rank), NORMAL


def _values(gen, shape, dist):
    if dist in (UNIT, DECAY, BONUS):
        lo, hi = {UNIT: (0.0, 1.0), DECAY: (-6.0, 1.0), BONUS: (-1.0, 1.0)}[dist]
        t = torch.rand(shape, generator=gen, device="cuda") * (hi - lo) + lo
    else:
        t = torch.randn(shape, generator=gen, device="cuda") * (1.0 if dist == WIDE else 0.02) + (1.0 if dist == NEAR_ONE else 0.0)
    return t.half().cpu().numpy()


_kept = {}  # what a serving program keeps for its life: the context and its models


def _context():
    if "ctx" not in _kept:
        torch.cuda.init()
        _kept["ctx"] = wrk.Context(0)
    return _kept["ctx"]


def _model(name, quant):
    if (name, quant) not in _kept:
        cfg = _config(name)
        gen = torch.Generator(device="cuda").manual_seed(WEIGHT_SEED)
        builder = rt.ModelBuilder(_context())
        for tensor, shape, dist in _tensors(*cfg):
            builder.add_tensor(tensor, _values(gen, shape, dist))
        builder.quant({i: QUANT[quant] for i in range(cfg[2])})
        _kept[name, quant] = builder.build()
    return _kept[name, quant]


# ---- device tensors of the library as torch tensors, without a copy -------------------------------------------------

_TORCH = {wrk.F32: "<f4", wrk.F16: "<f2", wrk.U8: "|u1", wrk.U16: "<u2", wrk.U32: "<u4"}


class _Alias:
    def __init__(self, tensor):
        ptr = ctypes.c_void_p()
        wrk.check(wrk.lib().wrk_tensor_device_ptr(tensor.handle, ctypes.byref(ptr)))
        self.keep = tensor
        self.__cuda_array_interface__ = {"shape": tuple(tensor.shape[::-1]), "typestr": _TORCH[tensor.dtype], "data": (ptr.value, False),
                                         "strides": None, "version": 3}


def _torch(tensor):
    return torch.as_tensor(_Alias(tensor), device="cuda")


def _state_tensors(bundle):
    """The bundle's own state buffers, one per layer."""
    out = []
    for layer in range(bundle.model.info.num_layer):
        h = ctypes.c_void_p()
        wrk.check(wrk.lib().wrk_state_layer(bundle.handle, layer, ctypes.byref(h)))
        wrk.check(wrk.lib().wrk_tensor_retain(h))
        out.append(_torch(wrk.Tensor(bundle.model.ctx, h)))
    return out


# ---- the cases ------------------------------------------------------------------------------------------------------------

def _read(bundle, inp, logits):
    """Runs an input's jobs until every token is read; per sequence the logits row of its last token."""
    last = [None] * bundle.num_batch
    while inp.num_token():
        for i, rows in enumerate(bundle.infer(inp, logits)):
            if len(rows):
                last[i] = rows[-1].copy()
    return last


def prepare(case, seed):
    rng = np.random.default_rng([seed, 7])
    ctx = _context()
    if case["kind"] == "quantize":
        gen = torch.Generator(device="cuda").manual_seed(seed)
        weights = ctx.tensor(wrk.F16, [case["k"], case["m"]])
        _torch(weights).copy_((torch.randn((1, 1, case["m"], case["k"]), generator=gen, device="cuda") * 0.02).half())
        torch.cuda.synchronize()
        make = {"int8": wrk.Matrix.quant_u8, "nf4": wrk.Matrix.quant_nf4, "sf4": wrk.Matrix.quant_sf4}[case["quant"]]
        return dict(case=case, weights=weights, make=make)

    vocab = _config(case["model"])[4]
    n = case["batch"]
    bundle = rt.Bundle(_model(case["model"], case["quant"]), n)
    if case["kind"] == "decode":
        # every sequence has read its prompt; what follows is one sampled token after the other
        logits = np.empty((max(n, 32), bundle.vocab), dtype=np.float32)
        _read(bundle, rt.RnnInput([(rng.integers(0, vocab, PROMPT), wrk.RNN_LAST) for _ in range(n)], 256), logits)
        inp = rt.RnnInput([([], wrk.RNN_LAST) for _ in range(n)], max(n, 32))
        return dict(case=case, bundle=bundle, inp=inp, logits=logits, tokens=[[int(t)] for t in rng.integers(0, vocab, n)],
                    states=_state_tensors(bundle))
    # every slot starts from the state that a common system prompt left
    logits = np.empty((max(n, 32), bundle.vocab), dtype=np.float32)
    _read(bundle, rt.RnnInput([(rng.integers(0, vocab, PROMPT), wrk.RNN_LAST)] + [([], wrk.RNN_LAST)] * (n - 1), 256), logits)
    start = bundle.state_read(0)
    prompts = [rng.integers(0, vocab, length).astype(np.uint32) for length in _lengths(case)]
    return dict(case=case, bundle=bundle, start=start, prompts=prompts, logits=logits, states=_state_tensors(bundle))


def run(state):
    case = state["case"]
    if case["kind"] == "quantize":
        _, w, scales, _ = state["make"](state["weights"]).parts()
        return [_torch(w), _torch(scales)]
    bundle = state["bundle"]
    if case["kind"] == "decode":
        inp = state["inp"]
        for i, token in enumerate(state["tokens"]):
            inp.append(i, token)
        rows = bundle.infer(inp, state["logits"])
        return [state["logits"][: len(rows)], state["states"]]
    for slot in range(bundle.num_batch):
        bundle.state_write(state["start"], slot)
    inp = rt.RnnInput([(p, wrk.RNN_LAST) for p in state["prompts"]], case["chunk"])
    return [np.stack(_read(bundle, inp, state["logits"])), state["states"]]


def _matrices(cfg):
    """(rows x columns of the layers' large matrices, of their adapters, of the head), in elements."""
    version, C, L, F, V = cfg
    large = L * (C * C * {5: 6, 6: 6, 7: 4}[version] + 2 * C * F)
    if version == 6:
        adapters = L * C * (2 * 5 * synth.V6_TIME_MIX + 2 * synth.V6_TIME_DECAY)
    else:
        adapters = L * C * 2 * (synth.V7_W + synth.V7_A + synth.V7_G + synth.V7_V) if version == 7 else 0
    return large, adapters, C * V


BYTES = {"fp16": 2.0, "int8": 1.0 + 4 / 128, "nf4": 0.5 + 2 / 64, "sf4": 0.5 + 2 / 64}


def work(case):
    if case["kind"] == "quantize":
        n = case["k"] * case["m"]
        return {"bytes": n * (2.0 + BYTES[case["quant"]]), "flops": 0}
    cfg = _config(case["model"])
    version, C, L, F, V = cfg
    large, adapters, head = _matrices(cfg)
    n = case["batch"]
    tokens = n if case["kind"] == "decode" else sum(_lengths(case))
    state = L * C * (synth.HEAD_SIZE + 2) * 4
    bytes_ = large * BYTES[case["quant"]] + 2 * (adapters + head) + 2 * n * state + 2 * C * tokens + 4 * V * n
    # the recurrence: about eight operations per state entry and token
    flops = 2 * (large + adapters) * tokens + 2 * head * n + 8 * L * C * synth.HEAD_SIZE * tokens
    return {"bytes": bytes_, "flops": flops}


def tolerance(case):
    # quantized bytes and scales are whole results: no rounding is left open
    if case["kind"] == "quantize":
        return "exact"
    # fp16 activations between the layers' matrices, f32 sums: the fp16 steps of two implementations differ, and the layers
    # after them magnify it; 4-bit weights also meet the code book's own rounding to fp16, before or after the scale
    return {"rel": 2e-2 if case["quant"] in ("nf4", "sf4") else 1e-2}
