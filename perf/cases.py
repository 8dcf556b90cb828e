"""The work a user of this library has it do, as cases that can be timed and compared.

Every case goes through the public entry points of ``glm_asr_stack_b200`` and is one call a program makes over and
over: one FP4 linear, the projections of a decoder layer (on device and on host buffers), a batched decode step, a
batched prefill, the audio path from samples to decoder embeddings, and a whole transcription.  The shapes are those
of the decoder and the audio tower in ``workloads.py`` (28 layers, hidden 2048, 16 / 4 heads of 128, ffn 6144,
vocabulary 59264; 32 encoder layers of 1280); the sizes that vary in use -- rows, sequences, context lengths, clip
lengths -- are what the cases and ``draw`` vary.

``mode`` is the arithmetic of the FP4 projections: ``w4a16`` (what the library does unless told otherwise: bf16
activations) or ``w4a4`` (GLMASR_USE_CUTLASS_NVFP4=1 GLMASR_NVFP4_PAIRS=1: activations quantised to e2m1 as well).
"""
from __future__ import annotations

import ctypes
import math
import os

import numpy as np
import torch

from glm_asr_stack_b200 import _lib, engine, ops, synth, workloads
from glm_asr_stack_b200.pipeline import AsrPipeline, audio_tokens, feature_frames, padded_feature_frames, synthetic_window

LAYERS, HIDDEN, FFN, HEADS, KV_HEADS, HEAD_DIM, VOCAB = 28, 2048, 6144, 16, 4, 128, 59264
KV = KV_HEADS * HEAD_DIM
QKV = HIDDEN + 2 * KV
ENC_LAYERS, ENC, ENC_FFN, MELS, PROJ_MID = 32, 1280, 5120, 128, 4096
RATE = 16000
PROMPT_EXTRA = 19                  # prompt tokens around the audio
# (N, K) of the projections of one decoder layer
PROJECTIONS = ((HIDDEN, HIDDEN), (KV, HIDDEN), (FFN, HIDDEN), (HIDDEN, FFN))
LAYER_PARAMS = QKV * HIDDEN + HIDDEN * HIDDEN + 2 * FFN * HIDDEN + HIDDEN * FFN
FP4_BYTES = 0.5 + 1.0 / 16         # a weight element: half a byte and its share of a block scale


def listed():
    return [
        # one row through one projection: the smallest call there is, all latency and host work
        {"name": "linear_w4a4_1", "op": "linear", "mode": "w4a4", "rows": 1, "n": HIDDEN, "k": HIDDEN},
        # the single FP4 linear of the benchmark: a full decode batch through one 6144 x 2048 projection
        {"name": "linear_w4a16_256", "op": "linear", "mode": "w4a16", "rows": 256, "n": FFN, "k": HIDDEN},
        # the projections of one decoder layer for a full prefill batch (the benchmark's headline) ...
        {"name": "layer_w4a4_10000", "op": "layer", "mode": "w4a4", "rows": 10000, "host": False},
        # ... and the same call for a program that keeps its activations in pinned host memory
        {"name": "layer_host_w4a4_10000", "op": "layer", "mode": "w4a4", "rows": 10000, "host": True},
        # a single live stream: one sequence decodes, every step waits for its token
        {"name": "decode_w4a16_1", "op": "decode", "mode": "w4a16", "seqs": 1, "ctx_lo": 300, "ctx_hi": 300},
        # a handful of streams, odd in number and uneven in length
        {"name": "decode_w4a16_19", "op": "decode", "mode": "w4a16", "seqs": 19, "ctx_lo": 40, "ctx_hi": 450},
        # the benchmark's decode step: a full batch of 256 sequences with 200 to 450 tokens each
        {"name": "decode_w4a4_256", "op": "decode", "mode": "w4a4", "seqs": 256, "ctx_lo": 200, "ctx_hi": 450},
        # the prompt of one short clip, alone
        {"name": "prefill_w4a16_1", "op": "prefill", "mode": "w4a16", "seqs": 1, "len_lo": 173, "len_hi": 173},
        # a prefill batch at the scheduler's limit of 10000 tokens
        {"name": "prefill_w4a4_10000", "op": "prefill", "mode": "w4a4", "seqs": 25, "len_lo": 400, "len_hi": 400},
        # the audio of one short utterance: samples -> log-mel -> encoder -> decoder embeddings
        {"name": "audio_1_short", "op": "audio", "windows": 1, "sec_lo": 3.7, "sec_hi": 3.7},
        # the benchmark's encoder batch: sixteen full 30 s windows, from their samples on
        {"name": "audio_16", "op": "audio", "windows": 16, "sec_lo": 30.0, "sec_hi": 30.0},
        # a batch of clips of uneven length from host samples to tokens
        {"name": "transcribe_20", "op": "transcribe", "mode": "w4a16", "windows": 20, "sec_lo": 4.0, "sec_hi": 30.0,
         "new_tokens": 24},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49)))))))


def draw(rng):
    op = rng.choice(["linear", "layer", "decode", "decode", "prefill", "prefill", "audio", "transcribe"])
    mode = rng.choice(["w4a16", "w4a4"])
    if op == "linear":
        n, k = rng.choice(PROJECTIONS)
        return {"op": op, "mode": mode, "rows": _log_int(rng, 1, 10000), "n": n, "k": k}
    if op == "layer":
        return {"op": op, "mode": mode, "rows": _log_int(rng, 1, 10000), "host": rng.random() < 0.25}
    if op == "decode":
        lo = _log_int(rng, 20, 400)
        return {"op": op, "mode": mode, "seqs": _log_int(rng, 1, 256), "ctx_lo": lo, "ctx_hi": rng.randint(lo, 450)}
    if op == "prefill":
        hi = rng.randint(24, 400)
        return {"op": op, "mode": mode, "seqs": _log_int(rng, 1, 25), "len_lo": rng.randint(24, hi), "len_hi": hi}
    hi = round(rng.uniform(1.0, 30.0), 2)
    lo = round(rng.uniform(1.0, hi), 2)
    if op == "audio":
        return {"op": op, "windows": _log_int(rng, 1, 16), "sec_lo": lo, "sec_hi": hi}
    return {"op": op, "mode": "w4a16", "windows": _log_int(rng, 1, 20), "sec_lo": lo, "sec_hi": hi,
            "new_tokens": rng.randint(4, 24)}


# ---- sizes that vary inside a case: fixed by the case, so that every seed asks for the same work ----------------------
def _spread(n, lo, hi, whole=True):
    """n values over [lo, hi], evenly spread and then mixed up."""
    v = np.linspace(lo, hi, n) if n > 1 else np.array([hi], dtype=np.float64)
    np.random.default_rng(n).shuffle(v)
    return [int(round(x)) for x in v] if whole else [float(x) for x in v]


def _contexts(case):
    return _spread(case["seqs"], case["ctx_lo"], case["ctx_hi"])


def _prompt_lens(case):
    return _spread(case["seqs"], case["len_lo"], case["len_hi"])


def _clip_samples(case):
    return [int(s * RATE) for s in _spread(case["windows"], case["sec_lo"], case["sec_hi"], whole=False)]


# ---- what a program keeps between its calls -------------------------------------------------------------------------
_kept = {}


def _model():
    """The one model a process serves: FP4 decoder and bf16 audio tower with random weights.  Two things are as in a
    trained model and not as in a random one: a layer adds a small part to the residual stream (embeddings of standard
    deviation 4), and the greedy token wins by a margin (output head tied to the embedding)."""
    if "model" not in _kept:
        m = workloads.build_asr_model(LAYERS, ENC_LAYERS)
        m.embed *= 4.0
        m.lm_head = ops.Fp4Tensor(*synth.quantize_weight(m.embed.float() * 0.005))
        _kept["model"] = m
        _kept["filters"] = synth.mel_filterbank()
    return _kept["model"], _kept["filters"]


def _select(mode):
    native = "1" if mode == "w4a4" else "0"
    if os.environ.get("GLMASR_USE_CUTLASS_NVFP4") != native or os.environ.get("GLMASR_NVFP4_PAIRS") != native:
        os.environ["GLMASR_USE_CUTLASS_NVFP4"] = os.environ["GLMASR_NVFP4_PAIRS"] = native
        _lib.load().glmasr_decoder_forget_weights()


def _normal(shape, gen):
    return torch.randn(shape, generator=gen, device="cuda", dtype=torch.float32).to(torch.bfloat16)


def _token_ids(n, gen):
    return torch.randint(0, VOCAB, (n,), generator=gen, device="cuda", dtype=torch.int32)


def _prepare_linear(case, seed, gen):
    w = synth.seeded_weight_fast(case["n"], case["k"], seed)
    x = _normal((case["rows"], case["k"]), gen)
    return {"x": x, "w": w, "input_scale": synth.default_input_scale(x),
            "out": torch.empty((case["rows"], case["n"]), dtype=torch.bfloat16, device="cuda")}


def _prepare_layer(case, seed, gen):
    dims = {"H": HIDDEN, "KV": KV, "F": FFN}
    ws = []
    for i, (name, n, k) in enumerate(workloads.PROJ):
        w = synth.seeded_weight_fast(dims[n], dims[k], 16 * seed + i)
        w.input_scale = 0.002 * {"self_attn.o_proj": 4.0, "mlp.down_proj": 0.5}.get(name, 1.0)   # about amax / 2688
        ws.append(w)
    x = _normal((case["rows"], HIDDEN), gen)
    s = {"weights": ws, "lw": ops.make_layer_weights(*ws, hidden=HIDDEN, ffn=FFN)}
    if case["host"]:
        s["x"] = x.cpu().pin_memory()
        s["out"] = torch.empty_like(s["x"]).pin_memory()
    else:
        s["x"], s["out"] = x, torch.empty_like(x)
    return s


def _pages(lens, seed):
    """A paged KV pool with pages for lens[i] + 1 tokens of sequence i, handed out in random order as a pool that has
    been in use hands them out."""
    size = 16
    need = [n // size + 1 for n in lens]
    pool = engine.KVPool(sum(need) + 16, size, LAYERS, KV_HEADS, HEAD_DIM, len(lens), max(need) + 1)
    perm = np.random.default_rng(seed).permutation(sum(need) + 16).tolist()
    return pool, engine.BlockTables(pool, [[perm.pop() for _ in range(b)] for b in need])


def _prepare_decode(case, seed, gen):
    ctx = _contexts(case)
    pool, bts = _pages(ctx, seed)
    for t in (pool.k, pool.v):
        for layer in t:
            layer.normal_(generator=gen)
    lens = torch.tensor(ctx, dtype=torch.int32, device="cuda")
    _model()
    return {"pool": pool, "bts": bts, "lens": lens, "d_lens": lens.clone(), "h_lens": (ctypes.c_int * len(ctx))(*ctx),
            "kept_lens": (ctypes.c_int * len(ctx))(*ctx), "ids": _token_ids(len(ctx), gen),
            "logits": torch.empty((len(ctx), VOCAB), dtype=torch.bfloat16, device="cuda")}


def _prepare_prefill(case, seed, gen):
    model, _ = _model()
    lens = _prompt_lens(case)
    offs = np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)
    pool, bts = _pages(lens, seed)
    x = ops.embedding_lookup(model.embed, _token_ids(int(offs[-1]), gen))
    return {"pool": pool, "bts": bts, "x": x, "lens": lens, "offs": [int(o) for o in offs[:-1]],
            "last": torch.as_tensor(offs[1:] - 1, device="cuda"),
            "logits": torch.empty((len(lens), VOCAB), dtype=torch.bfloat16, device="cuda")}


def _samples(case, seed):
    """Float samples [windows, 480000], zero after each clip's end."""
    n = _clip_samples(case)
    pcm = torch.zeros((len(n), 30 * RATE), dtype=torch.float32, device="cuda")
    for i, k in enumerate(n):
        pcm[i, :k] = synthetic_window(1000 * (seed % 100000) + i)[:k]
    return pcm, n


def _prepare_audio(case, seed, gen):
    model, _ = _model()
    pcm, n = _samples(case, seed)
    return {"pcm": pcm, "padded": [160 * padded_feature_frames(feature_frames(k)) for k in n],
            "mel": torch.zeros((len(n), 3000 * MELS), dtype=torch.bfloat16, device="cuda")}


def _prepare_transcribe(case, seed, gen):
    model, filters = _model()
    pcm, n = _samples(case, seed)
    return {"pipe": AsrPipeline(model, filters, max_seqs=case["windows"], new_tokens=case["new_tokens"]),
            "pcm": pcm.cpu().pin_memory(), "samples": n}


def prepare(case, seed):
    if case["op"] != "audio":
        _select(case["mode"])
    gen = torch.Generator(device="cuda").manual_seed(seed)
    state = globals()["_prepare_" + case["op"]](case, seed, gen)
    state["case"] = case
    return state


# ---- one pass ---------------------------------------------------------------------------------------------------------
def _run_linear(s):
    w = s["w"]
    if s["case"]["mode"] == "w4a16":
        return ops.fp4_linear(s["x"], w.w_packed, w.w_scales, w.w_global_scale, out=s["out"])
    if ops.nvfp4_linear(s["out"], s["x"], w.w_packed, w.w_scales, s["input_scale"], w.w_global_scale) != 0:
        raise RuntimeError("nvfp4_linear refused its arguments")
    return s["out"]


def _run_layer(s):
    mode = ops.MODE_W4A4 if s["case"]["mode"] == "w4a4" else ops.MODE_W4A16
    if s["case"]["host"]:
        return ops.layer_proj_host(mode, s["x"], s["out"], s["lw"])
    return ops.layer_proj(mode, s["x"], s["lw"], out=s["out"])


def _next_tokens(s, model, hidden):
    """w4a4: FP4 head and arg-max, tokens stay on the device.  w4a16: the engine's own end of a step, bf16 head and
    arg-max with the tokens on the host."""
    if s["case"]["mode"] == "w4a16":
        return ops.lm_head_argmax_batched(hidden, model.embed), None
    lm = model.lm_head
    if ops.nvfp4_linear(s["logits"], hidden, lm.w_packed, lm.w_scales, model.lm_head_input_scale, lm.w_global_scale) != 0:
        raise RuntimeError("nvfp4_linear refused its arguments")
    return ops.argmax_rows(s["logits"]), s["logits"]


def _run_decode(s):
    model, _ = _model()
    s["d_lens"].copy_(s["lens"])             # the same position every pass: the step advances the lengths
    ctypes.memmove(s["h_lens"], s["kept_lens"], ctypes.sizeof(s["h_lens"]))
    hidden = ops.embedding_lookup(model.embed, s["ids"])
    engine.decode_step(model.ws, model.cfg, s["pool"], s["bts"], hidden, s["d_lens"], s["h_lens"])
    tokens, logits = _next_tokens(s, model, hidden)
    return {"hidden": hidden, "tokens": tokens, "logits": logits, "k": s["pool"].k, "v": s["pool"].v, "lens": s["d_lens"]}


def _run_prefill(s):
    model, _ = _model()
    hidden = s["x"].clone()                  # updated in place
    engine.prefill_paged_batched(model.ws, model.cfg, s["pool"], s["bts"], hidden, s["lens"], s["offs"])
    tokens, logits = _next_tokens(s, model, hidden[s["last"]])
    return {"hidden": hidden, "tokens": tokens, "logits": logits, "k": s["pool"].k, "v": s["pool"].v}


def _run_audio(s):
    model, filters = _model()
    _, frames = ops.mel_spectrogram_batched(s["pcm"], s["padded"], filters, time_major=True, out=s["mel"])
    embeddings, _ = ops.audio_encode_batched(model.ws, model.cfg, s["mel"], frames)
    return embeddings


def _run_transcribe(s):
    tokens = s["pipe"].transcribe(s["pcm"], s["samples"])
    return {"tokens": tokens, "k": s["pipe"].pool.k, "v": s["pipe"].pool.v}


def run(state):
    return globals()["_run_" + state["case"]["op"]](state)


# ---- what a pass cannot do without -------------------------------------------------------------------------------------
def _head_work(mode, rows):
    elem = 2.0 if mode == "w4a16" else FP4_BYTES
    return elem * VOCAB * HIDDEN + (0.0 if mode == "w4a16" else 2.0 * rows * VOCAB), 2.0 * rows * VOCAB * HIDDEN


def _decoder_work(rows, pairs, kv_read):
    """28 layers over `rows` tokens; pairs: (query, key) pairs of attention; kv_read: tokens whose K and V are read."""
    b = LAYERS * (FP4_BYTES * LAYER_PARAMS + 4.0 * KV * (kv_read + rows)) + 4.0 * rows * HIDDEN
    return b, LAYERS * (2.0 * rows * LAYER_PARAMS + 4.0 * pairs * HIDDEN)


def _audio_work(case):
    b, f = 0.0, 0.0
    for k in _clip_samples(case):
        t1 = padded_feature_frames(feature_frames(k))
        t2 = (t1 + 1) // 2
        b += 4.0 * k + 2.0 * (t2 // 4) * HIDDEN
        f += 2.0 * t1 * ENC * 3 * MELS + 2.0 * t2 * ENC * 3 * ENC
        f += ENC_LAYERS * (2.0 * t2 * (4 * ENC * ENC + 2 * ENC * ENC_FFN) + 4.0 * ENC * t2 * t2)
        f += 2.0 * (t2 // 4) * (4 * ENC * PROJ_MID + PROJ_MID * HIDDEN)
    weights = 3 * ENC * (MELS + ENC) + ENC_LAYERS * (4 * ENC * ENC + 2 * ENC * ENC_FFN) + 4 * ENC * PROJ_MID + PROJ_MID * HIDDEN
    return b + 2.0 * weights, f


def _prompt_work(mode, lens):
    rows = sum(lens)
    b, f = _decoder_work(rows, sum(n * (n + 1) / 2 for n in lens), 0)
    hb, hf = _head_work(mode, len(lens))
    return b + hb, f + hf


def work(case):
    op = case["op"]
    if op == "linear":
        m, n, k = case["rows"], case["n"], case["k"]
        b, f = FP4_BYTES * n * k + 2.0 * m * (n + k), 2.0 * m * n * k
    elif op == "layer":
        b, f = FP4_BYTES * LAYER_PARAMS + 4.0 * case["rows"] * HIDDEN, 2.0 * case["rows"] * LAYER_PARAMS
    elif op == "decode":
        ctx = [c + 1 for c in _contexts(case)]
        b, f = _decoder_work(len(ctx), sum(ctx), sum(ctx) - len(ctx))
        hb, hf = _head_work(case["mode"], len(ctx))
        b, f = b + hb, f + hf
    elif op == "prefill":
        b, f = _prompt_work(case["mode"], _prompt_lens(case))
    elif op == "audio":
        b, f = _audio_work(case)
    else:
        b, f = _audio_work(case)
        lens = [audio_tokens(feature_frames(k)) + PROMPT_EXTRA for k in _clip_samples(case)]
        pb, pf = _prompt_work("w4a4", lens)      # the pipeline's head is FP4
        b, f = b + pb, f + pf
        for step in range(1, case["new_tokens"]):
            ctx = [n + step for n in lens]
            db, df = _decoder_work(len(ctx), sum(ctx), sum(ctx) - len(ctx))
            hb, hf = _head_work("w4a4", len(ctx))
            b, f = b + db + hb, f + df + hf
    return {"bytes": b, "flops": f}


def tolerance(case):
    """bf16 results of fp32 sums: 4e-3 for one product (one rounding of the result, another order of the sum).  A stack
    of bf16 layers adds such a difference per layer to the residual stream: 2e-2 after 28 or 32 of them, 3e-2 after
    both stacks.  Activations that are quantised to e2m1 again and again make a chain that differs by whole quantisation
    steps wherever one value falls on the other side of a rounding boundary; a chain in w4a4 is held to 3e-2 all the
    same.  Tokens are whole numbers and win by a wide margin."""
    op, w4a16 = case["op"], case.get("mode") == "w4a16"
    if op == "linear":
        return {"rel": 4e-3, "max": 0.05}
    if op == "layer":
        return {"rel": 1e-2 if w4a16 else 2e-2, "max": 0.5}
    if op == "audio":
        return {"rel": 2e-2, "max": 0.5}
    return {"rel": 2e-2 if w4a16 and op != "transcribe" else 3e-2, "max": 0.8, "differ": 0.005}
