"""The calls that a user of this package makes, as cases that can be timed.

A case is one layer's attention call as a model makes it, through the package's public entry points: a decode step
against a key cache, the prefill of a prompt, a prompt's next piece against the cache, dense attention for layers (or
diffusion steps) that do not go sparse, the mask study on the estimate alone, and full attention over the tokens of a
video.  Inputs come from the seeded generators of `xattn_b200.synth` on the GPU, because how many key blocks a row
keeps, and with it the work of the sparse calls, follows from the values.

    kind       entry point                                         what it stands for
    decode     llama_shim.attention_core, one query per sequence   a generated token against the cache
    layer      llama_shim.attention_core, "xattn"                  a decoder layer's prefill: q as the [B, L, H, D] view
                                                                   that the projection leaves, K/V from the cache
    full       llama_shim.attention_core, "full"                   the dense layer of the same model
    prefill    Xattention_prefill                                  the operator itself, [B, H, L, D] tensors
    estimate   xattn_estimate                                      block sums and mask, as for choosing thresholds
    dit        dit_shim.xattn_varlen_attention                     non-causal attention of a video-diffusion block

`tokens` names the generator: "text" (decoder text), "video" (text, frames, text), "dit" (frames x rows x columns plus
text).  `threshold` 0 stands for the per-head table that FastPrefillConfig loads for the stride; `chunk` 0 for the
default estimate chunk of the length.
"""
import math
import os
import sys

import torch

sys.path.insert(0, os.path.join(os.getcwd(), "x-attention_b200"))

import xattn_b200  # noqa: E402
from xattn_b200 import llama_shim, synth  # noqa: E402
from xattn_b200.dit_shim import xattn_varlen_attention  # noqa: E402

D = 128
BLOCK = 128
LAYER = 13                    # the layer whose row of the threshold table is used
TEXT_PRE, FRAME_TOKENS, TEXT_POST = 512, 256, 256
DIT_ROWS, DIT_COLS, DIT_TEXT = 45, 80, 256
DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}


def _case(kind, hq, hkv, q_len, k_len, **more):
    c = dict(kind=kind, batch=1, hq=hq, hkv=hkv, q_len=q_len, k_len=k_len, dtype="bf16", stride=16, chunk=0,
             threshold=0.9, tokens="text")
    c.update(more)
    return c


def listed():
    return [
        # a generated token after a short exchange: the smallest call there is, all latency and launches
        dict(_case("decode", 32, 8, 1, 2011), name="decode_2k"),
        # a generated token at the end of a long document: the key cache of one layer read once
        dict(_case("decode", 32, 8, 1, 131072), name="decode_128k"),
        # a short prompt with the model's own threshold table; no multiple of the block or of the stride
        dict(_case("layer", 32, 8, 1003, 1003, threshold=0.0), name="prompt_1k"),
        # the reference-sized layer in 32 bit (one key head per query head)
        dict(_case("prefill", 32, 32, 4096, 4096, dtype="fp32", chunk=2048), name="prefill_4k_fp32"),
        # an ordinary prompt of ragged length in fp16, the finer stride with its table
        dict(_case("layer", 32, 8, 9973, 9973, dtype="fp16", stride=8, threshold=0.0), name="prompt_10k_fp16"),
        # dense layer of the same model on a medium prompt (the baseline metric, and layers kept dense)
        dict(_case("full", 32, 8, 15000, 15000), name="full_15k"),
        # the benchmark's layer
        dict(_case("prefill", 32, 8, 32768, 32768, stride=8, chunk=16384), name="prefill_32k"),
        # the mask study at the same length: block sums and mask, default chunk
        dict(_case("estimate", 32, 8, 32768, 32768), name="estimate_32k"),
        # a long prompt arriving in pieces: 4096 new tokens at the end of 65536
        dict(_case("layer", 32, 8, 4096, 65536, threshold=0.0), name="continue_64k"),
        # a long document in one piece
        dict(_case("prefill", 32, 8, 131072, 131072), name="prefill_128k"),
        # video understanding: 240 frames between text, whose rows keep most of the past
        dict(_case("prefill", 28, 4, 62208, 62208, tokens="video"), name="video_62k"),
        # a video-diffusion block: 33 latent frames, text tail partly padding, both segment lengths ragged
        dict(_case("dit", 24, 24, 118940, 119056, stride=8, threshold=0.95, tokens="dit"), name="dit_119k"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["decode", "decode", "layer", "layer", "layer", "prefill", "prefill", "full", "estimate",
                       "continue", "video", "dit"])
    hq, hkv = rng.choice([(32, 8), (32, 8), (28, 4)])
    dtype = rng.choice(["bf16", "bf16", "fp16"])
    stride = rng.choice([8, 16])
    threshold = round(rng.uniform(0.8, 0.97), 3)
    if hq == 32 and rng.random() < 0.5:
        threshold = 0.0
    if kind == "decode":
        batch = rng.choice([1, 1, 2, 4, 8])
        return _case("decode", hq, hkv, 1, _log_int(rng, 200, 262144 // batch if batch > 1 else 131072), batch=batch,
                     dtype=dtype)
    if kind == "full":
        n = _log_int(rng, 300, 20000)
        return _case("full", hq, hkv, n, n, dtype=dtype)
    if kind == "continue":
        k_len = _log_int(rng, 4096, 131072)
        q_len = min(k_len // 2, _log_int(rng, 512, 8192))
        return _case("layer", hq, hkv, q_len, k_len, dtype=dtype, stride=stride, threshold=threshold)
    if kind == "video":
        n = TEXT_PRE + FRAME_TOKENS * _log_int(rng, 8, 240) + TEXT_POST
        return _case("prefill", 28, 4, n, n, dtype=dtype, threshold=round(rng.uniform(0.8, 0.9), 3), tokens="video")
    if kind == "dit":
        frames = rng.randint(3, 33)
        total = frames * DIT_ROWS * DIT_COLS + DIT_TEXT
        # a text of any length up to the padded one; the first denoising steps run dense (here: short clips)
        threshold = 1.0 if frames <= 8 and rng.random() < 0.3 else round(rng.uniform(0.9, 0.96), 3)
        return _case("dit", 24, 24, total - rng.randint(1, DIT_TEXT - 8), total, stride=8, threshold=threshold, tokens="dit")
    n = _log_int(rng, 200, 131072)
    if rng.random() < 0.3:                           # lengths that fill their chunks, as a padded batch has them
        n = max(2048, n // 2048 * 2048)
    if kind in ("prefill", "estimate"):
        threshold = threshold or 0.9
        if n <= 8192 and rng.random() < 0.4:
            return _case(kind, 32, 32, n, n, dtype="fp32", stride=stride, threshold=threshold)
        if n <= 32768 and rng.random() < 0.2:
            stride = 4
    return _case(kind, hq, hkv, n, n, dtype=dtype, stride=stride, threshold=threshold)


# ------------------------------------------------------------------------------------------------ inputs
def _blhd(x):
    """The same values behind [B, L, H, D] storage, seen as [B, H, L, D]: how a projection leaves them."""
    return x.transpose(1, 2).contiguous().transpose(1, 2)


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind, dt = case["kind"], DTYPES[case["dtype"]]
    B, hq, hkv, lq, lk = case["batch"], case["hq"], case["hkv"], case["q_len"], case["k_len"]
    if kind == "decode":
        q, k, v = (torch.randn(B, h, n, D, generator=gen, device="cuda").to(dt) for h, n in ((hq, 1), (hkv, lk), (hkv, lk)))
        return dict(case=case, q=_blhd(q), k=k, v=v, config=llama_shim.FastPrefillConfig(0.9, num_heads=hq))
    if case["tokens"] == "video":
        q, k, v = synth.video_like(gen, hq, hkv, TEXT_PRE, (lk - TEXT_PRE - TEXT_POST) // FRAME_TOKENS, FRAME_TOKENS, TEXT_POST)
    elif case["tokens"] == "dit":
        q, k, v = synth.dit_like(gen, hq, (lk - DIT_TEXT) // (DIT_ROWS * DIT_COLS), DIT_ROWS, DIT_COLS, DIT_TEXT, pad_to=1)
    else:
        q, k, v = synth.llama_like(gen, hq, hkv, lk)
    q, k, v = q.to(dt), k.to(dt), v.to(dt)
    state = dict(case=case, q=q, k=k, v=v)
    if kind == "dit":
        state["cu"] = torch.tensor([0, lq, lk], dtype=torch.int32)
    elif kind in ("layer", "full"):
        state["q"] = _blhd(q[:, :, lk - lq:])
        state["config"] = llama_shim.FastPrefillConfig(case["threshold"] or None, stride=case["stride"], num_heads=hq,
                                                       metric="full" if kind == "full" else "xattn")
    return state


def run(state):
    c, q, k, v = state["case"], state["q"], state["k"], state["v"]
    kind = c["kind"]
    if kind in ("decode", "layer", "full"):
        return llama_shim.attention_core(q, k, v, LAYER, state["config"])
    if kind == "dit":
        return xattn_varlen_attention(q, k, v, state["cu"], state["cu"], threshold=c["threshold"], stride=c["stride"])
    if kind == "estimate":
        more = dict(chunk_size=c["chunk"]) if c["chunk"] else {}
        return xattn_b200.xattn_estimate(q, k, BLOCK, c["stride"], threshold=c["threshold"], **more)
    return xattn_b200.Xattention_prefill(q, k, v, c["stride"], threshold=c["threshold"], chunk_size=c["chunk"] or None)


# ------------------------------------------------------------------------------------------------ work
def _chunk(case):
    """The estimate chunk of the call: the one given, the default of xattn_estimate, or that of the length."""
    if case["chunk"]:
        return case["chunk"]
    if case["kind"] == "estimate":
        return 16384
    n = case["q_len"] if case["kind"] == "dit" else case["k_len"]
    p = 1 << max(0, (n - 1).bit_length())
    return max(2048, min(max(p, 2048), 128 * 1024 * 2048 // p))


def _estimate_cells(case, chunk):
    """Visible (row, column) cells of the strided score matrix of one query head."""
    S = case["stride"]
    if case["kind"] == "dit":
        return (case["q_len"] / S) ** 2
    r, c = case["q_len"] / S, case["k_len"] / S
    if case["k_len"] % chunk == 0:                   # whole chunks: a row sees its own chunk only
        return r * min(chunk / S, c) / 2
    return r * (c - r / 2)


def _kept_blocks(case, chunk):
    """Key blocks that a query block keeps on these inputs at threshold 0.9, on average (diagonal counted as half a
    block): what the selection gives on the listed cases, rounded."""
    past = case["k_len"] / BLOCK - case["q_len"] / BLOCK / 2
    if case["tokens"] == "video":
        return KEPT_VIDEO * past
    if case["tokens"] == "dit":
        return min(case["q_len"] / BLOCK, KEPT_DIT)
    return min(past, KEPT_TEXT)


KEPT_TEXT, KEPT_VIDEO, KEPT_DIT = 2.0, 0.75, 30.0


def work(case):
    kind, size = case["kind"], 4 if case["dtype"] == "fp32" else 2
    B, hq, hkv, lq, lk = case["batch"], case["hq"], case["hkv"], case["q_len"], case["k_len"]
    if kind == "dit":
        tail = lk - lq
        io = 4 * hq * lk * D * size
        dense = 4.0 * D * hq * tail * tail
        if case["threshold"] >= 1:
            return {"bytes": io, "flops": dense + 4.0 * D * hq * lq * lq}
        chunk = _chunk(case)
        est = 2.0 * D * case["stride"] * hq * _estimate_cells(case, chunk)
        return {"bytes": io, "flops": dense + est + 4.0 * D * BLOCK * hq * lq * _kept_blocks(case, chunk)}
    io = B * (2 * hq * lq + 2 * hkv * lk) * D * size
    if kind == "decode":
        return {"bytes": io, "flops": 4.0 * D * B * hq * lk}
    if kind == "full":
        return {"bytes": io, "flops": 4.0 * D * hq * (lq * lk - lq * lq / 2)}
    chunk = _chunk(case)
    est = 2.0 * D * case["stride"] * hq * _estimate_cells(case, chunk)
    if kind == "estimate":
        pad = -(-lk // chunk) * chunk // BLOCK
        return {"bytes": (hq * lq + hkv * lk) * D * size + hq * pad * pad * (size + 1), "flops": est}
    return {"bytes": io, "flops": est + 4.0 * D * BLOCK * hq * lq * _kept_blocks(case, chunk)}


def tolerance(case):
    # bf16 carries 8 bits: probabilities and outputs are rounded to it (2^-9 each), and so are the block sums that
    # xattn_estimate returns; fp16 carries 11.  32-bit inputs are attended in bf16.  Whole values: the mask, where
    # blocks whose score lies at the threshold to within the rounding of 32-bit sums may go either way.
    if case["kind"] == "estimate":
        return {"rel": 1e-5 if case["dtype"] == "fp32" else (1e-3 if case["dtype"] == "fp16" else 4e-3), "differ": 1e-4}
    return {"rel": 4e-3 if case["dtype"] == "fp16" else 1e-2}
