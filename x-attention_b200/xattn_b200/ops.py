"""Torch-facing operators.  Argument checks, device memory and streams are handled by the CPython module _host
(csrc/host_ops.cpp) on top of the C ABI.

All compute happens in libxattn_b200.so.  Tensors must live on a CUDA device (sm_100); every op
launches on torch's current stream of that device and does not synchronise.
"""
from __future__ import annotations

import ctypes as C
from typing import Optional, Tuple, Union

import torch

from . import _lib


class _Host:
    """The functions of the CPython module _host, which is loaded at the first use of one: the package has to be
    importable before anything is built (the build itself is part of it)."""

    def __getattr__(self, name):
        try:
            from . import _host as module
        except ImportError as e:
            raise _lib.XattnB200Error(f"_host.so is missing or does not load ({e}): build it with `python -m "
                                      "xattn_b200.build` (there is no fallback for this path)") from e
        module.init(_lib.XattnB200Error, lambda index: _status(torch.device("cuda", index)).data_ptr())
        self.__dict__.update({k: v for k, v in vars(module).items() if not k.startswith("_")})
        return self.__dict__[name]


_host = _Host()
_DT = {torch.bfloat16: _lib.BF16, torch.float16: _lib.F16}
_SEM = {"torch": _lib.SEMANTICS_TORCH, "triton": _lib.SEMANTICS_TRITON}

# Which of the reference's two estimate code paths is reproduced.  The reference picks by GPU
# name (xattn/src/Xattention.py:57-63: Triton only when the name contains "100", i.e. A100/H100);
# on a B200 it therefore runs its torch branch, which is the default here.
_estimate_semantics = "torch"


def set_estimate_semantics(name: str) -> None:
    """'torch' (default; what the unmodified reference computes on a B200) or 'triton'
    (the reference's Triton kernels, which keep all earlier chunks visible to later query chunks)."""
    global _estimate_semantics
    if name not in _SEM:
        raise ValueError("semantics must be 'torch' or 'triton'")
    _estimate_semantics = name


def get_estimate_semantics() -> str:
    return _estimate_semantics


# ------------------------------------------------------------------------------ status word
_status_words = {}


def _status(device: torch.device) -> torch.Tensor:
    """One pinned, device-visible int32 per device that kernels write on a bounded-wait timeout."""
    key = device.index if device.index is not None else torch.cuda.current_device()
    w = _status_words.get(key)
    if w is None:
        w = torch.zeros(1, dtype=torch.int32).pin_memory()
        _status_words[key] = w
    return w


def check_device_status(device: Optional[torch.device] = None, synchronize: bool = True) -> None:
    """Raise if a kernel reported a timed-out wait.  With synchronize=False only work that has
    already finished is covered."""
    dev = torch.device("cuda", torch.cuda.current_device()) if device is None else device
    if synchronize:
        torch.cuda.synchronize(dev)
    w = _status(dev)
    code = int(w[0])
    if code != 0:
        w[0] = 0
        _lib.check(code, "device status")


def _stream(t: torch.Tensor) -> int:
    return torch.cuda.current_stream(t.device).cuda_stream


def _require_cuda(*ts: torch.Tensor) -> None:
    for t in ts:
        if not t.is_cuda:
            raise _lib.XattnB200Error("xattn_b200 ops need CUDA tensors: there is no CPU path")


def _strides3(t: torch.Tensor) -> Tuple[int, int, int]:
    if t.stride(3) != 1:
        raise ValueError("head_dim must have unit stride")
    return t.stride(0), t.stride(1), t.stride(2)


def geometry(q_len: int, k_len: int, chunk_size: int, stride: int, block_size: int = 128) -> dict:
    out = (C.c_int * 8)()
    _lib.check(_lib.load().xattn_b200_estimate_geometry(q_len, k_len, chunk_size, stride, block_size, out),
               "estimate_geometry")
    keys = ("lq", "lk", "qb", "kb", "q_chunks", "k_chunks", "bpc", "block_offset")
    return dict(zip(keys, list(out)))


def default_chunk_size(k_len: int) -> int:
    return _lib.load().xattn_b200_default_chunk_size(k_len)


# ------------------------------------------------------------------------------ phase 1
def band_applies(k_len: int, chunk_size: int, causal: bool, semantics: Optional[str] = None) -> bool:
    """True when the estimate leaves every key block outside a row's own chunk at zero (the reference's torch
    branch on un-padded keys, xattn/src/Xattention.py:201), so that the sums can be kept as a chunk-wide band.
    (Block counts that are not multiples of four keep the dense layout.)"""
    return (bool(causal) and (semantics or _estimate_semantics) == "torch" and k_len % chunk_size == 0
            and (chunk_size // 128) % 4 == 0)


def estimate_block_sums(q: torch.Tensor, k: torch.Tensor, stride: int, block_size: int = 128,
                        chunk_size: int = 16384, norm: float = 1.0, causal: bool = True,
                        semantics: Optional[str] = None, band: bool = False) -> torch.Tensor:
    """fp32 attn_sums [B, Hq, q_blocks_pad, k_blocks_pad] of the antidiagonal estimate.

    band=True (see band_applies): only the key blocks of each row's own chunk are produced,
    [B, Hq, q_blocks_pad, chunk_size/block_size]; every other block has sum zero under the torch branch.

    q [B,Hq,Lq,D], k [B,Hkv,Lk,D] in bf16/fp16, or fp32 (split into three bf16 terms on the device so
    that the tensor-core product keeps fp32 accuracy)."""
    if band and not band_applies(k.shape[2], chunk_size, causal, semantics):
        raise ValueError("band layout needs the torch branch, causal, and k_len a multiple of chunk_size")
    return _host.estimate(q, k, stride, block_size, chunk_size, float(norm), bool(causal),
                          _SEM[semantics or _estimate_semantics], bool(band))


# ------------------------------------------------------------------------------ phase 2
def select_blocks(sums: torch.Tensor, blocks_per_chunk: int, block_offset: int,
                  threshold: Union[float, torch.Tensor], causal: bool = True, diagonal_cleanup: bool = True,
                  keep_sink: bool = False, keep_recent: bool = False,
                  list_shape: Optional[Tuple[int, int]] = None, want_mask: bool = True,
                  band_k_blocks: Optional[int] = None):
    """Threshold selection over fp32 sums [B,H,qb,kb].  Returns (mask bool or None, block_idx, block_cnt);
    the lists are None unless list_shape=(q_len, k_len) is given.  band_k_blocks=kb: `sums` is the chunk band
    [B,H,qb,blocks_per_chunk] of estimate_block_sums(band=True) and kb the full number of key blocks."""
    lq, lk = list_shape if list_shape is not None else (0, 0)
    return _host.select(sums, blocks_per_chunk, block_offset, threshold, bool(causal), bool(diagonal_cleanup),
                        bool(keep_sink), bool(keep_recent), bool(want_mask), lq, lk, int(band_k_blocks or 0))


def apply_rotary_pos_emb_(q: torch.Tensor, k: torch.Tensor, cos: torch.Tensor, sin: torch.Tensor) -> None:
    """In-place rotary embedding of q [B,Hq,L,D] and k [B,Hkv,L,D] (any strides, unit stride on D) with
    cos/sin [B,L,D] (or [1,L,D]) of the same 16-bit dtype: bit-identical to the reference's
    `apply_rotary_pos_emb` (xattn/src/load_llama.py:41-65), one launch for both tensors."""
    _require_cuda(q, k, cos, sin)
    if q.dtype not in _DT or k.dtype != q.dtype or cos.dtype != q.dtype or sin.dtype != q.dtype:
        raise ValueError("apply_rotary_pos_emb_: q, k, cos, sin must share one 16-bit dtype (bf16 or fp16)")
    B, Hq, L, D = q.shape
    Hkv = k.shape[1]
    if k.shape != (B, Hkv, L, D):
        raise ValueError("apply_rotary_pos_emb_: q and k must share batch, length and head_dim")
    if cos.dim() != 3 or cos.shape[1:] != (L, D) or cos.shape[0] not in (1, B) or sin.shape != cos.shape:
        raise ValueError("apply_rotary_pos_emb_: cos/sin must be [batch or 1, len, head_dim]")
    if cos.stride(2) != 1 or sin.stride(2) != 1 or sin.stride() != cos.stride():
        cos, sin = cos.contiguous(), sin.contiguous()
    cs_b = cos.stride(0) if cos.shape[0] == B and B > 1 else 0
    lib = _lib.load()
    _lib.check(lib.xattn_b200_rope_qk(q.data_ptr(), k.data_ptr(), _DT[q.dtype], B, Hq, Hkv, L, D, *_strides3(q),
                                      *_strides3(k), cos.data_ptr(), sin.data_ptr(), cs_b, cos.stride(1),
                                      _stream(q)), "rope_qk")


def mask_to_lists(mask: torch.Tensor, q_len: int, k_len: int, causal: bool):
    _require_cuda(mask)
    lib = _lib.load()
    m = mask.contiguous()
    m = m.view(torch.uint8) if m.dtype == torch.bool else m.to(torch.uint8)
    B, H, MQ, MK = m.shape
    lqb, lkb = (q_len + 127) // 128, (k_len + 127) // 128
    idx = torch.empty(B, H, lqb, lkb, dtype=torch.int32, device=m.device)
    cnt = torch.empty(B, H, lqb, dtype=torch.int32, device=m.device)
    _lib.check(lib.xattn_b200_mask_to_lists(m.data_ptr(), B, H, MQ, MK, q_len, k_len, int(causal),
                                            idx.data_ptr(), cnt.data_ptr(), _stream(m)), "mask_to_lists")
    return idx, cnt


# ------------------------------------------------------------------------------ phase 3
# Causal calls are not offered scratch memory by default: the general kernel now loads K/V once for two query heads of a
# kv group itself, and the split into two kernels no longer gains (Llama-3.1-8B at 128K tokens, where 95 % of the blocks
# qualify for the pair kernel: 700 us with the split, 596 us without).
def pair_split_share(percent: Optional[int] = None) -> int:
    """Share (per cent) of a call's listed blocks that must qualify for the pair kernel before the library splits
    the call between the two attention kernels (process-wide; 0: whenever anything qualifies, 101: never).
    Returns the previous value; without an argument only reads it."""
    return int(_lib.load().xattn_b200_block_sparse_attn_split_share(-1 if percent is None else int(percent)))


def block_sparse_attention(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, block_idx: Optional[torch.Tensor],
                           block_cnt: Optional[torch.Tensor], causal: bool = True, scale: Optional[float] = None,
                           out: Optional[torch.Tensor] = None, use_workspace: Optional[bool] = None) -> torch.Tensor:
    """q [B,Hq,Lq,128], k/v [B,Hkv,Lk,128] (bf16/fp16; fp32 is computed in bf16) -> [B,Hq,Lq,128], returned
    as a transposed view of [B,Lq,Hq,128] storage, like the reference's output (Xattention.py:392-394).
    Without lists (block_idx and block_cnt None) the call is dense: every block that holds a visible key.
    `out`, if given, is a [B,Hq,Lq,128] tensor of the compute dtype (any strides, unit stride on the last
    dimension, 16-byte aligned rows) that receives the result instead.  `use_workspace=True` hands the library
    scratch memory (xattn_b200_block_sparse_attn_ws).  Causal calls: it may then send the rows whose kv group shares a
    list of one or two blocks to a kernel of their own, provided those rows list at least `pair_split_share()` per cent
    of the blocks, which it finds out on the device; by default (None) no memory is offered.  Non-causal calls: the
    work is sorted by list length before it is handed to the SMs (one small kernel); offered by default from
    16 items per SM on, with more than 40 key blocks from 4 on.  False: the general kernel alone, work in its natural order."""
    return _host.attention(q, k, v, block_idx, block_cnt, bool(causal), scale, out, use_workspace)


def decode_attention(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, scale: Optional[float] = None) -> torch.Tensor:
    """Dense attention of one query token per sequence: q [B,Hq,1,128] against the whole cache k/v [B,Hkv,Lk,128]
    (bf16/fp16; fp32 is computed in bf16) -> [B,Hq,1,128], a transposed view of [B,1,Hq,128] storage."""
    return _host.decode(q, k, v, scale)


def prefill(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, stride: int, norm: float, threshold, block_size: int,
            causal: bool, chunk_size: Optional[int], keep_sink: bool, keep_recent: bool,
            out: Optional[torch.Tensor] = None) -> torch.Tensor:
    """Estimate, selection and attention in one call (chunk_size None: the default of the length)."""
    return _host.prefill(q, k, v, stride, norm, threshold, block_size, causal, chunk_size, keep_sink, keep_recent,
                         _SEM[_estimate_semantics], out)


def estimate_and_select(q: torch.Tensor, k: torch.Tensor, stride: int, norm: float, threshold, block_size: int, causal: bool,
                        chunk_size: int, keep_sink: bool, keep_recent: bool):
    """(block sums in q's type, mask)"""
    return _host.estimate_and_select(q, k, stride, block_size, chunk_size, norm, causal, _SEM[_estimate_semantics], threshold,
                                     keep_sink, keep_recent)
