"""Full (non-causal) self-attention of a video-diffusion block in the reference's "xattn" mode.

Reference: eval/HunyuanVideo/hyvideo/modules/attenion.py:132-166.  The sequence of a sample is
[valid image+text tokens | padded text tail]; the two segments attend only within themselves
(`cu_seqlens = [0, valid, total]`).  The valid segment goes through XAttention (non-causal; dense attention
instead when threshold >= 1, which the model uses during its warm-up steps, models.py:211), the tail is dense.
Both dense cases run through the same attention kernel without block lists, so no third-party attention package is
involved.
"""
from __future__ import annotations

import torch

from . import ops


def _dense(q, k, v, out):
    ops.block_sparse_attention(q, k, v, None, None, causal=False, out=out)


def _xattn(q, k, v, out, threshold, stride):
    """Non-causal Xattention_prefill (xattn/src/Xattention.py:302-402) writing into `out`."""
    ops.prefill(q, k, v, stride, 1.0, threshold, 128, False, None, False, False, out)


def xattn_varlen_attention(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, cu_seqlens_q, cu_seqlens_kv,
                           threshold: float = 0.95, stride: int = 8) -> torch.Tensor:
    """q, k, v [1, heads, total, D] (16 bit, any strides with unit stride on D); cu_seqlens_* = [0, valid, total].
    Returns [1, heads, total, D] (a view of [1, total, heads, D] storage).  The two segments are read through
    strided views and written straight into their rows of the result: no copy of q, k, v or of the outputs,
    whatever the segment lengths."""
    v0q, v1q = int(cu_seqlens_q[1]), int(cu_seqlens_q[2])
    v0k, v1k = int(cu_seqlens_kv[1]), int(cu_seqlens_kv[2])
    B, H, _, D = q.shape
    res = torch.empty(B, v1q, H, D, dtype=q.dtype, device=q.device).transpose(1, 2)
    q1, k1, v1 = q[:, :, :v0q], k[:, :, :v0k], v[:, :, :v0k]
    if threshold < 1:
        _xattn(q1, k1, v1, res[:, :, :v0q], threshold, stride)
    else:
        _dense(q1, k1, v1, res[:, :, :v0q])
    if v1q > v0q:
        _dense(q[:, :, v0q:v1q], k[:, :, v0k:v1k], v[:, :, v0k:v1k], res[:, :, v0q:v1q])
    return res
