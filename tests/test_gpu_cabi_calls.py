"""Entry points of the C ABI that the Python layer does not call, against those that it does."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _stream():
    return torch.cuda.current_stream().cuda_stream


def _qkv(seed, hq, hkv, lq, lk, dtype):
    g = torch.Generator(device=DEV).manual_seed(seed)
    return [torch.randn(2, h, n, 128, device=DEV, generator=g).to(dtype) for h, n in ((hq, lq), (hkv, lk), (hkv, lk))]


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("kb,bpc", [(5, 5), (130, 13), (512, 128), (1024, 64)])
def test_select_rounded(kb, bpc, dtype):
    from xattn_b200 import _lib, ops
    g = torch.Generator(device=DEV).manual_seed(kb)
    qb = kb // bpc * bpc
    sums = torch.rand(2, 3, qb, kb, device=DEV, generator=g) ** 8
    off = kb - qb
    want = ops.select_blocks(sums, bpc, off, 0.9, True, True, True, False)[0]
    mask = torch.empty(sums.shape, dtype=torch.bool, device=DEV)
    rounded = torch.empty(sums.shape, dtype=dtype, device=DEV)
    _lib.check(_lib.load().xattn_b200_select_rounded(sums.data_ptr(), 2, 3, qb, kb, bpc, off, 1, 1, 0.9, None, 1, 0, mask.data_ptr(),
                                                     rounded.data_ptr(), _lib.BF16 if dtype == torch.bfloat16 else _lib.F16, None, _stream()),
               "select_rounded")
    assert torch.equal(mask, want) and torch.equal(rounded, sums.to(dtype))


@pytest.mark.parametrize("causal", [True, False])
def test_attention_with_scratch(causal):
    from xattn_b200 import _lib, ops
    lq, lk, hq, hkv = 2011, 2200, 4, 2
    q, k, v = _qkv(1, hq, hkv, lq, lk, torch.bfloat16)
    g = torch.Generator(device=DEV).manual_seed(2)
    mask = torch.rand(2, hq, 16, 18, device=DEV, generator=g) < 0.4
    idx, cnt = ops.mask_to_lists(mask, lq, lk, causal)
    want = ops.block_sparse_attention(q, k, v, idx, cnt, causal, use_workspace=True)
    lib = _lib.load()
    ws = torch.empty(max(16, lib.xattn_b200_block_sparse_attn_workspace_bytes(2, hq, hkv, lq, lk)), dtype=torch.uint8, device=DEV)
    out = torch.full_like(want, float("nan"))
    _lib.check(lib.xattn_b200_block_sparse_attn_ws(
        q.data_ptr(), k.data_ptr(), v.data_ptr(), _lib.BF16, 2, hq, hkv, lq, lk, 128, *q.stride()[:3], *k.stride()[:3], *v.stride()[:3],
        idx.data_ptr(), cnt.data_ptr(), int(causal), 128 ** -0.5, out.data_ptr(), *out.stride()[:3], ws.data_ptr(), ws.numel(), None, _stream()),
        "block_sparse_attn_ws")
    assert torch.equal(out, want)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("lq,lk,chunk", [(1003, 1003, 2048), (4096, 4096, 2048), (700, 9000, 1024), (8192, 8192, 8192)])
def test_estimate_and_selection_in_one_call(lq, lk, chunk, dtype):
    """Mask, lists and rounded sums of one call, which the Python layer asks for one at a time; in batch."""
    from xattn_b200 import _lib, ops
    hq, hkv, stride = 4, 2, 16
    q, k, _ = _qkv(lq, hq, hkv, lq, lk, dtype)
    geo = ops.geometry(lq, lk, chunk, stride)
    sums = ops.estimate_block_sums(q, k, stride, 128, chunk, 1.0, True)
    thr = torch.rand(hq, device=DEV) * 0.3 + 0.65
    want, idx, cnt = ops.select_blocks(sums, geo["bpc"], geo["block_offset"], thr, True, True, False, True, list_shape=(lq, lk))
    lib = _lib.load()
    ws = torch.empty(lib.xattn_b200_estimate_workspace_bytes_ex(2, hq, lq, lk, stride, 128, chunk, 1, _lib.SEMANTICS_TORCH), dtype=torch.uint8,
                     device=DEV)
    a = _lib.EstimateSelectArgs()
    a.q, a.k, a.dtype = q.data_ptr(), k.data_ptr(), _lib.BF16 if dtype == torch.bfloat16 else _lib.F16
    a.batch, a.hq, a.hkv, a.q_len, a.k_len, a.head_dim = 2, hq, hkv, lq, lk, 128
    a.q_stride_b, a.q_stride_h, a.q_stride_l = q.stride()[:3]
    a.k_stride_b, a.k_stride_h, a.k_stride_l = k.stride()[:3]
    a.stride, a.block_size, a.chunk_size, a.scale, a.causal, a.semantics = stride, 128, chunk, 128 ** -0.5 / stride, 1, _lib.SEMANTICS_TORCH
    got_sums, got_mask = torch.full_like(sums, float("nan")), torch.empty_like(want)
    rounded, got_idx, got_cnt = torch.empty(sums.shape, dtype=dtype, device=DEV), torch.full_like(idx, -1), torch.full_like(cnt, -1)
    a.attn_sums, a.workspace, a.workspace_bytes = got_sums.data_ptr(), ws.data_ptr(), ws.numel()
    a.threshold_per_head, a.keep_recent = thr.data_ptr(), 1
    a.mask, a.rounded, a.rounded_dtype = got_mask.data_ptr(), rounded.data_ptr(), a.dtype
    a.block_idx, a.block_cnt, a.list_q_len, a.list_k_len = got_idx.data_ptr(), got_cnt.data_ptr(), lq, lk
    _lib.check(lib.xattn_b200_estimate_select(ctypes.byref(a), _stream()), "estimate_select")
    assert torch.equal(got_sums, sums) and torch.equal(rounded, sums.to(dtype)) and torch.equal(got_mask, want) and torch.equal(got_cnt, cnt)
    listed = torch.arange(idx.shape[-1], device=DEV) < cnt[..., None]
    assert torch.equal(got_idx[listed], idx[listed]) and (got_idx[~listed] == -1).all()
    # what is refused leaves no work in flight
    n0 = lib.xattn_b200_launch_count()
    a.workspace_bytes = 0
    assert lib.xattn_b200_estimate_select(ctypes.byref(a), _stream()) != 0
    a.workspace_bytes, a.list_q_len = ws.numel(), 0
    assert lib.xattn_b200_estimate_select(ctypes.byref(a), _stream()) != 0
    assert lib.xattn_b200_estimate_select(None, _stream()) != 0
    assert lib.xattn_b200_launch_count() == n0
