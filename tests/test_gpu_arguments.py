"""What the operators refuse on the host, before anything is launched, and odd forms of tensors that they take."""
import os
import subprocess
import sys

import pytest
import torch

import xattn_b200
from xattn_b200 import api, llama_shim, ops
from xattn_b200._lib import XattnB200Error

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.fixture(autouse=True)
def _status_clean():
    yield
    xattn_b200.check_device_status()


def _qkv(lq, lk, hq=4, hkv=2, batch=1, dtype=torch.bfloat16):
    g = torch.Generator(device=DEV).manual_seed(lq + lk)
    return [torch.randn(batch, h, n, 128, generator=g, device=DEV).to(dtype) for h, n in ((hq, lq), (hkv, lk), (hkv, lk))]


def _calls(q, k, v):
    """Every operator that makes its tensor maps from q's and k's sizes."""
    cfg = llama_shim.FastPrefillConfig(0.9, num_heads=q.shape[1])
    calls = [lambda: llama_shim.attention_core(q, k, v, 0, cfg)] if q.shape[2] == 1 else [
        lambda: ops.block_sparse_attention(q, k, v, None, None, True), lambda: api.Xattention_prefill(q, k, v, 16)]
    return calls


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("lq,which,dim,size", [(1, 1, 0, 1), (1, 2, 0, 1), *[(n, w, d, s) for n in (1, 300) for w, d, s in (
    (2, 1, 0), (2, 1, 1), (2, 2, 200), (1, 3, 64), (2, 3, 64))]])
def test_smaller_keys_or_values_are_refused(lq, which, dim, size, dtype):
    """Keys or values (tensor 1, 2) whose batch, heads, length or head_dim is below what the call reads."""
    t = _qkv(lq, 300, batch=2 if dim == 0 else 1, dtype=dtype)
    t[which] = t[which].narrow(dim, 0, size)
    for call in _calls(*t):
        with pytest.raises(ValueError):
            call()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("lq", [1, 300])
def test_of_larger_values_the_leading_part_counts(lq, dtype):
    q, k, v = _qkv(lq, 300, dtype=dtype)
    longer = torch.full((2, 3, 345, 128), float("nan"), device=DEV, dtype=dtype)
    longer[:1, :2, :300] = v
    for call, want in zip(_calls(q, k, longer), _calls(q, k, v)):
        assert torch.equal(call(), want())


def test_lists_of_another_type_are_refused():
    q, k, v = _qkv(300, 300)
    idx, cnt = ops.mask_to_lists(torch.ones(1, 4, 3, 3, dtype=torch.bool, device=DEV), 300, 300, True)
    with pytest.raises(ValueError):
        ops.block_sparse_attention(q, k, v, idx.long(), cnt.long(), True)


def test_divisors_of_zero_raise():
    """No key heads, a chunk of no tokens, a norm of zero: errors of Python, not of the process."""
    q, k, v = _qkv(1, 300)
    for kk, vv in ((k[:, :0], v[:, :0]), (k[:, :0], v)):
        with pytest.raises(XattnB200Error):
            ops.decode_attention(q, kk, vv)
    q, k, v = _qkv(300, 300)
    for chunk in (0, -128, 100):
        with pytest.raises(XattnB200Error):
            api.Xattention_prefill(q, k, v, 16, chunk_size=chunk)
        with pytest.raises(XattnB200Error):
            api.xattn_estimate(q, k, 128, 16, chunk_size=chunk)
    with pytest.raises(XattnB200Error):
        api.Xattention_prefill(q, k, v, 0)
    for x in (q, q.float()):
        with pytest.raises(ZeroDivisionError):
            api.Xattention_prefill(x, k.to(x.dtype), v.to(x.dtype), 16, norm=0)
        with pytest.raises(ZeroDivisionError):
            api.xattn_estimate(x, k.to(x.dtype), 128, 16, norm=0)


@pytest.mark.parametrize("hq", [1, 4])
def test_decode_step_of_odd_batch_and_head_strides(hq):
    """A query whose strides of extent 1 are odd: a view of a longer row, contiguous as far as torch is concerned."""
    q, k, v = _qkv(1, 300, hq=hq, hkv=1)
    row = torch.randn(1, hq * 128 + 1, device=DEV).bfloat16()
    odd = row.as_strided(q.shape, (hq * 128 + 1, 128 if hq > 1 else 129, 128, 1))
    assert torch.equal(ops.decode_attention(odd, k, v), ops.decode_attention(odd.clone(), k, v))


def test_decode_step_of_more_sequences_than_a_grid_dimension_holds():
    q, k, v = _qkv(1, 2, hq=1, hkv=1, batch=65537)
    out = ops.decode_attention(q, k, v)
    want = torch.nn.functional.scaled_dot_product_attention(q[-5:].float(), k[-5:].float(), v[-5:].float())
    # probabilities and outputs are rounded to bf16, 2^-9 relative each, of values up to about 5
    assert (out[-5:].float() - want).abs().max() < 2e-2 and bool(torch.isfinite(out.float()).all())


def test_thresholds_are_what_float_takes():
    q, k, v = _qkv(300, 300)
    want = api.Xattention_prefill(q, k, v, 16, threshold=0.75)
    for threshold in ("0.75", torch.full((4,), 0.75), torch.full((1, 4, 1), 0.75, device=DEV, dtype=torch.float64)):
        assert torch.equal(api.Xattention_prefill(q, k, v, 16, threshold=threshold), want)
    with pytest.raises(ValueError):
        api.Xattention_prefill(q, k, v, 16, threshold="high")
    with pytest.raises(TypeError):
        api.Xattention_prefill(q, k, v, 16, threshold=None)


def test_a_failed_launch_is_not_reported_twice():
    """A launch refused by the runtime (into a stream capture that a synchronisation has invalidated) fails its own call and
    no later one.  In a process of its own: an abandoned capture is not for other tests to inherit."""
    code = """
import torch
from xattn_b200 import _lib, ops
lib = _lib.load()
mask = torch.ones(1, 2, 3, 3, dtype=torch.uint8, device="cuda")
idx, cnt = ops.mask_to_lists(mask, 300, 300, True)
def call():
    return lib.xattn_b200_mask_to_lists(mask.data_ptr(), 1, 2, 3, 3, 300, 300, 1, idx.data_ptr(), cnt.data_ptr(),
                                        torch.cuda.current_stream().cuda_stream)
torch.cuda.synchronize()
graph = torch.cuda.CUDAGraph()
with torch.cuda.stream(torch.cuda.Stream()):
    graph.capture_begin(capture_error_mode="global")
    try:
        torch.cuda.synchronize()
    except RuntimeError:
        pass
    refused = call()
    try:
        graph.capture_end()
    except RuntimeError:
        pass
print("codes", refused, call())
"""
    path = os.pathsep.join(p for p in sys.path if p)
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=120, env=dict(os.environ, PYTHONPATH=path))
    assert "codes 3 0" in r.stdout, r.stdout + r.stderr
