"""The selection inside the estimate's kernel against the selection as a kernel of its own on the same sums."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


# (tokens, stride, chunk): every way a row of sums is finished in the GEMM's epilogue -- clusters of four and of two CTAs, one tile
# per CTA and many, tiles of 128 and 256 columns, CTA pairs; ragged lengths, rows of padding, chunks of their own and all of the keys
@pytest.mark.parametrize("hq,hkv", [(4, 2), (3, 3), (32, 8)])
@pytest.mark.parametrize("q_len,k_len,stride,chunk", [
    (3, 3, 16, 2048), (200, 200, 4, 128), (1003, 1003, 16, 2048), (1003, 1003, 8, 2048), (1024, 1024, 8, 1024), (2000, 2000, 16, 4096),
    (513, 3000, 16, 1024), (4096, 4096, 16, 2048), (4096, 4096, 16, 4096), (700, 700, 32, 768), (16384, 16384, 16, 2048),
    (8192, 8192, 8, 2048), (2048, 65536, 16, 2048)])
def test_lists_and_masks(q_len, k_len, stride, chunk, hq, hkv):
    from xattn_b200 import api, ops
    g = torch.Generator(device=DEV).manual_seed(q_len * 7 + stride)
    for dtype in (torch.bfloat16, torch.float16, torch.float32):
        q = torch.randn(1, hq, q_len, 128, device=DEV, generator=g).to(dtype)
        k, v = (torch.randn(1, hkv, k_len, 128, device=DEV, generator=g).to(dtype) for _ in range(2))
        per_head = torch.rand(hq, device=DEV, generator=g) * 0.3 + 0.7
        geo = ops.geometry(q_len, k_len, chunk, stride)
        for causal, thr, sink, recent in ((True, 0.9, False, False), (True, per_head, True, True), (False, 0.6, False, True), (True, 0.0, False, False)):
            sums = ops.estimate_block_sums(q, k, stride, 128, chunk, 1.0, causal)
            want, idx, cnt = ops.select_blocks(sums, geo["bpc"], geo["block_offset"], thr, causal, True, sink, recent, list_shape=(q_len, k_len))
            got_sums, got = api.xattn_estimate(q, k, 128, stride, threshold=thr, chunk_size=chunk, causal=causal, keep_sink=sink, keep_recent=recent)
            assert torch.equal(got, want), (dtype, causal)
            assert torch.equal(got_sums, sums.to(dtype)), (dtype, causal)
            out = ops.prefill(q, k, v, stride, 1.0, thr, 128, causal, chunk, sink, recent)
            ref = ops.block_sparse_attention(q, k, v, idx, cnt, causal)
            assert torch.equal(out, ref), (dtype, causal)
    ops.check_device_status()
