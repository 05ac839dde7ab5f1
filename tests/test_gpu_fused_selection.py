"""The selection inside the estimate's kernel against the selection as a kernel of its own on the same sums."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


# (tokens, stride, chunk): every way a row of sums is finished in the GEMM's epilogue -- clusters of four, which select there, and
# those that leave it to a kernel behind them: clusters of two, single CTAs with a few tiles, tiles of 256 columns, CTA pairs -- and sixteen
# warps per row tile behind it; ragged lengths, rows of padding, chunks of their own and all of the keys
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


def _compare(hq, hkv, q_len, k_len, stride, chunk, dtype, causal=True, thr=0.9, sink=False, recent=False, launches=None):
    """Mask and lists of the combined calls against the selection kernel on the same sums; `launches`: kernels of the mask's call."""
    from xattn_b200 import _lib, api, ops
    g = torch.Generator(device=DEV).manual_seed(q_len * 7 + stride)
    q = torch.randn(1, hq, q_len, 128, device=DEV, generator=g, dtype=torch.float32).to(dtype)
    k, v = (torch.randn(1, hkv, k_len, 128, device=DEV, generator=g).to(dtype) for _ in range(2))
    geo = ops.geometry(q_len, k_len, chunk, stride)
    sums = ops.estimate_block_sums(q, k, stride, 128, chunk, 1.0, causal)
    want, idx, cnt = ops.select_blocks(sums, geo["bpc"], geo["block_offset"], thr, causal, True, sink, recent, list_shape=(q_len, k_len))
    ref = ops.block_sparse_attention(q, k, v, idx, cnt, causal)
    count = _lib.load().xattn_b200_launch_count
    n0 = count()
    got_sums, got = api.xattn_estimate(q, k, 128, stride, threshold=thr, chunk_size=chunk, causal=causal, keep_sink=sink, keep_recent=recent)
    n1 = count()
    out = ops.prefill(q, k, v, stride, 1.0, thr, 128, causal, chunk, sink, recent)
    n2 = count()
    assert torch.equal(got, want)
    assert torch.equal(got_sums, sums.to(dtype))
    assert torch.equal(out, ref)
    ops.check_device_status()
    if launches is not None:
        assert (n1 - n0, n2 - n1) == launches


# Clusters of one CTA with more than four tiles per SM: each selects on a tile while the next one's products run.  Bands of the chunk
# (the prefill) at every stride, dense rows of 128 sums (the mask), short ragged keys, no causality.
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("hq,hkv,L,stride,chunk,causal", [
    (32, 8, 40960, 16, 2048, True), (80, 8, 16384, 16, 2048, True), (40, 8, 16384, 8, 1024, True),
    (24, 8, 16384, 4, 512, True), (152, 8, 16384, 32, 4096, True), (600, 200, 1003, 16, 2048, True), (600, 200, 1999, 16, 2048, False)])
def test_under_the_next_tiles(hq, hkv, L, stride, chunk, causal, dtype):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    tiles = hq * -(-(L // stride) // 128)
    if tiles <= 4 * sms:
        pytest.skip("needs more than four tiles per SM")
    fused = 1 if tiles // hq <= 64 else 2              # (long calls: the tile tables are a kernel of their own)
    kb = -(-L // chunk) * chunk // 128
    mask = fused + (1 if kb > 8 * stride else 0)       # (dense rows of more than eight tiles: the kernel of the block sums)
    extra = 0 if causal else 1                         # (the ordered list of units of a non-causal attention)
    _compare(hq, hkv, L, L, stride, chunk, dtype, causal, 0.93, launches=(mask, fused + 1 + extra))


# Few row tiles: their query blocks, or where another kernel selects their key blocks, are divided over CTAs, and row tiles of
# padding follow; of 1, 5, 8, 16, 17 and 32 query blocks in a tile.  The last: more than sixteen column tiles per row, whose sums are the same ones
# whether a selection follows (eight warps) or not (sixteen).
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("hq,hkv,q_len,k_len,stride,chunk,causal", [
    (2, 1, 2048, 30000, 32, 16384, True), (4, 4, 2047, 30000, 16, 16384, True), (3, 1, 1000, 20000, 8, 16384, False), (1, 1, 4200, 40000, 32, 8192, True),
    (2, 2, 640, 9000, 16, 1024, True), (1, 1, 100, 20000, 16, 4096, True), (2, 1, 2176, 12000, 32, 2048, False), (1, 1, 2048, 30000, 4, 2048, True),
    (2, 1, 2048, 65536, 16, 16384, True), (2, 1, 100, 62000, 8, 20480, True)])
def test_row_tiles_in_parts(hq, hkv, q_len, k_len, stride, chunk, causal, dtype):
    _compare(hq, hkv, q_len, k_len, stride, chunk, dtype, causal)


# The kernel of the block sums selects on its row tiles: sixteen warps up to two row tiles per SM (the first three), eight beyond.  Bands
# of 128, 256 and 512 (the prefill) and dense rows of as many (the mask), every stride, ragged lengths.
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("hq,hkv,L,stride,chunk,causal,few", [
    (4, 2, 16384, 8, 16384, True, True), (4, 2, 32768, 16, 32768, True, True), (2, 1, 65536, 16, 65536, True, True),
    (32, 8, 32768, 8, 16384, True, False), (32, 8, 40955, 16, 2048, True, False), (40, 8, 15400, 16, 4096, True, False),
    (40, 40, 16384, 4, 16384, True, False), (20, 4, 32768, 32, 32768, True, True), (20, 20, 32760, 16, 8192, True, False),
    (20, 5, 31000, 16, 32768, True, False), (10, 5, 62000, 16, 4096, True, False), (10, 2, 65536, 8, 65536, True, False),
    (40, 8, 15400, 16, 2048, False, False), (10, 10, 61000, 8, 2048, False, False)])
def test_row_tiles_selected_on_behind_the_gemm(hq, hkv, L, stride, chunk, causal, few, dtype):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    if (hq * -(-L // (128 * stride)) <= 2 * sms) != few:
        pytest.skip("meant for another number of SMs")
    gemm = 1 if -(-L // chunk) * chunk // stride <= 64 * 128 else 2     # (long calls: the tile tables are a kernel of their own)
    for sink, recent in ((False, False), (True, True)):
        extra = 0 if causal else 1                     # (the ordered list of units of a non-causal attention)
        _compare(hq, hkv, L, L, stride, chunk, dtype, causal, 0.93, sink, recent, launches=(gemm + 1, gemm + 2 + extra))


def test_row_tiles_selected_on_behind_the_fp32_gemm():
    """fp32 inputs take the same kernel of the block sums behind a GEMM of their own."""
    _compare(40, 8, 15400, 15400, 16, 4096, torch.float32)
