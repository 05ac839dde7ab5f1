"""The estimate at the lengths where its tiling can go wrong, against the oracle."""
import pytest
import torch

from oracle import xattn_oracle as orc

pytestmark = pytest.mark.gpu
DEV = "cuda"
# Block sums are sums of at most 32 x 32 probabilities in fp32 against the oracle's fp32 product of the same values: scores
# differ by about 1e-6 relative of a few tens, probabilities by 1e-4 at most.
RTOL, ATOL = 2e-4, 2e-5


@pytest.fixture(autouse=True)
def _status_clean():
    import xattn_b200
    yield
    xattn_b200.check_device_status()


def _check(hq, hkv, lq, lk, stride, chunk, causal, dtype, semantics="torch"):
    from xattn_b200 import ops
    g = torch.Generator().manual_seed(lq * 7 + lk + stride)
    # storage longer than the tensors, so that reads past a ragged end would meet other values
    qs, ks = torch.randn(1, hq, lq + 40, 128, generator=g), torch.randn(1, hkv, lk + 40, 128, generator=g)
    q, k = qs[:, :, :lq].to(dtype), ks[:, :, :lk].to(dtype)
    dq, dk = qs.to(dtype).to(DEV)[:, :, :lq], ks.to(dtype).to(DEV)[:, :, :lk]
    got = ops.estimate_block_sums(dq, dk, stride, 128, chunk, 1.0, causal, semantics=semantics).cpu()
    want = orc.estimate_block_sums(q.float(), k.float().repeat_interleave(hq // hkv, 1), 128, stride, 1.0, chunk, causal, semantics)
    assert torch.allclose(got, want, rtol=RTOL, atol=ATOL), float((got - want).abs().max())


@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("stride", [4, 8, 16, 32])
@pytest.mark.parametrize("L", [3, 31, 128, 129, 1003, 2041, 2048, 2049, 4100])   # below a stride; edges of blocks, tiles, chunks
def test_ragged_and_short_lengths(L, stride, causal):
    _check(2, 1, L, L, stride, 2048, causal, torch.bfloat16)


@pytest.mark.parametrize("lq,lk,chunk", [(100, 1500, 2048), (1999, 4095, 2048), (700, 700, 16384), (384, 640, 128), (1, 2000, 512)])
@pytest.mark.parametrize("semantics", ["torch", "triton"])
def test_query_shorter_than_the_keys(lq, lk, chunk, semantics):
    _check(4, 2, lq, lk, 16, chunk, True, torch.float16, semantics)


@pytest.mark.parametrize("L,stride,chunk,causal", [(300, 16, 2048, True), (2048, 16, 2048, True), (2500, 8, 2048, False), (1900, 8, 2048, True),
                                                   (4096, 8, 4096, True), (5000, 16, 4096, True)])
def test_split_fp32_terms(L, stride, chunk, causal):
    """fp32 inputs as three bf16 terms: through the single-CTA kernel with 128- and 256-column tiles and the CTA pairs."""
    _check(3, 3, L, L, stride, chunk, causal, torch.float32)


@pytest.mark.parametrize("lq,lk,stride,chunk", [(2304, 2304, 8, 256), (1152, 1664, 4, 128), (5120, 5120, 16, 2560), (768, 3840, 4, 768), (1280, 1280, 32, 640)])
def test_dense_rows_of_a_few_chunks(lq, lk, stride, chunk):
    """Un-padded causal keys whose chunks are a tile or less each: the epilogue writes whole rows, zeros included; chunks that
    are not a multiple of a tile leave tiles that hang over the row's end."""
    _check(2, 2, lq, lk, stride, chunk, True, torch.bfloat16)
