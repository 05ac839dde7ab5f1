"""The threshold selection over the row lengths and score shapes where it changes its way of working, against the oracle."""
import pytest
import torch

from oracle import xattn_oracle as orc

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _scores(kind, H, R, N, g):
    x = torch.rand(1, H, R, N, generator=g)
    if kind == "peaked":
        return x ** 12
    if kind == "flat":
        return x + 0.5
    if kind == "ties":                               # few distinct values, many zeros
        return (x * 4).floor().clamp(0, 3) / 4
    return torch.where(x < 0.7, torch.zeros(()), x)  # sparse


@pytest.mark.parametrize("kind", ["peaked", "flat", "ties", "sparse"])
@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("N,bpc", [(4, 4), (33, 11), (128, 32), (130, 13), (256, 64), (260, 20), (512, 128), (516, 43), (1024, 256), (1023, 31),
                                   (1040, 104)])
def test_against_the_oracle(N, bpc, causal, kind):
    """Row lengths on both sides of every register-count and of the step to the shared-memory kernel; the first chunk (one
    forced block, whose decisions lag a rank behind) and later ones (two)."""
    from xattn_b200 import ops
    g = torch.Generator().manual_seed(N * 31 + bpc)
    R = N // bpc * bpc if causal else bpc
    R = min(R, 3 * bpc)
    for off in {0, N - R}:
        x = _scores(kind, 2, R, N, g)
        if causal:
            x = x * (torch.arange(N)[None, :] <= off + torch.arange(R)[:, None]).float()
        for thr in (0.0, 0.35, 0.9, 0.999):
            got, idx, cnt = ops.select_blocks(x.to(DEV), bpc, off, thr, causal, False, list_shape=(R * 128, N * 128))
            parts, exs = [], []
            for c in range(R // bpc):
                xc = x[:, :, c * bpc:(c + 1) * bpc]
                parts.append(orc.select_blocks_chunk(xc, off + c * bpc, thr, causal))
                exs.append(orc.margin_exempt_chunk(xc, off + c * bpc, thr, causal))
            want, ex = torch.cat(parts, -2), torch.cat(exs, -2)
            bad = (got.cpu() != want) & ~ex
            assert not bad.any(), (off, thr, bad.nonzero()[:5].tolist())
            # equal scores in column order: the number of blocks is the oracle's even where which of them is exempt
            if kind == "ties":
                assert torch.equal(got.cpu().sum(-1), want.sum(-1)) or ex.any()
            mask = got.cpu()
            if causal and off == N - R:              # the lists drop blocks the row's last token cannot see
                mask = mask & (torch.arange(N)[None, :] <= off + torch.arange(R)[:, None])
                for h in range(2):
                    for r in range(R):
                        assert idx[0, h, r, :cnt[0, h, r]].tolist() == mask[0, h, r].nonzero().flatten().tolist()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("L,chunk", [(100, 128), (1003, 384), (8192, 8192), (65536 + 640, 2048 + 128), (131200, 128)])   # 1 to 1025 key blocks
def test_returned_sums_are_the_selections_own_rounded(L, chunk, dtype):
    """The sums in the inputs' type, which the selection kernel writes for rows of up to 1024 blocks, bit by bit."""
    from xattn_b200 import api, ops
    g = torch.Generator(device=DEV).manual_seed(L)
    q, k = (torch.randn(1, h, L, 128, device=DEV, generator=g).to(dtype) for h in (2, 1))
    sums, mask = api.xattn_estimate(q, k, 128, 16, threshold=0.8, chunk_size=chunk, causal=True)
    want = ops.estimate_block_sums(q, k, 16, 128, chunk, 1.0, True)
    assert sums.dtype == dtype and mask.shape == sums.shape
    assert torch.equal(sums, want.to(dtype))
