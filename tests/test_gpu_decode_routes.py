"""The decode step where its cache is split in another way: the same results on either side of the line, and for any values."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.fixture(autouse=True)
def _status_clean():
    import xattn_b200
    yield
    xattn_b200.check_device_status()


def _step(seed, batch, hq, hkv, n, dtype):
    g = torch.Generator(device=DEV).manual_seed(seed)
    return [torch.randn(batch, h, m, 128, device=DEV, generator=g).to(dtype) for h, m in ((hq, 1), (hkv, n), (hkv, n))]


# clusters of four and of eight; a CTA with an SM to itself (few heads), and two CTAs per SM (the same sequence in a batch)
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("hq,hkv,n", [(32, 8, 500), (32, 8, 777), (32, 8, 2011), (32, 8, 4096), (28, 4, 1999), (28, 4, 4000), (16, 1, 3000)])
def test_a_sequence_alone_and_in_a_batch(hq, hkv, n, dtype):
    """Up to eight CTAs share the cache of a head in either case, each the same part of it: the same bits."""
    from xattn_b200 import ops
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    batch = sms // 8 // hkv                           # (more than three quarters of the SMs, eight CTAs per head)
    q, k, v = _step(n, batch, hq, hkv, n, dtype)
    together = ops.decode_attention(q, k, v)
    for b in (0, batch - 1):
        assert torch.equal(ops.decode_attention(q[b:b + 1], k[b:b + 1], v[b:b + 1])[0], together[b])
