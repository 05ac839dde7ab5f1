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


# every way to split a cache: one CTA, clusters of four, eight and sixteen, more CTAs and a second kernel
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("batch,hq,hkv,n", [(1, 8, 2, 100), (1, 32, 8, 500), (1, 32, 8, 2011), (4, 32, 8, 2011), (1, 32, 8, 5000), (1, 28, 4, 5000),
                                            (1, 8, 8, 4097), (3, 28, 4, 9000), (4, 32, 8, 9000), (1, 32, 8, 40000)])
def test_infinite_values(batch, hq, hkv, n, dtype):
    """A value that is infinite makes its column of the head infinite, whatever its key's probability rounds to; the other columns
    are what they are without it.  A NaN stays one."""
    from xattn_b200 import ops
    q, k, v = _step(n + hq, batch, hq, hkv, n, dtype)
    q = q * 0.1                                       # (no probability vanishes)
    want = ops.decode_attention(q, k, v)
    bad = v.clone()
    keys = torch.linspace(0, n - 1, 12, device=DEV).long().tolist()
    for i, key in enumerate(keys):
        bad[:, :, key, i] = float("inf")
        bad[:, :, key, 32 + i] = float("-inf")
    bad[:, :, keys[3], 64] = float("nan")
    got = ops.decode_attention(q, k, bad)
    assert (got[..., :12] == float("inf")).all()
    assert (got[..., 32:44] == float("-inf")).all()
    assert got[..., 64].isnan().all()
    rest = [c for c in range(128) if c not in (*range(12), *range(32, 44), 64)]
    # (the probabilities of such a call may be multiplied in one 16-bit term instead of two: at most half a unit in the last place
    # of the values' type per probability and per result, on averages of values of at most 6)
    tol = 6 * 2.0 ** (-8 if dtype == torch.bfloat16 else -11)
    assert (got[..., rest].float() - want[..., rest].float()).abs().max() <= tol


@pytest.mark.parametrize("n", [4097, 4500, 30000])
def test_two_ctas_per_sm_make_sixteen_per_head(n):
    """Heads for which two CTAs per SM come to sixteen each, but whose clusters of sixteen do not fit on the chip together: they take
    the second kernel, with its scratch, as one head fewer and one more do."""
    from xattn_b200 import _lib, ops
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    heads = 2 * sms // 16
    assert 2 * sms // heads == 16
    lib = _lib.load()
    q, k, v = _step(n, heads, 4, 1, n, torch.bfloat16)
    out = ops.decode_attention(q, k, v)
    for b in (0, heads // 2, heads - 1):
        s = q[b, :, 0].double() @ k[b, 0].double().T * 128 ** -0.5
        want = s.softmax(-1) @ v[b, 0].double()
        # probabilities and results rounded to 8 bits: each at most half a unit in the last place, both together less than one
        assert (out[b, :, 0].double() - want).norm() / want.norm() < 2.0 ** -8
    for h in (heads - 1, heads, heads + 1):
        assert lib.xattn_b200_decode_workspace_bytes(h, 4, 1, n) > 0, h
