"""The attention and decode kernels at the sizes where their tiling can go wrong, against plain fp32 attention."""
import pytest
import torch

from oracle import xattn_oracle as orc

pytestmark = pytest.mark.gpu
DEV = "cuda"
# Probabilities and outputs are rounded to the 16-bit type, 2^-9 relative each for bf16 (2^-12 for fp16): an output, an
# average of values of at most about 5, is off by at most 2 * 2^-9 * 5 = 2e-2; on average by a tenth of that.
MAX_ABS, MEAN_ABS = 2e-2, 2e-3


@pytest.fixture(autouse=True)
def _status_clean():
    import xattn_b200
    yield
    xattn_b200.check_device_status()


def _close(got, want, scale=1.0):
    err = (got.float().cpu() - want).abs()
    assert torch.isfinite(got.float()).all()
    assert err.max() < MAX_ABS * scale and err.mean() < MEAN_ABS * scale, (float(err.max()), float(err.mean()))


def _qkv(seed, b, hq, hkv, lq, lk, dtype=torch.bfloat16):
    g = torch.Generator().manual_seed(seed)
    return [torch.randn(b, h, n, 128, generator=g).to(dtype) for h, n in ((hq, lq), (hkv, lk), (hkv, lk))]


@pytest.mark.parametrize("k_len", [1, 17, 63, 64, 65, 129, 1000, 4097])       # edges of a warp's 16 keys, of a stage, of a split
@pytest.mark.parametrize("dtype,batch,hq,hkv", [(torch.bfloat16, 1, 8, 2), (torch.float16, 2, 7, 1), (torch.bfloat16, 1, 3, 3),
                                                (torch.bfloat16, 1, 16, 1), (torch.bfloat16, 1, 17, 1)])
def test_decode_step(k_len, dtype, batch, hq, hkv):
    from xattn_b200 import ops
    q, k, v = _qkv(k_len + hq, batch, hq, hkv, 1, k_len, dtype)
    k[:, :, k_len // 2] *= 4.0                                               # a dominant key: the running maximum moves
    cache = [torch.zeros(batch, hkv, k_len + 37, 128, dtype=dtype, device=DEV) for _ in range(2)]
    for c, x in zip(cache, (k, v)):
        c[:, :, :k_len] = x.to(DEV)
    out = ops.decode_attention(q.to(DEV), cache[0][:, :, :k_len], cache[1][:, :, :k_len])     # a slice of a longer cache
    assert out.shape == q.shape and out.dtype == dtype
    rep = hq // hkv
    want = torch.nn.functional.scaled_dot_product_attention(q.float(), k.float().repeat_interleave(rep, 1),
                                                            v.float().repeat_interleave(rep, 1))
    _close(out, want)


@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("batch,hq,hkv,lq,lk", [(1, 7, 1, 640, 640), (1, 3, 3, 300, 300), (2, 4, 2, 129, 1000), (1, 1, 1, 5, 5),
                                                (1, 2, 2, 127, 4200), (1, 5, 1, 1, 257)])
def test_dense_call_without_lists(causal, batch, hq, hkv, lq, lk):
    """Odd groups, odd numbers of query blocks, a query offset that is no multiple of the block, lists of more than 32
    blocks: every form of a work unit (two heads, two query blocks, one tile)."""
    from xattn_b200 import ops
    q, k, v = _qkv(lq + lk, batch, hq, hkv, lq, lk)
    out = ops.block_sparse_attention(q.to(DEV), k.to(DEV), v.to(DEV), None, None, causal)
    rep = hq // hkv
    keep = torch.ones(lq, lk, dtype=torch.bool).tril(lk - lq) if causal else None
    want = torch.nn.functional.scaled_dot_product_attention(q.float(), k.float().repeat_interleave(rep, 1),
                                                            v.float().repeat_interleave(rep, 1), attn_mask=keep)
    _close(out, want)


@pytest.mark.parametrize("causal,ordered", [(True, False), (False, False), (False, True)])
@pytest.mark.parametrize("hq,hkv,L", [(6, 2, 128 * 81), (3, 3, 128 * 160 - 1), (7, 1, 128 * 61)])
def test_more_units_than_sms(causal, ordered, hq, hkv, L):
    """CTAs take over further units: lists of 0 to 40 blocks that differ between the two tiles of a unit, runs of rows that
    list nothing, one row that lists everything."""
    from xattn_b200 import ops
    q, k, v = _qkv(L + hq, 1, hq, hkv, L, L)
    nb = (L + 127) // 128
    g = torch.Generator().manual_seed(L)
    want_n = (torch.rand(1, hq, nb, 1, generator=g) ** 3 * 40).long()
    mask = torch.rand(1, hq, nb, nb, generator=g).argsort(-1).argsort(-1) < want_n
    mask[:, :, nb // 3:nb // 3 + 12] = False
    mask[0, hq - 1, nb - 2] = True
    if causal:
        mask &= torch.tril(torch.ones(nb, nb, dtype=torch.bool))
    idx, cnt = ops.mask_to_lists(mask.to(DEV), L, L, causal)
    out = torch.full((1, hq, L, 128), float("nan"), dtype=torch.bfloat16, device=DEV)
    ops.block_sparse_attention(q.to(DEV), k.to(DEV), v.to(DEV), idx, cnt, causal, out=out, use_workspace=ordered)
    assert torch.isfinite(out.float()).all()
    rows = sorted({0, 1, 2, nb // 3, nb // 3 + 11, nb // 2, nb - 3, nb - 2, nb - 1})
    rep = hq // hkv
    for r in rows:
        r0, r1 = r * 128, min(L, (r + 1) * 128)
        keep = mask[:, :, r].repeat_interleave(128, -1)[:, :, None, :L].expand(-1, -1, r1 - r0, -1)
        if causal:
            keep = keep & (torch.arange(L)[None, :] <= torch.arange(r0, r1)[:, None])
        s = torch.einsum("bhqd,bhkd->bhqk", q[:, :, r0:r1].float(), k.float().repeat_interleave(rep, 1)) / 128 ** 0.5
        p = torch.where(keep.any(-1, keepdim=True), s.masked_fill(~keep, float("-inf")), torch.zeros(()))
        p = torch.where(keep, torch.softmax(p, -1), torch.zeros(()))
        want = p @ v.float().repeat_interleave(rep, 1)
        _close(out[:, :, r0:r1], want)


@pytest.mark.parametrize("batch,hkv,k_len", [(1, 8, 300), (1, 8, 4096), (1, 8, 4097), (4, 8, 9000), (8, 8, 3001), (3, 16, 700), (6, 8, 5000)])
def test_decode_step_merges(batch, hkv, k_len):
    """Caches that one CTA, a cluster of two, four or eight, or more CTAs than a cluster share; fully checked in batch."""
    from xattn_b200 import ops
    q, k, v = _qkv(k_len + batch, batch, 2 * hkv, hkv, 1, k_len)
    k[:, :, -1] *= 3.0
    out = ops.decode_attention(q.to(DEV), k.to(DEV), v.to(DEV))
    want = torch.nn.functional.scaled_dot_product_attention(q.float(), k.float().repeat_interleave(2, 1),
                                                            v.float().repeat_interleave(2, 1))
    _close(out, want)


def test_decode_ring_under_load():
    """Stages go back to TMA a dozen times per CTA: repeated calls agree bit by bit."""
    from xattn_b200 import ops
    q, k, v = (x.to(DEV) for x in _qkv(1, 2, 16, 8, 1, 16384))
    first = ops.decode_attention(q, k, v)
    for _ in range(100):
        assert torch.equal(ops.decode_attention(q, k, v), first)


def test_calls_in_a_row_without_a_pause():
    """The kernels of a call start before the ones in front of them have ended, and the lists lie where the estimate's scratch
    has just been: calls of several shapes in a row give what each gives alone."""
    from xattn_b200 import api
    inputs = []
    for i, (L, dtype) in enumerate([(1500, torch.bfloat16), (3000, torch.float16), (700, torch.float32), (5000, torch.bfloat16)]):
        q, k, v = (x.to(DEV) for x in _qkv(i, 1, 4, 2, L, L, dtype))
        inputs.append((q, k, v, 8, 1, 0.6, 128, True, i != 1, 1, 1024 if i < 2 else 2048))
    want = []
    for x in inputs:
        want.append(api.Xattention_prefill(*x))
        torch.cuda.synchronize()
    for _ in range(100):
        got = [api.Xattention_prefill(*x) for x in inputs]
        for a, b in zip(got, want):
            assert torch.equal(a, b)


@pytest.mark.parametrize("blocks,items_per_sm,ordered", [(41, 4, True), (41, 3, False), (40, 4, False), (40, 16, True)])
def test_which_non_causal_calls_are_ordered(blocks, items_per_sm, ordered):
    """The units of a call with long lists and a few of them per SM are sorted first: one launch more, the same results."""
    from xattn_b200 import _lib, ops
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    heads = -(-items_per_sm * sms // blocks) if ordered or blocks == 40 else items_per_sm * sms // blocks
    L = blocks * 128 - 5
    g = torch.Generator(device=DEV).manual_seed(blocks)
    q, k, v = (torch.randn(1, heads, L, 128, device=DEV, generator=g).bfloat16() for _ in range(3))
    mask = torch.rand(1, heads, blocks, blocks, device=DEV, generator=g) < 0.1
    mask[:, :, -2:] = True
    idx, cnt = ops.mask_to_lists(mask, L, L, False)
    count = _lib.load().xattn_b200_launch_count
    n0 = count()
    got = ops.block_sparse_attention(q, k, v, idx, cnt, False)
    n1 = count()
    assert n1 - n0 == (2 if ordered else 1)
    assert torch.equal(got, ops.block_sparse_attention(q, k, v, idx, cnt, False, use_workspace=False))


@pytest.mark.parametrize("dtype,out_dtype", [(torch.bfloat16, torch.bfloat16), (torch.float16, torch.float16), (torch.float32, torch.float32)])
@pytest.mark.parametrize("hq,hkv,lq,lk", [(2, 1, 70 * 128, 70 * 128), (7, 7, 300, 8400), (4, 2, 1, 9000), (1, 1, 127, 128 * 70 + 1), (74, 37, 256, 8193)])
def test_tiles_whose_streams_share_a_list(hq, hkv, lq, lk, dtype, out_dtype):
    """Up to a tile per SM: of none, one, an odd and an even number of blocks, of more than a window of a list; rows whose blocks are
    hidden from one stream altogether."""
    from xattn_b200 import ops
    q, k, v = _qkv(lq + hq, 1, hq, hkv, lq, lk, dtype)
    qb, kb = (lq + 127) // 128, (lk + 127) // 128
    g = torch.Generator().manual_seed(lk)
    want_n = torch.randint(0, 6, (1, hq, qb, 1), generator=g)
    want_n[:, :, ::3] = kb
    mask = torch.rand(1, hq, qb, kb, generator=g).argsort(-1).argsort(-1) < want_n
    rep = hq // hkv
    qf, kf, vf = (x.to(torch.bfloat16).float() if dtype == torch.float32 else x.float() for x in (q, k, v))
    kf, vf = kf.repeat_interleave(rep, 1), vf.repeat_interleave(rep, 1)
    visible = torch.ones(lq, lk, dtype=torch.bool).tril(lk - lq)
    idx, cnt = ops.mask_to_lists(mask.to(DEV), lq, lk, True)
    for lists in (True, False):
        out = ops.block_sparse_attention(q.to(DEV), k.to(DEV), v.to(DEV), idx if lists else None, cnt if lists else None, True)
        assert out.dtype == out_dtype
        for h in range(0, hq, max(1, hq // 4)):
            keep = visible & mask[0, h].repeat_interleave(128, 0)[:lq].repeat_interleave(128, 1)[:, :lk] if lists else visible
            s = (qf[0, h] @ kf[0, h].T * 128 ** -0.5).masked_fill(~keep, float("-inf"))
            want = torch.where(keep.any(1, keepdim=True), torch.softmax(s, -1).nan_to_num(0.0) @ vf[0, h], torch.zeros(()))
            _close(out[0, h], want)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("batch,hq,hkv,ragged", [(1, 28, 4, 100), (1, 2, 1, 3), (2, 12, 4, 127), (1, 7, 7, 0)])
def test_second_tiles_of_a_cta(batch, hq, hkv, ragged, dtype):
    """Dense prompts of one to two tiles per SM: a CTA takes a second tile, shorter than its first or of a single block, behind which a
    stream has none."""
    from xattn_b200 import ops
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    nb = 19 * sms // (10 * batch * hq)
    L = nb * 128 - ragged
    assert sms < nb * batch * hq <= 2 * sms
    q, k, v = (x.to(DEV) for x in _qkv(L, batch, hq, hkv, L, L, dtype))
    out = ops.block_sparse_attention(q, k, v, None, None, True)
    assert out.dtype == dtype
    qf, kf, vf = (x.to(torch.bfloat16).float() if dtype == torch.float32 else x.float() for x in (q, k, v))
    visible = torch.ones(L, L, dtype=torch.bool, device=DEV).tril()
    for b, h in {(0, 0), (batch - 1, hq - 1), (0, hq // 2)}:
        s = (qf[b, h] @ kf[b, h * hkv // hq].T * 128 ** -0.5).masked_fill(~visible, float("-inf"))
        _close(out[b, h], (torch.softmax(s, -1) @ vf[b, h * hkv // hq]).cpu())


def test_lists_of_a_batch_shared_by_the_streams():
    """Up to a tile per SM and more than 64 key blocks: a sequence alone has the bits that it has in a batch of two."""
    from xattn_b200 import ops
    q, k, v = (x.to(DEV) for x in _qkv(4, 2, 4, 2, 300, 8400))
    mask = torch.rand(2, 4, 3, 66, generator=torch.Generator().manual_seed(1)) < 0.3
    idx, cnt = ops.mask_to_lists(mask.to(DEV), 300, 8400, True)
    both = ops.block_sparse_attention(q, k, v, idx, cnt, True)
    for b in range(2):
        s = slice(b, b + 1)
        assert torch.equal(ops.block_sparse_attention(q[s], k[s], v[s], idx[s], cnt[s], True), both[s])
    want = orc.block_sparse_attention_oracle(q.cpu(), k.cpu(), v.cpu(), mask, True)
    _close(both, want)


def test_dense_calls_of_more_than_a_tile_per_sm_against_long_keys():
    """Their tiles go in twos, as those of larger calls do: a sequence alone has the bits that it has in a batch."""
    from xattn_b200 import ops
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    hq = 4 * (sms * 3 // 2 // 32)                        # of eight query blocks each: one and a half tiles per SM
    q, k, v = (x.to(DEV) for x in _qkv(1, 2, hq, hq // 4, 1024, 4096))
    assert sms < 8 * hq <= 2 * sms and 4 * hq <= sms
    both = ops.block_sparse_attention(q, k, v, None, None, True)
    assert torch.equal(ops.block_sparse_attention(q[:1], k[:1], v[:1], None, None, True), both[:1])


@pytest.mark.parametrize("count", [2 ** 30, -5, 4])
def test_counts_beyond_a_row_of_the_lists(count):
    """A count that no list can have is cut to the row of the lists (three blocks here), or to none."""
    from xattn_b200 import ops
    q, k, v = (x.to(DEV) for x in _qkv(7, 1, 4, 2, 300, 384))
    idx, cnt = ops.mask_to_lists(torch.ones(1, 4, 3, 3, dtype=torch.bool, device=DEV), 300, 384, False)
    want = ops.block_sparse_attention(q, k, v, idx, cnt, False)
    for workspace in (False, True):
        got = ops.block_sparse_attention(q, k, v, idx, torch.full_like(cnt, count), False, use_workspace=workspace)
        assert torch.equal(got, want if count > 0 else torch.zeros_like(want))


@pytest.mark.parametrize("hq,hkv", [(7, 1), (32, 8), (6, 3)])
def test_two_units_at_a_time(hq, hkv):
    """Causal calls of many units with short lists take them in twos and keep K/V tiles in their slots from one to the next: against the same call
    head by head, whose units are too few for that.  Lists as the selection leaves them and worse: the same in all heads, the same in
    some, of 0 to 12 blocks, with and without the diagonal; odd groups, and (7 heads) an odd number of units."""
    from xattn_b200 import _lib, ops
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    rows = -(-24 * sms // hq) | 1                     # pairs of query blocks
    L = 256 * rows - 131                              # ragged; an even number of query blocks
    g = torch.Generator(device=DEV).manual_seed(hq)
    q = torch.randn(1, hq, L, 128, device=DEV, generator=g).bfloat16()
    k, v = (torch.randn(1, hkv, L, 128, device=DEV, generator=g).bfloat16() for _ in range(2))
    n = (L + 127) // 128
    cnt = torch.randint(0, 4, (1, 1, n), device=DEV, generator=g)
    cnt = torch.where(torch.rand(1, 1, n, device=DEV, generator=g) < 0.1, torch.randint(5, 13, (1, 1, n), device=DEV, generator=g), cnt).expand(1, hq, n)
    r = torch.arange(n, device=DEV)
    # per head and row: block 0, the diagonal, then blocks in between, sorted, without repeats
    mid = torch.rand(1, 1, n, 12, device=DEV, generator=g).expand(1, hq, n, 12).clone()
    own = torch.rand(1, hq, n, 1, device=DEV, generator=g) < 0.3            # lists of their own
    mid = torch.where(own, torch.rand(1, hq, n, 12, device=DEV, generator=g), mid)
    cand = (mid * (r + 1)[:, None]).long()
    cand[..., 0] = r
    cand[..., 1] = 0
    cand = torch.where(torch.arange(12, device=DEV) < cnt[..., None], cand, n)
    cand = cand.sort(-1).values
    keep = (cand < n) & torch.cat([torch.ones_like(cand[..., :1], dtype=torch.bool), cand[..., 1:] != cand[..., :-1]], -1)
    order = (~keep).long().sort(dim=-1, stable=True).indices
    idx = torch.zeros(1, hq, n, n, dtype=torch.int32, device=DEV)
    idx[..., :12] = cand.gather(-1, order).clamp(max=n - 1)
    cnt = keep.sum(-1).to(torch.int32)
    out = torch.empty(1, L, hq, 128, dtype=q.dtype, device=DEV).transpose(1, 2)
    lib = _lib.load()
    _lib.check(lib.xattn_b200_block_sparse_attn_bounded(
        q.data_ptr(), k.data_ptr(), v.data_ptr(), _lib.BF16, 1, hq, hkv, L, L, 128, *q.stride()[:3], *k.stride()[:3], *v.stride()[:3],
        idx.data_ptr(), cnt.data_ptr(), 1, 128 ** -0.5, out.data_ptr(), *out.stride()[:3], None, 0, 13, None,
        torch.cuda.current_stream().cuda_stream), "block_sparse_attn_bounded")
    assert torch.equal(out, ops.block_sparse_attention(q, k, v, idx, cnt, True))
    for h in range(hq):
        kv = h // (hq // hkv)
        one = ops.block_sparse_attention(q[:, h:h + 1], k[:, kv:kv + 1], v[:, kv:kv + 1], idx[:, h:h + 1], cnt[:, h:h + 1], True)
        assert torch.equal(out[:, h], one[:, 0]), h
    ops.check_device_status()


# (batch, query heads, kv heads, keys): clusters of eight and of sixteen and the second kernel, and the lines between them; deep
# rings and not; ragged last stages, CTAs of unequal numbers of stages; 1 to 16 rows per kv head; strided caches
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("B,hq,hkv,n", [
    (1, 32, 8, 4096), (1, 32, 8, 4097), (1, 32, 8, 4160), (1, 32, 8, 36864), (1, 32, 8, 36865), (1, 28, 4, 5000), (1, 28, 4, 65536),
    (1, 28, 4, 65537), (1, 16, 1, 4111), (7, 1, 1, 6000), (2, 14, 7, 4500), (3, 5, 5, 4500), (2, 32, 8, 4500), (1, 12, 2, 20001), (3, 28, 4, 2500)])
def test_decode_splits(B, hq, hkv, n, dtype):
    from xattn_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(n + hq)
    q = torch.randn(B, 1, hq, 128, device=DEV, generator=g).to(dtype).transpose(1, 2)
    k = torch.randn(B, n, hkv, 128, device=DEV, generator=g).to(dtype).transpose(1, 2)
    v = torch.randn(B, hkv, n, 128, device=DEV, generator=g).to(dtype)
    out = ops.decode_attention(q, k, v)
    rep = hq // hkv
    for b in range(B):
        for h in range(hkv):
            s = q[b, h * rep:(h + 1) * rep, 0].double() @ k[b, h].double().T * 128 ** -0.5
            want = s.softmax(-1) @ v[b, h].double()
            # probabilities and results rounded to 8 or 11 bits: each at most half a unit in the last place, both together less than one
            tol = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
            err = (out[b, h * rep:(h + 1) * rep, 0].double() - want).norm() / want.norm()
            assert err < tol, (b, h, float(err))
    ops.check_device_status()
