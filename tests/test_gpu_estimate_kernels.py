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


@pytest.mark.parametrize("hq,hkv,lq,lk,stride,chunk", [(1, 1, 2600, 4096, 8, 2048), (28, 4, 5596, 8192, 16, 4096), (3, 1, 2100, 6144, 8, 2048),
                                                       (7, 1, 413, 16384, 8, 8192)])
def test_pair_of_a_row_tile_and_one_that_sees_nothing(hq, hkv, lq, lk, stride, chunk):
    """Un-padded keys, chunks of 256 columns, an odd group: a CTA pair whose second row tile lies past the queries computes its
    first one's column tile only, whose epilogue writes whole rows of the output."""
    _check(hq, hkv, lq, lk, stride, chunk, True, torch.bfloat16)


@pytest.mark.parametrize("hkv", [3, 1])
@pytest.mark.parametrize("L,stride,chunk,causal", [(300, 16, 2048, True), (2048, 16, 2048, True), (2500, 8, 2048, False), (1900, 8, 2048, True),
                                                   (4096, 8, 4096, True), (5000, 16, 4096, True), (9001, 8, 16384, True), (8192, 4, 8192, True)])
def test_split_fp32_terms(L, stride, chunk, causal, hkv):
    """fp32 inputs as three bf16 terms: split as the tiles are loaded (128- and 256-column tiles, one per row and several) and,
    for the longest, before."""
    _check(3, hkv, L, L, stride, chunk, causal, torch.float32)


@pytest.mark.parametrize("D,dtype", [(32, torch.float32), (96, torch.float32), (192, torch.float32), (64, torch.bfloat16), (192, torch.float16)])
@pytest.mark.parametrize("lq,lk,stride,chunk,causal", [(300, 300, 16, 2048, True), (1900, 2500, 8, 2048, True), (3000, 3000, 4, 1024, False),
                                                       (8192, 8192, 8, 4096, True)])
def test_other_head_dims(lq, lk, stride, chunk, causal, D, dtype):
    """16-bit rows of any multiple of 64, fp32 rows of any multiple of 32: an odd number of 32-column steps per token."""
    from xattn_b200 import ops
    g = torch.Generator().manual_seed(D + lq)
    q, k = torch.randn(1, 2, lq, D, generator=g).to(dtype), torch.randn(1, 1, lk, D, generator=g).to(dtype)
    got = ops.estimate_block_sums(q.to(DEV), k.to(DEV), stride, 128, chunk, 1.0, causal).cpu()
    want = orc.estimate_block_sums(q.float(), k.float().repeat_interleave(2, 1), 128, stride, 1.0, chunk, causal, "torch")
    assert torch.allclose(got, want, rtol=RTOL, atol=ATOL), float((got - want).abs().max())
    if dtype == torch.float32:
        with pytest.raises(Exception, match="argument"):
            ops.estimate_block_sums(q.to(DEV)[..., :24], k.to(DEV)[..., :24], stride, 128, chunk, 1.0, causal)


@pytest.mark.parametrize("L,chunk", [(900, 2048), (8192, 8192)])          # split in the GEMM, split before
def test_fp32_operands_in_any_memory(L, chunk):
    """fp32 tensors off a 16-byte boundary, of odd row strides, expanded or transposed: the results of contiguous copies, bit by
    bit."""
    from xattn_b200 import api, ops
    g = torch.Generator(device=DEV).manual_seed(L)
    flat = torch.randn(4 * L * 131 + 1, device=DEV, generator=g)
    forms = [flat[1:1 + 4 * L * 128].view(1, 4, L, 128), flat[:4 * L * 131].view(1, 4, L, 131)[..., :128],
             flat[:L * 128].view(1, 1, L, 128).expand(1, 4, L, 128), flat[:128].view(1, 1, 1, 128).expand(1, 4, L, 128),
             flat[:4 * L * 128].view(1, 4, 128, L).transpose(2, 3)]
    k = torch.randn(1, 4, L, 128, device=DEV, generator=g)
    for x in forms:
        for a, b in ((x, k), (k, x)):
            got = ops.estimate_block_sums(a, b, 16, 128, chunk)
            assert torch.equal(got, ops.estimate_block_sums(a.clone(memory_format=torch.contiguous_format),
                                                            b.clone(memory_format=torch.contiguous_format), 16, 128, chunk))
        out = api.Xattention_prefill(k, x, x, 16, chunk_size=chunk)
        c = x.clone(memory_format=torch.contiguous_format)
        assert torch.equal(out, api.Xattention_prefill(k, c, c, 16, chunk_size=chunk))


def test_ring_of_fp32_units_under_load():
    """Units go from the converters back to TMA thousands of times per call: repeated calls agree bit by bit."""
    from xattn_b200 import ops
    q, k = (torch.randn(1, 16, 4096, 128, device=DEV, generator=torch.Generator(device=DEV).manual_seed(s)) for s in (1, 2))
    first = ops.estimate_block_sums(q, k, 16, 128, 2048)
    for _ in range(100):
        assert torch.equal(ops.estimate_block_sums(q, k, 16, 128, 2048), first)


@pytest.mark.parametrize("lq,lk", [(862, 1024), (1024, 1030), (12, 12)])
def test_ragged_operands_of_other_head_dims_in_any_memory(lq, lk):
    """16-bit rows of 64 or 192: off a 16-byte boundary, or with expanded heads."""
    from xattn_b200 import ops
    for D in (64, 192):
        g = torch.Generator(device=DEV).manual_seed(D)
        flat = torch.randn(2 * 1030 * D + 1, device=DEV, generator=g).bfloat16()
        for q, k in ((flat[1:1 + 2 * lq * D].view(1, 2, lq, D), flat[:lk * D].view(1, 1, lk, D).expand(1, 2, lk, D)),
                     (flat[:lq * D].view(1, 1, lq, D).expand(1, 2, lq, D), flat[1:1 + lk * D].view(1, 1, lk, D))):
            want = ops.estimate_block_sums(q.clone(memory_format=torch.contiguous_format), k.clone(memory_format=torch.contiguous_format), 16, 128, 1024)
            assert torch.equal(ops.estimate_block_sums(q, k, 16, 128, 1024), want)


@pytest.mark.parametrize("lq,lk,stride,chunk,causal,semantics", [
    (1003, 1003, 16, 2048, True, 0), (4096, 4096, 16, 2048, True, 2), (3000, 3000, 8, 4096, True, 1), (2000, 2500, 8, 2048, False, 0),
    (2048, 6144, 16, 2048, True, 2), (3, 5, 16, 2048, True, 0)])       # the last but one: keys that no tile reads
def test_bf16_roundings_of_fp32_operands(lq, lk, stride, chunk, causal, semantics):
    """The roundings written along with the estimate are those of every token, bit by bit."""
    from xattn_b200 import _lib, ops
    lib = _lib.load()
    g = torch.Generator(device="cuda").manual_seed(5)
    q, k = (torch.randn(2, h, n, 128, device="cuda", generator=g) for h, n in ((4, lq), (2, lk)))
    q16, k16 = (torch.full(x.shape, float("nan"), device="cuda", dtype=torch.bfloat16) for x in (q, k))
    gm = ops.geometry(lq, lk, chunk, stride)
    sums = torch.empty(2, 4, gm["qb"], gm["bpc"] if semantics == 2 else gm["kb"], device="cuda")
    ws = torch.empty(lib.xattn_b200_estimate_workspace_bytes(2, 4, lq, lk, stride, 128, chunk), dtype=torch.uint8, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    _lib.check(lib.xattn_b200_estimate_f32(q.data_ptr(), k.data_ptr(), 2, 4, 2, lq, lk, 128, *q.stride()[:3], *k.stride()[:3], stride, 128,
                                           chunk, 0.01, int(causal), semantics, sums.data_ptr(), ws.data_ptr(), ws.numel(), q16.data_ptr(),
                                           k16.data_ptr(), status.data_ptr(), torch.cuda.current_stream().cuda_stream), "estimate_f32")
    assert int(status) == 0 and bool(torch.isfinite(sums).all())
    assert torch.equal(q16, q.to(torch.bfloat16)) and torch.equal(k16, k.to(torch.bfloat16))


@pytest.mark.parametrize("D", [5, 64, 128])
def test_rows_of_six_terms(D):
    """The widened rows of either side, bit by bit, and (head dimensions that the estimate takes) the product over them."""
    from xattn_b200 import _lib, ops
    lib = _lib.load()
    B, H, L, padded, stream = 2, 3, 133, 136, torch.cuda.current_stream().cuda_stream
    g = torch.Generator().manual_seed(D)
    x = [torch.randn(B, H, L, D + 3, generator=g)[..., :D] for _ in range(2)]
    wide = []
    for role, order in ((0, (0, 0, 1, 0, 2, 1)), (1, (0, 1, 0, 2, 0, 1))):
        d = x[role].to(DEV)
        out = torch.full((B, H, padded, 6 * D), float("nan"), dtype=torch.bfloat16, device=DEV)
        _lib.check(lib.xattn_b200_split_f32(d.data_ptr(), B, H, padded, L, D, *d.stride()[:3], role, out.data_ptr(), stream), "split_f32")
        hi = x[role].bfloat16()
        mid = (x[role] - hi.float()).bfloat16()
        terms = (hi, mid, (x[role] - hi.float() - mid.float()).bfloat16())
        assert torch.equal(out[:, :, :L].cpu(), torch.cat([terms[t] for t in order], -1)) and not out[:, :, L:].any()
        wide.append(out)
    assert lib.xattn_b200_split_f32(d.data_ptr(), B, H, padded, L, D, *d.stride()[:3], 3, out.data_ptr(), stream) != 0
    if D % 64 == 0:
        got = ops.estimate_block_sums(wide[0], wide[1], 8, 128, 256, norm=(6 * D) ** -0.5 * D ** 0.5).cpu()
        pad = [torch.nn.functional.pad(t, (0, 0, 0, padded - L)) for t in x]
        assert torch.allclose(got, orc.estimate_block_sums(pad[0], pad[1], 128, 8, 1.0, 256, True, "torch"), rtol=RTOL, atol=ATOL)


@pytest.mark.parametrize("lq,lk,stride,chunk", [(2304, 2304, 8, 256), (1152, 1664, 4, 128), (5120, 5120, 16, 2560), (768, 3840, 4, 768), (1280, 1280, 32, 640)])
def test_dense_rows_of_a_few_chunks(lq, lk, stride, chunk):
    """Un-padded causal keys whose chunks are a tile or less each: the epilogue writes whole rows, zeros included; chunks that
    are not a multiple of a tile leave tiles that hang over the row's end."""
    _check(2, 2, lq, lk, stride, chunk, True, torch.bfloat16)


@pytest.mark.parametrize("stride,hkv,chunk,causal,semantics", [(4, 20, 16384, True, "torch"), (8, 8, 16384, True, "triton"),
                                                               (16, 20, 8192, True, "torch"), (32, 8, 16384, False, "torch")])
def test_many_query_blocks(stride, hkv, chunk, causal, semantics):
    """Calls of many row tiles, several column tiles per row: the first and the last head."""
    from xattn_b200 import ops
    hq, L = 40, 15400                                    # 40 * 128 (padded) query blocks; several column tiles per row
    g = torch.Generator().manual_seed(stride)
    k = torch.randn(1, hkv, L, 128, generator=g).bfloat16()
    q = torch.randn(1, hq, L, 128, generator=g).bfloat16()
    got = ops.estimate_block_sums(q.to(DEV), k.to(DEV), stride, 128, chunk, 1.0, causal, semantics=semantics).cpu()
    for h in (0, hq - 1):
        want = orc.estimate_block_sums(q[:, h:h + 1].float(), k[:, h * hkv // hq:h * hkv // hq + 1].float(), 128, stride, 1.0, chunk, causal,
                                       semantics)
        assert torch.allclose(got[:, h:h + 1], want, rtol=RTOL, atol=ATOL), float((got[:, h:h + 1] - want).abs().max())


@pytest.mark.parametrize("lq,lk,stride,chunk", [(1, 70000, 8, 16384), (300, 66001, 16, 2048), (2500, 40000, 4, 2048), (129, 70001, 32, 4096)])
@pytest.mark.parametrize("causal", [True, False])
def test_key_blocks_over_several_ctas(lq, lk, stride, chunk, causal):
    """Few row tiles against many key blocks: a row tile's are divided over CTAs, the last part being a short one."""
    _check(2, 1, lq, lk, stride, chunk, causal, torch.bfloat16)


@pytest.mark.parametrize("lq,lk,stride,chunk", [(8192, 8192, 16, 8192), (1024, 8192, 8, 2048), (3, 40000, 16, 16384)])
def test_sums_off_a_16_byte_boundary(lq, lk, stride, chunk):
    """Sums stored as vectors where their memory allows it: the same ones, and nothing beside them, where it does not."""
    from xattn_b200 import _lib, ops
    lib = _lib.load()
    g = torch.Generator(device=DEV).manual_seed(lq)
    q, k = torch.randn(1, 4, lq, 128, device=DEV, generator=g).bfloat16(), torch.randn(1, 2, lk, 128, device=DEV, generator=g).bfloat16()
    want = ops.estimate_block_sums(q, k, stride, 128, chunk)
    memory = torch.full((want.numel() + 8,), float("nan"), device=DEV)
    sums = memory[1:1 + want.numel()]
    ws = torch.empty(lib.xattn_b200_estimate_workspace_bytes(1, 4, lq, lk, stride, 128, chunk), dtype=torch.uint8, device=DEV)
    _lib.check(lib.xattn_b200_estimate(q.data_ptr(), k.data_ptr(), _lib.BF16, 1, 4, 2, lq, lk, 128, *q.stride()[:3], *k.stride()[:3], stride, 128,
                                       chunk, 128 ** -0.5 / stride, 1, 0, sums.data_ptr(), ws.data_ptr(), ws.numel(), None,
                                       torch.cuda.current_stream().cuda_stream), "estimate")
    assert torch.equal(sums.view(want.shape), want) and bool(memory[:1].isnan().all()) and bool(memory[1 + want.numel():].isnan().all())


@pytest.mark.parametrize("stride,column,chunk,dtype", [(16, 256, 8192, torch.bfloat16), (16, 512, 16384, torch.bfloat16), (8, 768, 8192, torch.float32),
                                                       (32, 256, 16384, torch.float16), (4, 512, 4096, torch.bfloat16)])
def test_a_column_tile_that_shows_a_row_nothing_but_nan(stride, column, chunk, dtype):
    """The last row sees one column of its last tile, and its scores there are NaN: that key block's sum is NaN, and the others are
    those of the row without it."""
    from xattn_b200 import ops
    L = (column + 1) * stride
    g = torch.Generator().manual_seed(stride)
    q, k = (torch.randn(1, 2, L, 128, generator=g).to(dtype) for _ in range(2))
    want = orc.estimate_block_sums(q.float(), k.float(), 128, stride, 1.0, chunk, True, "torch")
    k[:, :, column * stride + 1, 7] = float("nan")
    got = ops.estimate_block_sums(q.to(DEV), k.to(DEV), stride, 128, chunk, 1.0, True).cpu()
    last = column * stride // 128                        # query and key block of the last row and its column
    want, got = want[:, :, last], got[:, :, last]
    assert bool(got[..., last].isnan().all())
    want = want[..., :last] / (1 - want[..., last:last + 1])
    assert torch.allclose(got[..., :last], want, rtol=RTOL, atol=ATOL), float((got[..., :last] - want).abs().max())


@pytest.mark.parametrize("stride,chunk,lq,lk", [(16, 512, 4096, 4096), (16, 1536, 4608, 9216), (8, 512, 1536, 3072), (4, 1024, 5120, 5120), (32, 2560, 5120, 5120)])
def test_row_tiles_that_span_chunks(stride, chunk, lq, lk):
    """The chunk band of row tiles of which every query block has a chunk of its own: the columns of it in the dense sums (which
    another kernel may finish: sums of up to 128 x 32 probabilities in another order, 2^-24 each)."""
    from xattn_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(chunk)
    q, k = torch.randn(1, 4, lq, 128, device=DEV, generator=g).bfloat16(), torch.randn(1, 2, lk, 128, device=DEV, generator=g).bfloat16()
    dense, band = (ops.estimate_block_sums(q, k, stride, 128, chunk, 1.0, True, band=b) for b in (False, True))
    bpc, first = chunk // 128, (lk - lq) // 128
    for c in range(lq // chunk):
        rows = slice(c * bpc, (c + 1) * bpc)
        assert torch.allclose(band[:, :, rows], dense[:, :, rows, first + c * bpc:first + (c + 1) * bpc], rtol=1e-5, atol=1e-6)
    got = dense.cpu()
    want = orc.estimate_block_sums(q.float().cpu(), k.float().cpu().repeat_interleave(2, 1), 128, stride, 1.0, chunk, True, "torch")
    assert torch.allclose(got, want, rtol=RTOL, atol=ATOL), float((got - want).abs().max())


@pytest.mark.parametrize("lq,lk,stride,chunk,causal", [(3, 3, 32, 2048, True), (1, 5, 16, 16384, False), (413, 4096, 8, 2048, True),
                                                       (2500, 2500, 4, 8192, False), (1000, 1000, 16, 2048, True)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_operands_at_the_end_of_their_memory(dtype, lq, lk, stride, chunk, causal):
    """Nothing past the end of q and k is named by a load: both end where an allocation of their own does (its size a multiple
    of what the allocator maps), stored as a projection leaves them.  Lengths below the stride, row and column tiles past the
    end, a ragged last group."""
    from xattn_b200 import ops
    hq, hkv = 9, 3
    ends = []
    for h, n in ((hq, lq), (hkv, lk)):
        memory = torch.zeros((64 << 20) // torch.finfo(dtype).bits * 8, dtype=dtype, device=DEV)
        ends.append(memory[-n * h * 128:].view(1, n, h, 128).transpose(1, 2))
        ends[-1].copy_(torch.randn(1, h, n, 128, generator=torch.Generator().manual_seed(n)).to(dtype))
    got = ops.estimate_block_sums(*ends, stride, 128, chunk, 1.0, causal)
    assert torch.equal(got, ops.estimate_block_sums(*(x.clone() for x in ends), stride, 128, chunk, 1.0, causal))
