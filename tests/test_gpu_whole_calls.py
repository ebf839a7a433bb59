"""Calls that one native call carries out as a whole (buffers, quantisation without padded copies, LSE
shift, FP32 rows) against the same work done in separate steps through the ctypes surface, resident
CTAs that walk many units, and per-query masks fetched as tiles.  Everything here keeps every operation
and its order, so bits are compared."""
import pytest
import torch

pytestmark = pytest.mark.gpu

import risaattention_b200 as risa  # noqa: E402
from risaattention_b200 import _backend, compare_native  # noqa: E402
from risaattention_b200.host_pipeline import int8_attention_from_host  # noqa: E402


def _inputs(head_dim, q_len, k_len, dtype, q_heads=4, kv_heads=2, batch=2, token_major=False):
    g = torch.Generator(device="cuda").manual_seed(head_dim * 10007 + k_len)

    def make(heads, n):
        x = torch.randn(batch, heads, n, head_dim, device="cuda", generator=g).to(dtype)
        return x.transpose(1, 2).contiguous().transpose(1, 2) if token_major else x

    return make(q_heads, q_len), make(kv_heads, k_len), make(kv_heads, k_len)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("head_dim,k_len", [(40, 300), (64, 63), (80, 1025), (77, 200), (128, 129),
                                            (200, 1500), (256, 257)])
@pytest.mark.parametrize("mode", ["absmax", "midpoint_affine"])
def test_whole_calls_give_the_bits_of_the_separate_steps(dtype, head_dim, k_len, mode):
    q, k, v = _inputs(head_dim, 130, k_len, dtype, token_major=k_len % 2 == 0)

    def calls():
        out, lse = risa.int8_attention(q, k, v, v_quantization=mode, return_lse=True)
        packed = risa.prequantize_int8_attention(q, k, v, v_quantization=mode, return_lse=True)
        nhd, lse2 = risa.int8_attention_from_prequantized(packed, output_layout="nhd",
                                                          return_lse=True)
        return [risa.int8_attention(q, k, v, v_quantization=mode), out, lse, nhd, lse2, packed.q,
                packed.k, packed.v, packed.q_scale, packed.k_scale, packed.v_scale,
                packed.v_center, packed.lse_shift]

    whole = calls()
    steps = compare_native.with_native(_backend._ABI, calls)
    for ours, want in zip(whole, steps):
        assert ours.dtype == want.dtype and ours.shape == want.shape
        assert ours.stride() == want.stride() and torch.equal(ours, want)
    _backend._C.device_status()


@pytest.mark.parametrize("is_causal", [False, True])
@pytest.mark.parametrize("head_dim,q_len,k_len", [(64, 700, 333), (128, 700, 320), (128, 300, 1500),
                                                  (256, 500, 129)])
def test_resident_ctas_over_many_units(head_dim, q_len, k_len, is_causal):
    """More (query block, head) units than SMs: each head alone -- a launch whose CTAs have one unit
    each -- gives the same rows.  (No shape here is one whose last round is cut into parts.)"""
    q, k, v = _inputs(head_dim, q_len, k_len, torch.bfloat16, q_heads=40, kv_heads=20, batch=3)
    out = risa.int8_attention(q, k, v, is_causal=is_causal)
    for b, h in ((0, 0), (1, 17), (2, 39), (2, 24)):
        alone = risa.int8_attention(q[b:b + 1, h:h + 1], k[b:b + 1, h // 2:h // 2 + 1],
                                    v[b:b + 1, h // 2:h // 2 + 1], is_causal=is_causal)
        assert torch.equal(alone[0, 0], out[b, h])
    _backend._C.device_status()


@pytest.mark.parametrize("dtype", [torch.bool, torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("head_dim,k_len,heads", [(64, 1000, 4), (64, 64, 4), (128, 1025, 4),
                                                  (256, 700, 4), (64, 200, 48), (128, 260, 48),
                                                  (256, 130, 48)])
@pytest.mark.parametrize("shared_heads", [False, True])
def test_mask_tiles_give_the_bits_of_the_all_paths_kernel(dtype, head_dim, k_len, heads, shared_heads):
    """Masks that are windows of wider rows (aligned rows of any length), with entries that hide: false,
    -inf, and the +inf and NaN that an additive mask also hides by; few units and several per CTA."""
    q, k, v = _inputs(head_dim, 300, k_len, torch.bfloat16, q_heads=heads)
    g = torch.Generator(device="cuda").manual_seed(k_len)
    wide = torch.randn(2, 1 if shared_heads else heads, 300, (k_len + 127) // 64 * 64, device="cuda",
                       generator=g)
    if dtype is torch.bool:
        wide = wide > -1
    else:
        wide = wide.to(dtype)
        wide[..., 7::13] = float("-inf")
        wide[..., 5, 9] = float("inf")
        wide[..., 6, 11] = float("nan")
    wide[..., 130, :] = False if dtype is torch.bool else float("-inf")
    mask = wide[..., :k_len]
    results = []
    for path in (0, 2):
        previous = _backend._C.set_attention_path(path)
        try:
            results.append(risa.int8_attention(q, k, v, attn_mask=mask, return_lse=True))
        finally:
            _backend._C.set_attention_path(previous)
    (own, own_lse), (every, every_lse) = results
    assert torch.equal(own, every)
    assert torch.equal(own_lse.view(torch.int32), every_lse.view(torch.int32))
    assert own[:, :, 130].count_nonzero() == 0
    _backend._C.device_status()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("head_dim", [64, 128, 256])
@pytest.mark.parametrize("k_len", [64 + 1, 200, 1100])
@pytest.mark.parametrize("what", ["largest_bias", "hiding_bias", "q", "k"])
def test_mask_tiles_with_scores_that_are_not_finite(dtype, head_dim, k_len, what):
    """A score that is not finite although its bias is -- infinite operands, or a bias whose product with
    log2(e) overflows -- does not hide its key; a bias of +inf or NaN does.  As in the all-paths kernel."""
    q, k, v = _inputs(head_dim, 300, k_len, torch.bfloat16)
    g = torch.Generator(device="cuda").manual_seed(k_len)
    wide = torch.randn(2, 4, 300, (k_len + 15) // 16 * 16, device="cuda", generator=g).to(dtype)
    mask = wide[..., :k_len]
    if what == "largest_bias":
        mask[:, 1, 5, 7] = mask[:, 1, 140, k_len - 1] = torch.finfo(dtype).max
        mask[:, 2, ::3, ::5] = torch.finfo(dtype).min
    elif what == "hiding_bias":
        mask[:, 1, 5, 7] = mask[:, 2, 299, k_len - 1] = float("inf")
        mask[:, 1, 140, 63] = mask[:, 2, 37, 64] = float("nan")
    else:
        (q if what == "q" else k)[:, 1, 33, 9] = float("inf")
    results = []
    for path in (0, 2):
        previous = _backend._C.set_attention_path(path)
        try:
            results.append(risa.int8_attention(q, k, v, attn_mask=mask, return_lse=True))
        finally:
            _backend._C.set_attention_path(previous)
    for own, every in zip(*results):  # as bits: NaN equals NaN
        assert torch.equal(own.view(torch.uint8), every.view(torch.uint8))
    _backend._C.device_status()


@pytest.mark.parametrize("rows", [1, 31, 32, 33, 255, 256, 257, 1024, 5000])
@pytest.mark.parametrize("key_blocks", [1, 33, 70])
def test_pack_selected_offsets_and_ids(rows, key_blocks):
    """Offsets, ids and summary of counts whose slices end in every position of the scan."""
    g = torch.Generator().manual_seed(rows)
    kept = torch.rand(rows, key_blocks, generator=g) < 0.4
    words = (key_blocks + 31) // 32
    weights = 2 ** torch.arange(32, dtype=torch.int64)
    bits = torch.nn.functional.pad(kept, (0, words * 32 - key_blocks)).view(rows, words, 32)
    bitmaps = (bits.long() * weights).sum(-1)
    bitmaps = torch.where(bitmaps >= 2**31, bitmaps - 2**32, bitmaps).int().cuda()
    counts = kept.sum(-1).int().cuda()
    totals = torch.ones(rows, 2, dtype=torch.float64, device="cuda")  # sums of ones are exact
    offsets = torch.full((rows + 1,), -1, dtype=torch.int32, device="cuda")
    ids = torch.full((rows * key_blocks,), -1, dtype=torch.int32, device="cuda")
    summary = torch.zeros(3, dtype=torch.float64, pin_memory=True)
    _backend._C.pack_selected(counts, bitmaps, totals, offsets, ids, summary, key_blocks,
                              _backend.current_stream_ptr(counts.device))
    torch.cuda.synchronize()
    total = int(kept.sum())
    assert offsets.tolist() == [0] + kept.sum(-1).cumsum(0).tolist()
    assert torch.equal(ids[:total].cpu(), kept.nonzero()[:, 1].int())
    assert (ids[total:] == -1).all() and summary.tolist() == [rows, rows, total]


def test_host_buffers_under_a_default_device_of_the_gpu():
    """Construction reads its summary from pinned host memory, and the host pipeline returns it: both
    name the host, so that ``torch.set_default_device`` does not move the buffer."""
    q, k, v = _inputs(128, 300, 1500, torch.bfloat16)
    out, pattern = risa.construct_sparse_int8_attention(q, k, v, theta=0.9)
    host = [x.cpu().pin_memory() for x in (q, k, v)]
    with torch.device("cuda"):
        again, same = risa.construct_sparse_int8_attention(q, k, v, theta=0.9)
        streamed = int8_attention_from_host(*host)
    assert torch.equal(out, again)
    assert torch.equal(pattern.row_offsets, same.row_offsets)
    assert torch.equal(pattern.block_indices, same.block_indices)
    assert not streamed.is_cuda and torch.equal(streamed, risa.int8_attention(q, k, v).cpu())


def _rows_of_any_length(heads, q_len, k_len, cta_k, scale, seed):
    """A pattern whose rows keep from one tile to all of them."""
    g = torch.Generator().manual_seed(seed)
    q_blocks, tiles = -(-q_len // 128), -(-k_len // cta_k)
    rows = heads * q_blocks
    counts = torch.randint(1, tiles + 1, (rows,), generator=g)
    kept = torch.rand(rows, tiles, generator=g).argsort(1).argsort(1) < counts[:, None]
    offsets = torch.cat([torch.zeros(1, dtype=torch.long), counts.cumsum(0)])
    return [risa.RetainedMassPattern(
        row_offsets=(offsets[first:last + 1] - offsets[first]).int().cuda(),
        block_indices=kept[first:last].nonzero()[:, 1].int().cuda(), batch_size=1,
        q_heads=(last - first) // q_blocks, q_length=q_len, kv_length=k_len, query_block_size=128,
        key_block_size=cta_k, attention_scale=scale, retained_mass_target=0.9,
        measured_retained_mass=0.9)
        for first, last in [(0, rows), *((h * q_blocks, (h + 1) * q_blocks) for h in range(heads))]]


@pytest.mark.parametrize("head_dim,q_len,k_len", [(64, 300, 1000), (128, 700, 1500), (128, 300, 700),
                                                  (256, 500, 1300), (128, 100, 4000)])
def test_units_of_any_length_are_drawn(head_dim, q_len, k_len):
    """Pattern rows of one to all tiles over many more units than SMs, on two streams at once and replayed
    from a graph: the rows of each head alone, whose few units all start at once."""
    heads = 150
    q, k, v = _inputs(head_dim, q_len, k_len, torch.bfloat16, q_heads=heads, kv_heads=heads // 2, batch=1)
    packed = risa.prequantize_int8_attention(q, k, v)
    whole, *single = _rows_of_any_length(heads, q_len, k_len, packed.cta_k, packed.attention_scale, 5)
    out = risa.int8_attention_from_prequantized(packed, sparse_pattern=whole)
    for h in (0, 1, 74, 149):
        alone = risa.sparse_int8_attention(q[:, h:h + 1], k[:, h // 2:h // 2 + 1],
                                           v[:, h // 2:h // 2 + 1], single[h])
        assert torch.equal(alone[0, 0], out[0, h])
    streams = [torch.cuda.Stream() for _ in range(2)]
    results = []
    for _ in range(3):
        for stream in streams:
            stream.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(stream):
                results.append(risa.int8_attention_from_prequantized(packed, sparse_pattern=whole))
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):
        results.append(risa.int8_attention_from_prequantized(packed, sparse_pattern=whole))
    results[-1].zero_()
    graph.replay()
    torch.cuda.synchronize()
    assert all(torch.equal(out, x) for x in results)
    _backend._C.device_status()


@pytest.mark.parametrize("head_dim", [64, 128, 256])
@pytest.mark.parametrize("dtype", [torch.bool, torch.bfloat16])
def test_sequences_of_any_length_are_drawn(head_dim, dtype):
    """A padded batch from no visible key at all to all of them, many units: each sequence alone."""
    batch, q_len, k_len = 12, 400, 2100
    q, k, v = _inputs(head_dim, q_len, k_len, torch.bfloat16, q_heads=8, kv_heads=4, batch=batch)
    lengths = torch.tensor([2100, 0, 1, 127, 128, 129, 2099, 0, 1024, 64, 700, 2048], device="cuda")
    mask = (torch.arange(k_len, device="cuda") < lengths[:, None])[:, None, None, :]
    if dtype is not torch.bool:
        mask = torch.zeros(mask.shape, device="cuda").masked_fill(~mask, float("-inf")).to(dtype)
    out, lse = risa.int8_attention(q, k, v, attn_mask=mask, return_lse=True)
    for i in range(batch):
        alone, its_lse = risa.int8_attention(q[i:i + 1], k[i:i + 1], v[i:i + 1],
                                             attn_mask=mask[i:i + 1], return_lse=True)
        assert torch.equal(alone[0], out[i]) and torch.equal(its_lse[0], lse[i])
    assert out[1].count_nonzero() == 0 and torch.isneginf(lse[1]).all()
    _backend._C.device_status()


def _split_shape(head_dim):
    """160 units, 12 more than SMs, whose last ones are cut into key-range parts."""
    q_len = 2000 if head_dim > 128 else 4000
    kernel_dim = 256 if head_dim > 128 else 128
    assert _backend._ABI.lib.risa_b200_attention_scratch_size(1, 5, q_len, 4000, kernel_dim, 128) > 0
    return _inputs(head_dim, q_len, 4000, torch.float32, q_heads=5, kv_heads=5, batch=1)


@pytest.mark.parametrize("head_dim", [80, 128, 200, 256])
def test_fp32_rows_and_shifted_lse_of_a_split_last_wave(head_dim):
    """The launch that merges key-range parts stores FP32 rows of the caller's width and adds the LSE
    shift: the bits of BF16 rows converted and of the shift added afterwards."""
    q, k, v = _split_shape(head_dim)

    def calls():
        packed = risa.prequantize_int8_attention(q, k, v, return_lse=True)
        nhd, lse = risa.int8_attention_from_prequantized(packed, output_layout="nhd", return_lse=True)
        return [*risa.int8_attention(q, k, v, return_lse=True), nhd, lse, risa.int8_attention(q, k, v)]

    for ours, want in zip(calls(), compare_native.with_native(_backend._ABI, calls)):
        assert ours.dtype == want.dtype and torch.equal(ours, want)
    _backend._C.device_status()


def test_calls_that_are_never_split_reserve_no_parts():
    """The parts of a split last wave are room that only plain calls need."""
    q, k, v = _split_shape(128)
    parts = _backend._ABI.lib.risa_b200_attention_scratch_size(1, 5, 4000, 4000, 128, 128)
    mask = torch.ones(1, 1, 1, 4000, dtype=torch.bool, device="cuda")

    def peak(**options):
        torch.cuda.synchronize()
        before = torch.cuda.memory_allocated()
        torch.cuda.reset_peak_memory_stats()
        risa.int8_attention(q, k, v, **options)
        return torch.cuda.max_memory_allocated() - before

    plain = peak()
    for options in ({"attn_mask": mask}, {"is_causal": True}):
        assert peak(**options) <= plain - parts + 65536  # the tile list of the mask
