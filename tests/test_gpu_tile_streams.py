"""The attention kernels where tiles and chunks of very different lengths follow one another on one SM, against a plain
fp32 softmax on the GPU.

Tolerance: P and the result are rounded to 16 bits (relative 2^-9 in bf16), so an element is off by at most about
2 * 2^-9 * max|v| plus its own rounding; max|v| of the normal draws below is under 5, hence 2e-2, and a tenth of it on average."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.fixture(autouse=True)
def _needs_gpu(built_library):
    if not torch.cuda.is_available():
        pytest.fail("GPU tests need a CUDA device")


def _close(got, ref):
    err = (got.float() - ref).abs()
    assert err.max().item() <= 2e-2 and err.mean().item() <= 2e-3, (err.max().item(), err.mean().item())


@pytest.mark.parametrize("pq", [64, 128])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("longest,rise", [(2, 0.0), (300, 0.0), (300, 6.0)])
def test_tiles_of_unequal_length(pq, dtype, longest, rise):
    """More tiles than SMs several times over, with 0, 1, 2 ... chunks in no order.  ``rise``: scores that grow along the
    list, so that the running maximum moves in every chunk and the partial results are rescaled."""
    from vecattention_b200.api import _sparse_attn_bhsd
    g = torch.Generator(device=DEV).manual_seed(5 + longest)
    h, hkv, sk = 6, 2, 2000
    nq = 900 // h
    sq = nq * pq - 7
    q = torch.randn(1, h, sq, 128, generator=g, device=DEV)
    k = torch.randn(1, hkv, sk, 128, generator=g, device=DEV)
    if rise:
        q[..., 0] = 8.0
        k[..., 0] = torch.linspace(0, rise * 11.3 / 8.0 * 4, sk, device=DEV)
    q, k = q.to(dtype), k.to(dtype)
    v = torch.randn(1, hkv, sk, 128, generator=g, device=DEV).to(dtype)
    count = (torch.rand(1, h, nq, generator=g, device=DEV) ** 2 * (longest + 1)).int().clamp(max=longest)
    cap = (longest + 3) // 4 * 4
    order = torch.rand(h, nq, sk, generator=g, device=DEV).argsort(-1)[..., :cap].sort(-1).values
    index = order.int()[None].contiguous()
    out = _sparse_attn_bhsd(q, k, v, pq, None, None, count, index, False)
    valid = torch.arange(cap, device=DEV) < count[0, :, :, None]
    for i in range(h):
        kk, vv = k[0, i // 3].float()[index[0, i].long()], v[0, i // 3].float()[index[0, i].long()]
        qq = torch.nn.functional.pad(q[0, i].float(), (0, 0, 0, 7)).view(nq, pq, 128)
        s = torch.bmm(qq, kk.transpose(1, 2)) / math.sqrt(128)
        s.masked_fill_(~valid[i][:, None], -math.inf)
        ref = torch.bmm(torch.softmax(s, -1).nan_to_num(0.0), vv).view(nq * pq, 128)[:sq]
        _close(out[0, i], ref)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("s", [1, 127, 128, 129, 700, 2500])
@pytest.mark.parametrize("bshd", [False, True])
def test_dense_rows(dtype, s, bshd):
    from vecattention_b200.dispatch import Full_prefill
    g = torch.Generator(device=DEV).manual_seed(s)

    def make(n):
        x = torch.randn(2, s, n, 128, generator=g, device=DEV).to(dtype).transpose(1, 2)
        return x if bshd else x.contiguous()

    q, k, v = make(6), make(2), make(2)
    out = Full_prefill(q, k, v)
    ref = torch.nn.functional.scaled_dot_product_attention(q.float(), k.float().repeat_interleave(3, 1),
                                                           v.float().repeat_interleave(3, 1), is_causal=True)
    _close(out, ref)


@pytest.mark.parametrize("pq", [64, 128])
def test_repeated_rows(pq):
    """V of one row that is read as many (a stride of 0): its row comes out, whatever the weights."""
    from vecattention_b200.api import _sparse_attn_bhsd
    from vecattention_b200.dispatch import Full_prefill
    g = torch.Generator(device=DEV).manual_seed(9)
    q, k = (torch.randn(1, 2, 400, 128, generator=g, device=DEV).bfloat16() for _ in range(2))
    one = torch.randn(1, 2, 1, 128, generator=g, device=DEV).bfloat16()
    v = one.expand(1, 2, 400, 128)
    nq = -(-400 // pq)
    count = torch.full((1, 2, nq), 200, dtype=torch.int32, device=DEV)
    index = torch.arange(0, 400, 2, dtype=torch.int32, device=DEV).expand(1, 2, nq, 200).contiguous()
    _close(_sparse_attn_bhsd(q, k, v, pq, None, None, count, index, False), v.float())
    _close(Full_prefill(q, k, v), v.float())


@pytest.mark.parametrize("s,row", [(700, 0), (700, 63), (700, 64), (700, 100), (700, 320), (700, 699), (100, 99)])
@pytest.mark.parametrize("bad", [math.inf, math.nan])
def test_dense_rows_and_values_that_are_not_finite(s, row, bad):
    """Keys after a row's own have weight zero, and a row of V that is not finite reaches back no further than its 64-key
    block, which the operator's tiles take as a whole.  (One batch entry and head has it, the others none.)"""
    from vecattention_b200.dispatch import Full_prefill
    g = torch.Generator(device=DEV).manual_seed(row)
    q = torch.randn(2, 4, s, 128, generator=g, device=DEV).bfloat16()
    k, v = (torch.randn(2, 2, s, 128, generator=g, device=DEV).bfloat16() for _ in range(2))
    ref = Full_prefill(q, k, v)
    v[1, 1, row] = bad
    out = Full_prefill(q, k, v)
    before = row // 64 * 64
    assert torch.equal(out[1, 2:, :before], ref[1, 2:, :before])
    assert not out[1, 2:, row:].isfinite().any()
    assert torch.equal(out[0], ref[0]) and torch.equal(out[1, :2], ref[1, :2])


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("begin,end", [(37, 3300), (0, 3500), (1, 3499), (1000, 1087), (3000, 3300)])
def test_vision_span_over_many_tiles(dtype, begin, end):
    """The one-launch composition with several tiles for every SM: sparse and dense tiles and skipped ones (those before
    the span) follow one another in a CTA.  Dense rows against a plain softmax; all rows the same bits as three launches."""
    from vecattention_b200 import VecAttention_prefill_vision
    g = torch.Generator(device=DEV).manual_seed(begin + end)
    s, h, hkv = 3500, 28, 4
    q = torch.randn(1, h, s, 128, generator=g, device=DEV).to(dtype)
    k, v = (torch.randn(1, hkv, s, 128, generator=g, device=DEV).to(dtype) for _ in range(2))
    one, three = (VecAttention_prefill_vision(q, k, v, 0.8, 64, 16, 16, True, 65536, vision_start_position=begin,
                                              vision_end_position=end, fused=f) for f in (True, False))
    assert torch.equal(one, three)
    ref = torch.nn.functional.scaled_dot_product_attention(q.float(), k.float().repeat_interleave(h // hkv, 1),
                                                           v.float().repeat_interleave(h // hkv, 1), is_causal=True)
    for rows in (slice(0, begin), slice(end, s)):
        if rows.start < rows.stop:
            _close(one[:, :, rows], ref[:, :, rows])


@pytest.mark.parametrize("pq,bk,group", [(64, 16, 16), (128, 128, 1)])
def test_causal_tiles_head_by_head(pq, bk, group):
    """Heads whose K and V have at most 64 MB together are listed together, tile by tile: the same bits in any grouping.
    16 heads of 8700 tokens are 68 MB (two groups of eight), four of them 17 (one group)."""
    from vecattention_b200 import VecAttention_prefill
    g = torch.Generator(device=DEV).manual_seed(pq)
    h, s = 16, 8700
    q, k, v = (torch.randn(1, h, s, 128, generator=g, device=DEV).bfloat16() for _ in range(3))
    run = lambda i, n: VecAttention_prefill(*(t[:, i:i + n] for t in (q, k, v)), 0.8, pq, bk, group, True, 16384)  # noqa: E731
    assert torch.equal(run(0, h), torch.cat([run(i, 4) for i in range(0, h, 4)], dim=1))


@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("heads,kv,s", [(5, 5, 45000), (6, 3, 45001), (3, 3, 140000)])
def test_groups_of_heads(heads, kv, s, causal):
    """Groups of unequal size (5 KV heads of 23 MB: 2 + 2 + 1), of several query heads per KV head, and of one head because
    its K and V alone exceed 64 MB: the same bits as a call per KV head."""
    from vecattention_b200 import VecAttention_prefill
    g = torch.Generator(device=DEV).manual_seed(s)
    q = torch.randn(1, heads, s, 128, generator=g, device=DEV, dtype=torch.bfloat16)
    k, v = (torch.randn(1, kv, s, 128, generator=g, device=DEV, dtype=torch.bfloat16) for _ in range(2))
    rep = heads // kv
    run = lambda i, n: VecAttention_prefill(q[:, i * rep:(i + n) * rep], k[:, i:i + n], v[:, i:i + n], 0.97, 64, 16, 16, causal, 32768)  # noqa: E731
    assert torch.equal(run(0, kv), torch.cat([run(i, 1) for i in range(kv)], dim=1))


@pytest.mark.parametrize("heads,kv,s,pq,bk,group,causal", [
    (4, 4, 2048, 64, 16, 16, False),    # segments of one group each
    (3, 3, 700, 64, 16, 1, True),       # fewer tiles than segments
    (14, 2, 9001, 64, 16, 1, True),     # groups inside a tile; row blocks of several heads
    (14, 2, 9001, 64, 16, 3, True),     # a group starts with a tile every third tile only
    (5, 5, 12800, 64, 32, 5, False),    # ... every fifth
    (14, 2, 20011, 64, 16, 100, True),  # ... every 25th, longer than some segments
    (28, 4, 9001, 64, 16, 8192, True),  # one group: segments walk all keys before them
    (3, 3, 30000, 64, 16, 8192, False),
    (40, 20, 5000, 64, 64, 2, False),   # 40 row blocks in three segments each
    (80, 20, 16000, 64, 16, 16, False), # 160 row blocks: a whole wave on 148 SMs, and the other 12 in eleven segments each
    (4, 4, 9000, 128, 128, 1, True),
    (4, 2, 9000, 128, 64, 4, True),
])
@pytest.mark.parametrize("chunk_tiles", [0, 24])
def test_selection_in_segments(heads, kv, s, pq, bk, group, causal, chunk_tiles):
    """The work of a selection is cut into row blocks and key segments by the number of both: the same lists as one query
    head at a time with 64 tiles a call, which cuts it elsewhere (and, causal, orders the rows differently)."""
    from vecattention_b200.api import average_vector, fuse_qk_softmax_minp_wo_causal
    g = torch.Generator(device=DEV).manual_seed(s + group)
    q = average_vector(torch.randn(1, heads, s, 128, generator=g, device=DEV).bfloat16() + 0.5, pq)
    k = torch.randn(1, kv, s, 128, generator=g, device=DEV).bfloat16()
    gap = torch.rand(heads, generator=g, device=DEV) * 0.1 + 0.1

    def lists(q, k, offset, gap):
        count, index = fuse_qk_softmax_minp_wo_causal(q, k, offset, gap, causal, pq, bk, causal, group, trim=False, chunk_tiles=chunk_tiles)
        return index.masked_fill_(torch.arange(index.shape[-1], device=DEV) >= count[..., None], -1)

    whole = lists(q, k, 0, gap)
    step = chunk_tiles or 64
    for h in range(heads):
        kh = h // (heads // kv)
        for t in range(0, q.shape[2], step):
            part = lists(q[:, h:h + 1, t:t + step], k[:, kh:kh + 1], t, gap[h:h + 1])
            assert torch.equal(part, whole[:, h:h + 1, t:t + step])


@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("pq,bk", [(64, 16), (128, 128)])
def test_calls_in_a_row_and_in_a_graph(pq, bk, causal):
    """The kernels of a call are launched before the ones ahead of them have ended.  Calls on alternating inputs that share one
    workspace and one output, without waiting in between, and a captured call that is replayed on new inputs, give what
    each gives alone."""
    from vecattention_b200 import VecAttention_prefill
    g = torch.Generator(device=DEV).manual_seed(pq)
    sets = [[torch.randn(1, n, 1500, 128, generator=g, device=DEV).bfloat16() for n in (6, 2, 2)] for _ in range(3)]
    run = lambda x, **kw: VecAttention_prefill(*x, 0.8, pq, bk, 1, causal, 16384, **kw)  # noqa: E731
    alone = []
    for x in sets:
        alone.append(run(x).clone())
        torch.cuda.synchronize()
    out, kept = torch.empty_like(sets[0][0]), []
    for i in range(30):
        run(sets[i % 3], out=out)
        kept.append(out.clone())
    for i, o in enumerate(kept):
        assert torch.equal(o, alone[i % 3])
    x = [t.clone() for t in sets[0]]
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        run(x, out=out)
        run(x, out=out)
    for i in (1, 2, 0):
        for a, b in zip(x, sets[i]):
            a.copy_(b)
        graph.replay()
        assert torch.equal(out, alone[i])


@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("pq,bk", [(64, 16), (128, 128)])
def test_selection_and_attention_in_a_row_on_the_same_buffers(pq, bk, causal):
    """Selection and attention through the C interface, again and again on alternating inputs with one set of scratch, counts and
    lists, with nothing launched between them and nothing waited for: every kernel overlaps the end of the one that
    writes what it reads.  Each call gives what it gives alone."""
    import ctypes as C
    from vecattention_b200 import _lib as L
    from vecattention_b200.api import _check, _stream, _t4, average_vector, block_tables
    heads, kv, s = 6, 2, 1500
    nq, cap = -(-s // pq), (s + 3) // 4 * 4
    g = torch.Generator(device=DEV).manual_seed(pq)
    sets = [[torch.randn(1, n, s, 128, generator=g, device=DEV).bfloat16() for n in (heads, kv, kv)] for _ in range(3)]
    avg = [average_vector(x[0], pq) for x in sets]
    bcnt, bidx = block_tables(1, heads, s, pq, causal, DEV)
    count = torch.empty(1, heads, nq, dtype=torch.int32, device=DEV)
    index = torch.empty(1, heads, nq, cap, dtype=torch.int32, device=DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    outs = [torch.empty_like(sets[0][0]) for _ in range(33)]
    ws, calls = None, []
    for i, out in enumerate(outs):
        q, k, v = sets[i % 3]
        sel = L.SelectArgs(L.VA_BF16, 1, heads, kv, nq, s, 128, pq, bk, 1, causal, causal, 64, 0, avg[i % 3].data_ptr(), _t4(k),
                           0.2, None, 0, count.data_ptr(), index.data_ptr(), cap, status.data_ptr(), 0, None, 0)
        if ws is None:
            nbytes = C.c_size_t(0)
            _check(L.lib().va_select_workspace_bytes(C.byref(sel), C.byref(nbytes)))
            ws = torch.empty(nbytes.value, dtype=torch.uint8, device=DEV)
        sel.workspace, sel.workspace_bytes = ws.data_ptr(), ws.numel()
        calls.append((sel, L.AttnArgs(L.VA_BF16, 1, heads, kv, s, s, 128, pq, causal, 0, _t4(q), _t4(k), _t4(v), _t4(out), bcnt.data_ptr(),
                                      bidx.data_ptr(), bidx.shape[-1], count.data_ptr(), index.data_ptr(), cap, 0.0, status.data_ptr(),
                                      None, 0, 0, 0)))
    torch.cuda.synchronize()
    for i, (sel, att) in enumerate(calls):
        _check(L.lib().va_select(C.byref(sel), _stream()))
        _check(L.lib().va_sparse_attn(C.byref(att), _stream()))
        if i < 3:  # alone
            torch.cuda.synchronize()
    torch.cuda.synchronize()
    assert status.item() == 0 and not torch.equal(outs[0], outs[1])
    for i, out in enumerate(outs):
        assert torch.equal(out, outs[i % 3])


@pytest.mark.parametrize("what", ["dense", "vision", "operator"])
def test_calls_right_behind_the_kernels_that_write_their_inputs(what):
    """Inputs written by the launches just before the call, in the same stream, and in a captured call that starts behind an
    event of the stream in which they are written."""
    from vecattention_b200 import VecAttention_prefill, VecAttention_prefill_vision
    from vecattention_b200.dispatch import Full_prefill
    call = {"dense": lambda q, k, v: Full_prefill(q, k, v),
            "vision": lambda q, k, v: VecAttention_prefill_vision(q, k, v, 0.8, 64, 16, 16, True, 16384, vision_start_position=100,
                                                                  vision_end_position=1300),
            "operator": lambda q, k, v: VecAttention_prefill(q, k, v, 0.8, 64, 16, 16, True, 16384)}[what]
    g = torch.Generator(device=DEV).manual_seed(3)
    sets = [[torch.randn(1, n, 1500, 128, generator=g, device=DEV).bfloat16() for n in (6, 2, 2)] for _ in range(3)]
    alone = []
    for x in sets:
        alone.append(call(*x))
        torch.cuda.synchronize()
    x, got = [torch.empty_like(t) for t in sets[0]], []
    for i in range(30):
        for a, b in zip(x, sets[i % 3]):
            torch.add(b, 0.0, out=a)
        got.append(call(*x))
    for i, o in enumerate(got):
        assert torch.equal(o, alone[i % 3])
    source = [t.clone() for t in sets[0]]
    graph, side = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with torch.cuda.graph(graph):
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            for a, b in zip(x, source):
                torch.add(b, 0.0, out=a)
        torch.cuda.current_stream().wait_stream(side)
        out = call(*x)
    for i in (1, 2, 0, 2):
        for a, b in zip(source, sets[i]):
            a.copy_(b)
        graph.replay()
        assert torch.equal(out, alone[i])


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("heads,kv,s", [(300, 100, 200), (40, 40, 1400), (30, 5, 1281)])
def test_dense_tiles_that_follow_one_another(dtype, heads, kv, s):
    """Several dense tiles for every SM, of 1 to 11 chunks, with scores that grow along the keys, so that the running maximum
    moves and partial results are rescaled.  A value that is not finite in the last row reaches only the last block."""
    from vecattention_b200.dispatch import Full_prefill
    g = torch.Generator(device=DEV).manual_seed(s)
    q = torch.randn(1, heads, s, 128, generator=g, device=DEV)
    k = torch.randn(1, kv, s, 128, generator=g, device=DEV)
    q[..., 0] = 8.0
    k[..., 0] = torch.linspace(0, 40.0, s, device=DEV)
    q, k = q.to(dtype), k.to(dtype)
    v = torch.randn(1, kv, s, 128, generator=g, device=DEV).to(dtype)
    out = Full_prefill(q, k, v)
    rep = heads // kv
    ref = torch.nn.functional.scaled_dot_product_attention(q.float(), k.float().repeat_interleave(rep, 1),
                                                           v.float().repeat_interleave(rep, 1), is_causal=True)
    _close(out, ref)
    v[:, :, -1] = math.inf
    again = Full_prefill(q, k, v)
    whole = (s - 1) // 64 * 64
    assert torch.equal(again[:, :, :whole], out[:, :, :whole]) and not again[:, :, -1].isfinite().any()


@pytest.mark.parametrize("n", [1, 28, 127, 128, 129, 70000])
def test_gaps_of_thresholds(n):
    """Gaps from thresholds on the device: the bits of the expression they stand for, also at 0, 1, infinity, NaN and below
    zero, and of a part of a larger tensor.  Other types and layouts take that expression itself."""
    from vecattention_b200.api import _gap_of
    dev = torch.device(DEV, torch.cuda.current_device())
    g = torch.Generator(device=DEV).manual_seed(n)
    t = torch.rand(n + 5, generator=g, device=DEV) ** 3
    t[5:][:5] = torch.tensor([0.0, 1.0, math.inf, math.nan, -1.0], device=DEV)[:min(n, 5)]
    for x in (t[5:], t[5:].double(), t[5:].half(), t.expand(3, n + 5)[:, 5:], t[5:].cpu()):
        want = -torch.log(x.to(dev) + 1e-9)
        got = _gap_of(x, dev)
        assert got.dtype == want.dtype and got.shape == want.shape
        assert torch.equal(got.nan_to_num(7.0, 8.0, 9.0), want.nan_to_num(7.0, 8.0, 9.0)) and torch.equal(got.isnan(), want.isnan())
