"""GPU: the dense-stage kernels for one-tile items (chunks of at most 512 keys, in all but long calls of at most 1024, at
head dim 256 of at most 256, and query windows with at most 128 rows per kv head), the row gathers, and the small kernels around them, at the sizes and
strides where their branches change.

Outputs are compared with the mma.sync dense stage.  Both round P to 16 bits and a partial row to 11
significant bits and sum in fp32, so an output element, a weighted mean of values of order one, differs by the
rounding of P (2^-9 bf16, 2^-11 fp16 relative, averaging out over the keys) and one rounding of the output:
at most two units of the output type at magnitude 4, 2^-5 in bf16 and 2^-8 in fp16; the mean
difference is an order of magnitude below one unit at magnitude 1."""
import ctypes as C

import pytest
import torch

from baselinebenchmark_b200 import _lib, parallel
from oracle import moba_oracle as O
from tests import gpu_util as G

pytestmark = pytest.mark.gpu

DTYPES = [pytest.param(torch.bfloat16, id="bf16"), pytest.param(torch.float16, id="fp16")]


def _inputs(lens, hq, hkv, d, chunk, dtype, seed):
    q, k, v, cu = O.make_inputs(list(lens), hq, hkv, d, chunk, seed=seed)
    return (*G.to_dev(q.to(dtype), k.to(dtype), v.to(dtype)), torch.from_numpy(cu).cuda())


def _close(out, ref, dtype):
    mx, mean = G.rel_stats(out, ref)
    unit = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    assert mx <= 8 * unit and mean <= 0.25 * unit, (mx, mean)


def _kernel(q, k, v, cu, max_len, chunk, topk, begin=None):
    prob = parallel.make_problem(q, k, v, torch.empty_like(q), cu, max_len, chunk, topk, None, begin)
    return _lib.lib().moba_problem_attend_kernel(C.byref(prob))


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("d", [64, 96, 128, 256])
@pytest.mark.parametrize("chunk", [16, 64, 127, 128, 129, 200, 256, 257, 512, 513, 1025])
def test_chunk_sizes_around_the_tiles(chunk, d, dtype):
    lens, hq, hkv, topk = (1, 130, max(1025, 2 * chunk + 1), 700), 6, 2, 5
    q, k, v, cu = _inputs(lens, hq, hkv, d, chunk, dtype, seed=chunk + d)
    out, lse, sel = parallel.moba_forward(q, k, v, cu, max(lens), chunk, topk, return_lse=True, return_selected=True)
    ref, ref_lse, ref_sel = parallel.moba_forward(q, k, v, cu, max(lens), chunk, topk, return_lse=True,
                                                  return_selected=True, attend_impl=_lib.ATTEND_MMA_SYNC)
    assert torch.equal(sel, ref_sel)
    _close(out, ref, dtype)
    assert (lse - ref_lse).abs().max().item() < 1e-3       # scores in fp32, exponentials to 7.5e-5


@pytest.mark.parametrize("d,dtype", [(64, torch.float16), (96, torch.bfloat16), (128, torch.bfloat16)])
@pytest.mark.parametrize("chunk", [63, 64, 95, 96, 128])
@pytest.mark.parametrize("lens,hq,hkv", [((5000,), 16, 1), ((700, 9000), 16, 4), ((4100, 3, 4095), 12, 12), ((33,), 16, 2)])
def test_streams_of_one_tile_items(lens, hq, hkv, chunk, d, dtype):
    """Chunks of 96 to 128 keys (64 and up at head dim 64) on the one-tile kernel, below and in small calls the kernel for short items: a CTA's
    items run through a ring of descriptions, of Q, K and V tiles and of places in tensor memory, each many times over in the
    longer calls; lists of many tiles (few kv heads) and of one, K and V shared by the heads of a group and not.  Windows, some of
    more rows than one tile, run either kernel: the same bits."""
    topk = 9
    q, k, v, cu = _inputs(lens, hq, hkv, d, chunk, dtype, seed=chunk + d + hq)
    q *= 3                                                   # a moving softmax reference
    args = (k, v, cu, max(lens), chunk, topk)
    one_tile = chunk >= (64 if d == 64 else 96) and lens != (33,)
    assert _kernel(q, *args) == (_lib.KERNEL_ONE_TILE if one_tile else _lib.KERNEL_SHORT)
    out, lse, sel = parallel.moba_forward(q, *args, return_lse=True, return_selected=True)
    ref, ref_lse, ref_sel = parallel.moba_forward(q, *args, return_lse=True, return_selected=True,
                                                  attend_impl=_lib.ATTEND_MMA_SYNC)
    assert torch.equal(sel, ref_sel)
    _close(out, ref, dtype)
    assert (lse - ref_lse).abs().max().item() < 1e-3
    total, few = sum(lens), 128 // (hq // hkv)
    for begin, n in ((total - few, few), (total // 2, few + 1), (total // 3, min(400, total - total // 3)), (total - 1, 1)):
        if begin < 0 or begin + n > total:
            continue
        o, l, s = parallel.moba_forward(q[begin:begin + n], *args, return_lse=True, return_selected=True, q_token_begin=begin)
        assert torch.equal(s, sel[:, :, begin:begin + n])
        assert torch.equal(o, out[begin:begin + n]) and torch.equal(l, lse[:, begin:begin + n]), (begin, n)


@pytest.mark.parametrize("d,dtype", [(64, torch.float16), (96, torch.bfloat16), (128, torch.bfloat16)])
@pytest.mark.parametrize("chunk", [1000, 1024, 1025])
def test_chunks_of_up_to_1024_keys_on_either_kernel(chunk, d, dtype):
    """Chunks of 513 to 1024 keys are items of half a 256-row tile (the last half of a list may be empty or ragged); one
    key more and the 256-row kernel runs."""
    lens, hq, hkv, topk = (1, 3 * chunk + 77, 1023, 5 * chunk), 6, 2, 4
    q, k, v, cu = _inputs(lens, hq, hkv, d, chunk, dtype, seed=chunk + d)
    out, lse, sel = parallel.moba_forward(q, k, v, cu, max(lens), chunk, topk, return_lse=True, return_selected=True)
    ref, ref_lse, ref_sel = parallel.moba_forward(q, k, v, cu, max(lens), chunk, topk, return_lse=True,
                                                  return_selected=True, attend_impl=_lib.ATTEND_MMA_SYNC)
    assert torch.equal(sel, ref_sel)
    _close(out, ref, dtype)
    assert (lse - ref_lse).abs().max().item() < 1e-3
    for begin, n in ((100, 200), (3 * chunk - 5, 131)):                       # windows of more rows than one tile
        o, l, s = parallel.moba_forward(q[begin:begin + n], k, v, cu, max(lens), chunk, topk, return_lse=True,
                                        return_selected=True, q_token_begin=begin)
        assert torch.equal(s, sel[:, :, begin:begin + n])
        assert torch.equal(o, out[begin:begin + n]) and torch.equal(l, lse[:, begin:begin + n])


def test_a_long_call_equals_its_windows_and_its_head_groups():
    """At head dim 128 and chunks of 769 to 1024 keys a call of more than 2^21 partial rows runs the 256-row kernel; its
    windows and, in a small workspace, its kv heads one by one are calls of fewer rows and run the kernel for one-tile
    items.  Large scores, so that the softmax reference of many rows moves inside a chunk."""
    tokens, hq, hkv, d, chunk, topk = 8200, 32, 8, 128, 1024, 8
    assert tokens * hq * topk > 1 << 21
    q, k, v, cu = _inputs((tokens,), hq, hkv, d, chunk, torch.bfloat16, seed=5)
    q *= 4
    args = (k, v, cu, tokens, chunk, topk)
    out, lse, sel = parallel.moba_forward(q, *args, return_lse=True, return_selected=True)
    prob, _ = G.problem_for(q, k, v, cu, tokens, chunk, topk)
    assert G.dims_of(prob).rows * G.dims_of(prob).partials == tokens * hq * topk
    least = C.c_size_t()
    _lib.check(_lib.lib().moba_workspace_size_min(C.byref(prob), C.byref(least)))
    out2, lse2, sel2 = parallel.moba_forward(q, *args, return_lse=True, return_selected=True, workspace_limit=least.value)
    assert torch.equal(sel2, sel) and torch.equal(out2, out) and torch.equal(lse2, lse)
    for begin, n in ((0, 700), (5 * chunk - 3, 2000), (tokens - 33, 33), (tokens - 32, 32), (tokens - 1, 1)):
        o, l, s = parallel.moba_forward(q[begin:begin + n], *args, return_lse=True, return_selected=True, q_token_begin=begin)
        assert torch.equal(s, sel[:, :, begin:begin + n])
        assert torch.equal(o, out[begin:begin + n]) and torch.equal(l, lse[:, begin:begin + n]), (begin, n)


@pytest.mark.parametrize("hq,hkv", [(4, 4), (8, 2), (16, 1)])
@pytest.mark.parametrize("d,chunk", [(128, 128), (128, 512), (128, 4096), (256, 128), (256, 256), (256, 257)])
def test_windows_around_the_row_limit_equal_full_run(d, chunk, hq, hkv):
    """128 rows per kv head is the largest window of the short kernel, whose own-chunk items then cover all heads of
    a group; one token more and, with chunks of more than 1024 keys, the 256-row kernel runs.  At head dim 256
    the chunk alone decides between the kernels (256, 257).  Windows cross chunk and sequence boundaries."""
    lens, topk = (700, 5000), 4
    q, k, v, cu = _inputs(lens, hq, hkv, d, chunk, torch.bfloat16, seed=7)
    full, lse, sel = parallel.moba_forward(q, k, v, cu, max(lens), chunk, topk, return_lse=True, return_selected=True)
    limit = 128 // (hq // hkv)
    for begin in (0, 690, 700 + 505, 700 + 4096 - 3, 5700 - limit - 1):
        for n in {1, 2, limit - 1, limit, limit + 1}:
            if n < 1:
                continue
            o, l, s = parallel.moba_forward(q[begin:begin + n], k, v, cu, max(lens), chunk, topk, return_lse=True,
                                            return_selected=True, q_token_begin=begin)
            assert torch.equal(s, sel[:, :, begin:begin + n])
            assert torch.equal(o, full[begin:begin + n]), (begin, n)
            assert torch.equal(l, lse[:, begin:begin + n]), (begin, n)


@pytest.mark.parametrize("hq,hkv", [(4, 4), (6, 2), (8, 1)])
@pytest.mark.parametrize("chunk", [100, 128, 512, 4096])
@pytest.mark.parametrize("d,dtype", [(96, torch.float16), (128, torch.bfloat16)])
def test_decode_windows_of_up_to_eight_rows(d, dtype, chunk, hq, hkv):
    """Windows of at most eight rows per kv head run a kernel with the operands of both products exchanged, one row more the
    kernel for short items: the bits of the full run on either side.  Scores large enough that the reference of a row
    moves from tile to tile; ragged tiles, windows across chunk and sequence boundaries, a list of its own for each row and shared ones."""
    lens, topk = (700, 9001), 6
    q, k, v, cu = _inputs(lens, hq, hkv, d, chunk, dtype, seed=chunk + d)
    q *= 4
    args = (k, v, cu, max(lens), chunk, topk)
    full, lse, sel = parallel.moba_forward(q, *args, return_lse=True, return_selected=True)
    limit = 8 // (hq // hkv)
    for begin in (0, 699, 700 + 505, 700 + 4095, sum(lens) - limit - 1):
        for n in sorted({1, limit, limit + 1}):
            assert _kernel(q[begin:begin + n], *args, begin) == (_lib.KERNEL_FEW_ROWS if n <= limit else _lib.KERNEL_SHORT)
            o, l, s = parallel.moba_forward(q[begin:begin + n], *args, return_lse=True, return_selected=True, q_token_begin=begin)
            assert torch.equal(s, sel[:, :, begin:begin + n])
            assert torch.equal(o, full[begin:begin + n]), (begin, n)
            assert torch.equal(l, lse[:, begin:begin + n]), (begin, n)


def _layouts(t, name):
    """The same values in another memory layout."""
    n, h, d = t.shape
    if name == "fused":                                    # heads of a fused projection: gaps between tokens
        return torch.cat([t, t[:, :1], t[:, :1]], 1)[:, :h]
    if name == "head_major":                               # [H, T, D] storage
        return t.permute(1, 0, 2).contiguous().permute(1, 0, 2)
    if name == "padded_dim":                               # rows longer than head_dim
        return torch.nn.functional.pad(t, (0, 8))[..., :d]
    assert name == "odd_token"                             # a token stride that is no multiple of the head stride
    store = torch.zeros(n * (h * d + 8), dtype=t.dtype, device=t.device)
    view = store.as_strided((n, h, d), (h * d + 8, d, 1))
    view.copy_(t)
    return view


@pytest.mark.parametrize("d", [64, 96, 128])
@pytest.mark.parametrize("layout", ["fused", "head_major", "padded_dim", "odd_token"])
@pytest.mark.parametrize("chunk", [128, 1024, 1025])
def test_layouts_of_q_give_the_same_bits(chunk, layout, d):
    """Forward, a decode-sized window and the gradients read the rows of q by its token and head strides."""
    lens, hq, hkv, topk = (1500, 2100), 4, 2, 3
    q, k, v, cu = _inputs(lens, hq, hkv, d, chunk, torch.bfloat16, seed=3)
    args = (k, v, cu, max(lens), chunk, topk)
    out, lse, sel = parallel.moba_forward(q, *args, return_lse=True, return_selected=True)
    ql = _layouts(q, layout)
    assert torch.equal(ql, q)
    out2, lse2, sel2 = parallel.moba_forward(ql, *args, return_lse=True, return_selected=True)
    assert torch.equal(sel2, sel) and torch.equal(out2, out) and torch.equal(lse2, lse)
    w = parallel.moba_forward(ql[3590:3595], *args, q_token_begin=3590)[0]
    assert torch.equal(w, out[3590:3595])
    g = torch.randn_like(out)
    dq, dk, dv = parallel.moba_backward(q, *args, out, lse, sel, g)
    dq2, dk2, dv2 = parallel.moba_backward(ql, *args, out, lse, sel, g)
    assert torch.equal(dq2, dq)
    # the rows of a list are added in the order of the compaction: fp32 sums, one rounding to bf16
    for a, b in ((dk2, dk), (dv2, dv)):
        assert (a.float() - b.float()).abs().max().item() <= 2.0 ** -7 * b.float().abs().max().item()


@pytest.mark.parametrize("d", [64, 96, 128, 256])
@pytest.mark.parametrize("topk", [1, 9, 16, 17, 33, 64])
def test_merge_of_few_and_many_partials(topk, d):
    """The merge has forms for rows on a part of a warp (few partials, with one sum or the sums of the other form) and
    for rows of a warp, with one or two LSEs in a lane: outputs and LSEs against the merge in float64, on rows that fill no
    block.  A partial is a value of order one at its scale; the result is rounded once to bf16 (2^-9 of values up to 4)
    and the exponentials are good to 2^-22."""
    tokens, hq, hkv, chunk = 333, 6, 2, 16                 # 21 chunks
    rows = tokens * hq
    g = torch.Generator(device="cuda").manual_seed(topk + d)
    q = torch.empty(tokens, hq, d, device="cuda", dtype=torch.bfloat16)
    kv = torch.empty(tokens, hkv, d, device="cuda", dtype=torch.bfloat16)
    cu = torch.tensor([0, tokens], dtype=torch.int32, device="cuda")
    out, lse = torch.empty_like(q), torch.empty(hq, tokens, device="cuda")
    for max_len in (16 * 3, 16 * 11, tokens, 16 * 100):    # partials: the chunks, where top-k allows for more
        prob = parallel.make_problem(q, kv, kv, out, cu, max_len, chunk, topk)
        n = G.dims_of(prob).partials
        assert n == min(topk, -(-max_len // chunk))
        part = torch.randn(rows, n, d, device="cuda", generator=g).half()
        pl = torch.randn(rows, n, device="cuda", generator=g) * 3
        pl[:, 1:][torch.rand(rows, n - 1, device="cuda", generator=g) < 0.3] = -float("inf")    # ranks without a chunk
        inv_scale = torch.exp2(torch.randint(-2, 3, (rows, n), device="cuda", generator=g).float())
        pairs = torch.stack([pl, inv_scale], 2).contiguous()
        _lib.check(_lib.lib().moba_merge(C.byref(prob), part.data_ptr(), pairs.data_ptr(), None, out.data_ptr(),
                                         lse.data_ptr(), G.stream()))
        w = torch.softmax(pl.double(), 1)
        ref = ((w * inv_scale.double())[:, :, None] * part.double()).sum(1)
        err = (out.view(rows, d).double() - ref).abs()
        assert (err <= 2.0 ** -8 * ref.abs() + 2.0 ** -16).all(), err.max().item()
        ref_lse = torch.logsumexp(pl.double(), 1).view(tokens, hq).t()
        assert (lse.double() - ref_lse).abs().max().item() < 1e-5


@pytest.mark.parametrize("d", [64, 96, 128, 256])
@pytest.mark.parametrize("topk", [8, 24, 64])
@pytest.mark.parametrize("tokens", [450, 700, 1100])
def test_rows_do_not_depend_on_the_chunks_max_seqlen_allows_for(tokens, topk, d):
    """A longer max_seqlen only adds ranks that hold no chunk: the same bits, also where top-k exceeds the chunks (8, 11
    and 18 of them here) and the merge adds a row's partials another way."""
    lens, hq, hkv, chunk = (tokens, 150), 4, 2, 64
    q, k, v, cu = _inputs(lens, hq, hkv, d, chunk, torch.bfloat16, seed=topk)
    out, lse, _ = parallel.moba_forward(q, k, v, cu, max(lens), chunk, topk, return_lse=True)
    for longer in (20 * chunk, 100 * chunk):
        out2, lse2, _ = parallel.moba_forward(q, k, v, cu, longer, chunk, topk, return_lse=True)
        assert torch.equal(out2, out) and torch.equal(lse2, lse)


@pytest.mark.parametrize("chunks", [65, 128])
def test_prefix_sums_in_the_gating_kernel_and_apart(chunks):
    """Up to 128 lists (chunks x kv heads of a pass) the gating kernel computes their offsets (calls of many rows), beyond a
    kernel of its own does.  Both heads in one pass have too many for it, one head a pass (a small workspace) has not: the
    same bits, and the chunk selection and values of the oracle on some rows."""
    tokens = 16 * chunks - 5
    q, k, v, cu = _inputs((tokens,), 4, 2, 64, 16, torch.bfloat16, seed=chunks)
    args = (q, k, v, cu, tokens, 16, 3)
    out, lse, sel = parallel.moba_forward(*args, return_lse=True, return_selected=True)
    prob, _ = G.problem_for(q, k, v, cu, tokens, 16, 3)
    least = C.c_size_t()
    _lib.check(_lib.lib().moba_workspace_size_min(C.byref(prob), C.byref(least)))
    out2, lse2, sel2 = parallel.moba_forward(*args, return_lse=True, return_selected=True, workspace_limit=least.value)
    assert torch.equal(sel2, sel) and torch.equal(out2, out) and torch.equal(lse2, lse)
    rows = [(t, h) for t in range(0, tokens, 97) for h in (0, 3)]
    ref, _ = O.attend_rows(q.cpu(), k.cpu(), v.cpu(), cu.cpu().numpy(), tokens, 16, sel.cpu().numpy(), rows)
    got = torch.stack([out[t, h] for t, h in rows])
    _close(got.cpu(), ref, torch.bfloat16)


@pytest.mark.parametrize("chunks", [256, 257])
def test_prefix_sums_of_a_window_of_few_rows(chunks):
    """The line lies at 256 lists for calls of few rows: windows on both sides of it equal the rows of the full run."""
    tokens = 16 * chunks - 5
    q, k, v, cu = _inputs((tokens,), 4, 1, 64, 16, torch.bfloat16, seed=chunks)
    args = (k, v, cu, tokens, 16, 3)
    full, lse, sel = parallel.moba_forward(q, *args, return_lse=True, return_selected=True)
    for begin, n in ((tokens - 1, 1), (2000, 3), (7, 1000)):
        o, l, s = parallel.moba_forward(q[begin:begin + n], *args, return_lse=True, return_selected=True, q_token_begin=begin)
        assert torch.equal(s, sel[:, :, begin:begin + n]) and torch.equal(o, full[begin:begin + n])
        assert torch.equal(l, lse[:, begin:begin + n])


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("d", [64, 96, 128, 256])
@pytest.mark.parametrize("chunk,chunks", [(16, 400), (100, 400), (300, 5), (300, 160)])
def test_chunk_means_of_few_and_many_chunks(chunk, chunks, d, dtype):
    """The mean kernel holds fewer registers when more CTAs come than fit otherwise, and splits long chunks over
    the dims when few do: bit for bit the oracle's means in every form."""
    tokens = chunk * chunks + 1
    _, k, _, cu = _inputs((tokens,), 2, 2, d, chunk, dtype, seed=chunks)
    prob, _ = G.problem_for(k, k, k, cu, tokens, chunk, 3)
    cu_chunk, _, valid, _ = O.chunk_slots(cu.cpu().numpy(), tokens, chunk)
    want = O.chunk_means(k.cpu(), cu_chunk, valid, chunk)
    assert torch.equal(G.means(prob, k, cu).cpu().view(torch.int16), want.view(torch.int16))


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("d", [64, 96, 128, 256])
@pytest.mark.parametrize("chunk", [511, 512, 1025, 2047, 2048, 2049, 4111])
def test_chunk_means_of_one_or_two_long_chunks(chunk, d, dtype):
    """Few long chunks: batches of 64 rows a lane, of 16, then single rows; a chunk whose sequence ends with it has no mean."""
    lens, hkv = (2 * chunk + 1, chunk), 3
    _, k, _, cu = _inputs(lens, hkv, hkv, d, chunk, dtype, seed=chunk)
    prob, _ = G.problem_for(k, k, k, cu, max(lens), chunk, 3)
    cu_chunk, _, valid, _ = O.chunk_slots(cu.cpu().numpy(), max(lens), chunk)
    want = O.chunk_means(k.cpu(), cu_chunk, valid, chunk)
    assert torch.equal(G.means(prob, k, cu).cpu().view(torch.int16), want.view(torch.int16))


@pytest.mark.parametrize("topk", [1, 4])
@pytest.mark.parametrize("chunk", [128, 1024, 1025])
def test_a_call_waits_for_its_inputs_from_another_stream(chunk, topk):
    """The kernels of a call may become resident before the work in front of them is done.  Inputs written on another
    stream, behind a kernel that takes milliseconds, must all the same be there when the first of them reads:
    eagerly behind wait_stream, and captured, where the call follows the join of the two streams."""
    lens, hq, hkv, d = (1500, 2100), 4, 2, 128
    src = [_inputs(lens, hq, hkv, d, chunk, torch.bfloat16, seed=s) for s in (1, 2)]
    want = [parallel.moba_forward(*x, max(lens), chunk, topk)[0] for x in src]
    bufs = [torch.zeros_like(t) for t in src[0][:3]]
    stage = [torch.empty_like(t) for t in src[0][:3]]
    cu = src[0][3]
    main, side = torch.cuda.Stream(), torch.cuda.Stream()

    def call():
        side.wait_stream(main)
        with torch.cuda.stream(side):
            torch.cuda._sleep(6_000_000)                   # about 3 ms
            for b, t in zip(bufs, stage):
                b.copy_(t)
        main.wait_stream(side)
        return parallel.moba_forward(*bufs, cu, max(lens), chunk, topk)[0]

    main.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(main):
        for i in (0, 1):
            for t, x in zip(stage, src[i]):
                t.copy_(x)
            out = call()
            main.synchronize()
            assert torch.equal(out, want[i])
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=main):
        out = call()
    with torch.cuda.stream(main):
        for i in (0, 1):
            for b in bufs:
                b.zero_()
            for t, x in zip(stage, src[i]):
                t.copy_(x)
            graph.replay()
            main.synchronize()
            assert torch.equal(out, want[i])


@pytest.mark.parametrize("layout", ["fused", "head_major", "padded_dim", "odd_token"])
@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("d", [96, 128])
@pytest.mark.parametrize("hq,hkv,topk,n", [(16, 16, 12, 1), (16, 16, 12, 8), (8, 2, 6, 2)])
def test_decode_windows_over_layouts_and_types(hq, hkv, topk, n, d, dtype, layout):
    """The kernel for few rows with more items than SMs (two CTAs on one, three K/V tiles each) and with fewer (six), both types, q in other
    layouts: the bits of the full run on contiguous rows."""
    chunk, total = 128, 4500
    q, k, v, cu = _inputs((total,), hq, hkv, d, chunk, dtype, seed=d + topk)
    args = (k, v, cu, total, chunk, topk)
    out, lse, sel = parallel.moba_forward(q, *args, return_lse=True, return_selected=True)
    ql = _layouts(q, layout)
    assert torch.equal(ql, q)
    for begin in (total - n, 4352 - n // 2):                  # the end of the sequence; across the boundary of a chunk
        w = ql[begin:begin + n]
        assert _kernel(w, *args, begin) == _lib.KERNEL_FEW_ROWS
        o, l, s = parallel.moba_forward(w, *args, return_lse=True, return_selected=True, q_token_begin=begin)
        assert torch.equal(s, sel[:, :, begin:begin + n])
        assert torch.equal(o, out[begin:begin + n]) and torch.equal(l, lse[:, begin:begin + n])


def _same(a, b):
    """Equal, NaN in the same places."""
    return torch.equal(torch.isnan(a), torch.isnan(b)) and torch.equal(a[~torch.isnan(a)], b[~torch.isnan(b)])


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("d", [64, 96, 128])
@pytest.mark.parametrize("where", ["q", "k", "v"])
@pytest.mark.parametrize("value", [float("inf"), float("-inf"), float("nan"), 6e4])
def test_values_that_are_not_finite_on_every_kernel_of_short_chunks(value, where, d, dtype):
    """Infinities, NaN and values whose products overflow the partial rows' or the scores' type, in a row in seven of one input: the
    one-tile kernel, the kernel for short items and (head dims 96 and 128) the one for few rows give the same bits, NaN in the same places."""
    hq, hkv, chunk, topk, total = 8, 4, 128, 5, 4000
    q, k, v, cu = _inputs((total,), hq, hkv, d, chunk, dtype, seed=d)
    g = torch.Generator(device="cuda").manual_seed(d)
    x = {"q": q, "k": k, "v": v}[where]
    hit = torch.rand(x.shape[:2], device="cuda", generator=g) < (1 / 7 if where == "q" else 1 / 200)
    dim = torch.randint(0, d, hit.shape, device="cuda", generator=g)
    x[hit] = x[hit].scatter(1, dim[hit][:, None], value)
    args = (k, v, cu, total, chunk, topk)
    assert _kernel(q, *args) == _lib.KERNEL_ONE_TILE
    out, lse, sel = parallel.moba_forward(q, *args, return_lse=True, return_selected=True)
    if value != 6e4:
        assert not torch.isfinite(out).all()
    assert torch.isfinite(out).any()
    ran = set()
    for begin, n in ((0, 64), (700, 64), (1111, 5), (2048, 4), (2049, 3), (2900, 4), (3991, 2), (3996, 4), (3999, 1)):
        w = q[begin:begin + n]
        ran.add(_kernel(w, *args, begin))
        o, l, s = parallel.moba_forward(w, *args, return_lse=True, return_selected=True, q_token_begin=begin)
        assert torch.equal(s, sel[:, :, begin:begin + n])
        assert _same(o, out[begin:begin + n]) and _same(l, lse[:, begin:begin + n]), (begin, n)
    assert ran == ({_lib.KERNEL_SHORT} if d == 64 else {_lib.KERNEL_SHORT, _lib.KERNEL_FEW_ROWS})


@pytest.mark.parametrize("rows,hq,hkv", [(1, 8, 1), (2, 8, 2), (1, 3, 3)])
@pytest.mark.parametrize("d,dtype", [(96, torch.float16), (128, torch.bfloat16)])
def test_a_list_with_a_row_several_times(d, dtype, rows, hq, hkv):
    """The staged entry points take any selection, also one that names a chunk for several ranks of a row: a list of a decode window is
    then longer than the window has rows per kv head.  Every rank gets its partial result, those of the mma.sync stage."""
    chunk, topk, total = 200, 5, 1500
    q, k, v, cu = _inputs((total,), hq, hkv, d, chunk, dtype, seed=rows + d)
    q = q[-rows:].contiguous()
    out = torch.empty_like(q)
    sel = torch.full((topk - 1, hq, rows), 2, dtype=torch.int32, device="cuda")
    sel[3] = 5                                                # slot 2 three times, slot 5 once
    parts = []
    for impl in (_lib.ATTEND_TCGEN05, _lib.ATTEND_MMA_SYNC):
        prob = parallel.make_problem(q, k, v, out, cu, total, chunk, topk, impl, total - rows)
        dims = G.dims_of(prob)
        assert _lib.lib().moba_problem_attend_kernel(C.byref(prob)) == (
            _lib.KERNEL_FEW_ROWS if impl == _lib.ATTEND_TCGEN05 else _lib.KERNEL_MMA_SYNC)
        counts = torch.zeros(dims.lists, dtype=torch.int32, device="cuda").view(-1, hkv)
        counts[2], counts[5] = 3 * rows * hq // hkv, rows * hq // hkv
        counts = counts.reshape(-1).contiguous()
        offsets, tiles, row_list, plse = G.compact(prob, cu, sel, counts, _lib.lib().moba_problem_tile_rows(C.byref(prob)))
        partial = torch.full((dims.rows * dims.partials, d), 7.0, dtype=torch.float16, device="cuda")
        work = torch.zeros(2, dtype=torch.int32, device="cuda")
        plse.fill_(-9.0)
        _lib.check(_lib.lib().moba_attend(C.byref(prob), q.data_ptr(), k.data_ptr(), v.data_ptr(), cu.data_ptr(), counts.data_ptr(),
                                          offsets.data_ptr(), tiles.data_ptr(), row_list.data_ptr(), partial.data_ptr(),
                                          plse.data_ptr(), work.data_ptr(), G.stream()))
        torch.cuda.synchronize()
        assert work[1].item() == 0
        parts.append((partial.float() * plse[:, 1:], plse[:, 0].clone()))
    (a, la), (b, lb) = parts
    assert (la - lb).abs().max().item() < 1e-3               # scores in fp32, exponentials to 7.5e-5
    _close(a, b, dtype)
    by_rank = a.view(rows * hq, topk, d)
    assert torch.equal(by_rank[:, 1], by_rank[:, 2]) and torch.equal(by_rank[:, 1], by_rank[:, 3])
