"""GPU: the gating kernel's two decision paths.

The kernel estimates every score of a row on the tensor core and evaluates in the
contract order (oracle.moba_oracle._tree_dot) only the candidates whose rank the estimate
cannot settle.  Whatever path a row takes, `selected` must equal the oracle's bit for bit;
the statistics output shows how many rows took which path and how far the estimate was
from the exact score relative to the bound the kernel assumes."""
import zlib

import numpy as np
import pytest
import torch

from oracle import moba_oracle as O
from tests import gpu_util as G

pytestmark = pytest.mark.gpu

DTYPES = [pytest.param(torch.bfloat16, id="bf16"), pytest.param(torch.float16, id="fp16")]
NORMAL, FORCE_EXACT, FORCE_RECHECK = 0, 1, 2

# (name, head_dim, seq_lens, Hq, Hkv, chunk, topk)
CASES = [
    ("d128_gqa", 128, (700, 333, 1290), 8, 2, 128, 4),
    ("d128_many_chunks", 128, (4161,), 4, 2, 16, 8),
    ("d128_k64_many_chunks", 128, (4161,), 4, 2, 16, 64),
    ("d64_tail_k64", 64, (513, 2049), 4, 2, 32, 64),
    ("d96_gqa", 96, (127, 128, 129, 900), 8, 2, 64, 5),
    ("d256_mqa", 256, (900,), 4, 1, 64, 8),
    ("g3_odd_group", 128, (1000, 500), 6, 2, 64, 4),
]


def _oracle_selection(q, k, cu, max_seqlen, chunk, topk):
    cu_chunk, _, valid, mc = O.chunk_slots(cu, max_seqlen, chunk)
    hist = O.historical_topk(topk, mc)
    means = O.chunk_means(k, cu_chunk, valid, chunk)
    return means, O.select_chunks(q, means, cu, max_seqlen, chunk, hist)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("case", CASES, ids=lambda c: c[0])
def test_every_decision_path_gives_the_oracle_selection(case, dtype):
    name, d, lens, hq, hkv, chunk, topk = case
    q, k, v, cu = O.make_inputs(list(lens), hq, hkv, d, chunk, zlib.crc32(name.encode()) % 1000, dtype=dtype)
    means_o, sel_o = _oracle_selection(q, k, cu, max(lens), chunk, topk)
    qd, kd = q.cuda(), k.cuda()
    cud = torch.from_numpy(cu).cuda()
    prob, _ = G.problem_for(qd, kd, kd, cud, max(lens), chunk, topk)
    m = G.means(prob, kd, cud)
    assert torch.equal(m.cpu().view(torch.int16), means_o.view(torch.int16))
    rows_with_candidates = sum(max(n - chunk, 0) for n in lens) * hq
    for flags in (NORMAL, FORCE_EXACT, FORCE_RECHECK):
        sel, counts, stats = G.gate_stats(prob, qd, m, cud, flags)
        np.testing.assert_array_equal(sel.cpu().numpy(), sel_o, err_msg=f"flags={flags}")
        assert counts.sum().item() == (sel_o >= 0).sum()
        assert stats[2] == 0, f"estimate outside its bound on {stats[2]} rows (flags={flags})"
        if flags == FORCE_EXACT:
            assert stats[3] == rows_with_candidates and stats[0] == 0
        if flags == FORCE_RECHECK:
            assert stats[0] + stats[3] == rows_with_candidates
            # the tensor-core estimate stays far inside the bound the kernel assumes
            assert stats[1] < 0.25 * 65536, stats
        if flags == NORMAL and topk <= 8:
            # near-ties among a few selected chunks are rare on random inputs: most rows are settled by the
            # estimate (with 63 selected chunks most rows have some pair of scores within the bound)
            assert stats[0] + stats[3] < 0.25 * rows_with_candidates + 64, stats


def _gate_with_means(q, means, lens, chunk, topk, hkv):
    cu = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    mc = O.cdiv(max(lens), chunk)
    hist = O.historical_topk(topk, mc)
    sel_o = O.select_chunks(q, means, cu, max(lens), chunk, hist)
    qd, md = q.cuda(), means.cuda()
    cud = torch.from_numpy(cu).cuda()
    count_o = np.bincount((sel_o.astype(np.int64) * hkv + (np.arange(q.shape[1]) // (q.shape[1] // hkv))[None, :, None])[sel_o >= 0],
                          minlength=(len(cu) - 1) * mc * hkv)
    kdummy = torch.zeros(q.shape[0], hkv, q.shape[2], dtype=q.dtype, device="cuda")
    prob, _ = G.problem_for(qd, kdummy, kdummy, cud, max(lens), chunk, topk)
    out = {}
    for flags in (NORMAL, FORCE_EXACT, FORCE_RECHECK):
        sel, counts, stats = G.gate_stats(prob, qd, md, cud, flags)
        np.testing.assert_array_equal(sel.cpu().numpy(), sel_o, err_msg=f"flags={flags}")
        np.testing.assert_array_equal(counts.cpu().numpy(), count_o, err_msg=f"flags={flags}")
        assert stats[2] == 0
        out[flags] = stats
    return out


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("topk", [8, 64])
def test_exact_ties_and_one_ulp_near_ties_across_many_candidates(dtype, topk):
    """Adversarial means: 300 candidate chunks whose scores tie exactly (identical mean
    vectors), tie in groups, differ in the last bit of one input element, or are all +-0.
    The lower chunk must win every tie and the order of the near-ties must be the contract's."""
    g = torch.Generator().manual_seed(7 + topk)
    chunk, nchunks, hq, hkv, d = 8, 301, 4, 2, 128
    lens = [chunk * nchunks]
    t = lens[0]
    q = torch.randn(t, hq, d, generator=g).to(dtype)
    base = (torch.randn(hkv, d, generator=g) * 0.5).to(dtype)

    # 1. every chunk has the same mean: all scores of a row tie exactly
    same = base[None].repeat(nchunks, 1, 1).contiguous()
    stats = _gate_with_means(q, same, lens, chunk, topk, hkv)
    assert stats[NORMAL][0] + stats[NORMAL][3] > 0.9 * (t - chunk) * hq        # nothing is settled by the estimate

    # 2. five distinct means repeated: ties in groups of sixty
    five = (torch.randn(5, hkv, d, generator=g) * 0.5).to(dtype)
    _gate_with_means(q, five[torch.arange(nchunks) % 5].contiguous(), lens, chunk, topk, hkv)

    # 3. one element one ulp up or down per chunk: scores differ by about 2^-9 |q_i m_i| relative
    bits = same.clone().view(torch.int16)
    dim = torch.randint(0, d, (nchunks,), generator=g)
    step = torch.randint(0, 3, (nchunks,), generator=g).to(torch.int16) - 1
    bits[torch.arange(nchunks), :, dim] += step[:, None]
    _gate_with_means(q, bits.view(dtype), lens, chunk, topk, hkv)

    # 4. zero means of either sign (scores +0.0 and -0.0: +0.0 ranks first, routing.py:778-784)
    zeros = torch.zeros(nchunks, hkv, d, dtype=dtype)
    zeros.view(torch.int16)[1::2] = -32768                                    # -0.0
    _gate_with_means(q, zeros, lens, chunk, topk, hkv)

    # 5. zero query rows mixed in
    q0 = q.clone()
    q0[::3] = 0
    _gate_with_means(q0, bits.view(dtype), lens, chunk, topk, hkv)


@pytest.mark.parametrize("nchunks,topk,d,dtype", [
    (34, 2, 64, torch.float16), (34, 8, 128, torch.bfloat16), (65, 13, 96, torch.bfloat16), (66, 14, 128, torch.float16),
    (129, 29, 64, torch.bfloat16), (130, 8, 256, torch.bfloat16), (257, 12, 128, torch.bfloat16), (258, 28, 128, torch.bfloat16),
    (258, 13, 64, torch.float16)])
def test_more_than_32_candidates_at_the_edges_of_tiles_and_lists(nchunks, topk, d, dtype):
    """Numbers of candidates around those of a tile (64, 128, 256, and two tiles), list lengths around those of
    the networks (16, 32).  Random means, and means whose large scores all lie in one column of each step
    of 32 (every step replaces a place of the list) or rise with the chunk (every step replaces the whole list)."""
    g = torch.Generator().manual_seed(nchunks * 64 + topk)
    chunk, hq, hkv = 8, 4, 2
    lens = [chunk * nchunks, 3 * chunk + 5]
    q = torch.randn(sum(lens), hq, d, generator=g).to(dtype)
    means = (torch.randn(2 * nchunks, hkv, d, generator=g) * 0.5).to(dtype)
    _gate_with_means(q, means, lens, chunk, topk, hkv)
    c = torch.arange(2 * nchunks) % nchunks
    q = (q.abs() + 0.1).to(dtype)
    hot = torch.where(c % 32 == 5, 1.0 + c / 1000.0, 0.01 * (c % 7))
    _gate_with_means(q, (means.float().abs() * hot[:, None, None]).to(dtype), lens, chunk, topk, hkv)
    _gate_with_means(q, ((0.1 + c / 100.0)[:, None, None] * (1 + means.float().abs())).to(dtype), lens, chunk, topk, hkv)


def _adversarial_means(nchunks, hkv, d, dtype, g):
    """(what the scores of a row do, means of the chunks)."""
    base = (torch.randn(hkv, d, generator=g) * 0.5).to(dtype)
    same = base[None].repeat(nchunks, 1, 1).contiguous()
    yield "all tie", same
    five = (torch.randn(5, hkv, d, generator=g) * 0.5).to(dtype)
    yield "tie in groups", five[torch.arange(nchunks) % 5].contiguous()
    bits = same.clone().view(torch.int16)
    bits[torch.arange(nchunks), :, torch.randint(0, d, (nchunks,), generator=g)] += \
        torch.randint(-1, 2, (nchunks, 1), generator=g).to(torch.int16)
    yield "one ulp of one element apart", bits.view(dtype)
    half = (torch.randn(nchunks, hkv, d, generator=g) * 0.5).to(dtype)
    half[::2] = bits.view(dtype)[::2]
    yield "runs of near-ties between others", half
    zeros = torch.zeros(nchunks, hkv, d, dtype=dtype)
    zeros.view(torch.int16)[1::2] = -32768                                    # -0.0
    yield "zeros of either sign", zeros
    at = torch.arange(nchunks)
    for value in (float("inf"), float("nan")):
        some = (torch.randn(nchunks, hkv, d, generator=g) * 0.5).to(dtype)
        some[at[2::4], :, torch.randint(0, d, (nchunks,), generator=g)[2::4]] = value
        if value == float("inf"):
            some[at[1::4], :, 3] = -value
        yield f"some {value}", some


@pytest.mark.parametrize("d,dtype", [(64, torch.float16), (96, torch.bfloat16), (128, torch.bfloat16), (128, torch.float16),
                                     (256, torch.bfloat16)])
@pytest.mark.parametrize("nchunks,topk", [(2, 2), (2, 8), (9, 2), (9, 8), (9, 17), (31, 17), (32, 8), (32, 9), (32, 32),
                                          (33, 2), (33, 8), (33, 9), (33, 16), (33, 17), (33, 31), (33, 32), (33, 33)])
def test_at_most_32_candidates_ties_zeros_infinities(nchunks, topk, d, dtype):
    """The kernel for rows of at most 32 candidates (33 chunks), which decides in registers: every width of its
    network (lists of 8, 16 and 32) from both sides, and with lists of 33 the other kernel.  A call of at most 16 row
    tiles runs it at every width, a larger one the other kernel at widths where that is ahead.  Infinite and NaN
    scores rank by their bits (NaN of positive sign here, above +inf), equal ones by the chunk."""
    chunk = 8
    _few_candidates([chunk * nchunks], 2, 1, nchunks, topk, d, dtype)
    _few_candidates([chunk * nchunks, chunk - 1, chunk * (nchunks // 2) + 3], 4, 4, nchunks, topk, d, dtype)


@pytest.mark.parametrize("d,dtype", [(64, torch.float16), (128, torch.bfloat16), (256, torch.bfloat16)])
@pytest.mark.parametrize("nchunks,topk", [(34, 2), (34, 8), (40, 17), (66, 8), (129, 12), (129, 30), (300, 8)])
def test_more_than_32_candidates_ties_zeros_infinities(nchunks, topk, d, dtype):
    """The same where a row's list goes through several steps of 32 candidates: the networks compare the estimates as floats,
    which drop NaN; rows with a score that is not finite are ranked over all their candidates."""
    chunk = 8
    _few_candidates([chunk * nchunks], 2, 1, nchunks, topk, d, dtype)
    _few_candidates([chunk * nchunks, chunk - 1, chunk * (nchunks // 2) + 3], 4, 4, nchunks, topk, d, dtype)


def _few_candidates(lens, hq, hkv, nchunks, topk, d, dtype):
    chunk, slots = 8, len(lens) * nchunks
    g = torch.Generator().manual_seed(nchunks * 64 + topk)
    q = torch.randn(sum(lens), hq, d, generator=g).to(dtype)
    q[q == 0] = 1                                                             # (inf * 0)
    for what, means in _adversarial_means(slots, hkv, d, dtype, g):
        _gate_with_means(q, means, lens, chunk, topk, hkv)
        if what.startswith("one ulp"):
            q0 = q.clone()
            q0[::3] = 0
            _gate_with_means(q0, means, lens, chunk, topk, hkv)
    finite = (torch.randn(slots, hkv, d, generator=g) * 0.5).to(dtype)
    finite[finite == 0] = 1
    _gate_with_means(q, finite, lens, chunk, topk, hkv)
    for value in (float("inf"), float("nan")):
        q1 = q.clone()
        q1[::5, 1, 7] = value
        _gate_with_means(q1, finite, lens, chunk, topk, hkv)


@pytest.mark.parametrize("d", [64, 96, 128, 256])
@pytest.mark.parametrize("topk", [5, 8, 12, 24])
def test_at_most_32_candidates_many_tiles_of_rows(topk, d):
    """Enough tiles of rows that every CTA takes several: tiles with and without candidates, tiles beyond the end of their
    sequence and sequences shorter than a chunk follow one another in it.  (Lists of more than 8 run the kernel for
    any number of candidates here, without its scratch for a second step of 32.)"""
    g = torch.Generator().manual_seed(topk)
    chunk, hq, hkv = 8, 16, 4
    lens = [(264, 3, 130, 7, 8, 9, 40, 1)[(i + i // 8) % 8] for i in range(56)]
    tiles = len(lens) * hkv * -(-264 // (128 // (hq // hkv)))
    assert tiles >= 3 * 148 * 4
    q = torch.randn(sum(lens), hq, d, generator=g).to(torch.bfloat16)
    means = (torch.randn(33 * len(lens), hkv, d, generator=g) * 0.5).to(torch.bfloat16)
    means[::3] = means[0]                                                     # ties in every sequence
    _gate_with_means(q, means, lens, chunk, topk, hkv)


def test_long_candidate_lists_sampled():
    """More candidates than one tensor-core tile holds (625 > 256), top-k 8 and 64, against the
    oracle on sampled tokens; all three decision paths."""
    lens, hq, hkv, chunk = [40000], 4, 2, 64
    q, k, v, cu = O.make_inputs(lens, hq, hkv, 128, chunk, seed=99)
    cu_chunk, _, valid, mc = O.chunk_slots(cu, lens[0], chunk)
    means_o = O.chunk_means(k, cu_chunk, valid, chunk)
    rng = np.random.default_rng(5)
    rows = sorted(set(rng.integers(0, lens[0], 600).tolist()) | {63, 64, 65, 16383, 16384, 16447, 39999})
    qd, kd = q.cuda(), k.cuda()
    cud = torch.from_numpy(cu).cuda()
    for topk in (8, 64):
        hist = O.historical_topk(topk, mc)
        sel_o = O.select_chunks(q, means_o, cu, lens[0], chunk, hist, rows=rows)
        prob, _ = G.problem_for(qd, kd, kd, cud, lens[0], chunk, topk)
        m = G.means(prob, kd, cud)
        for flags in (NORMAL, FORCE_RECHECK, FORCE_EXACT):
            sel, _, stats = G.gate_stats(prob, qd, m, cud, flags)
            np.testing.assert_array_equal(sel.cpu().numpy()[:, :, rows], sel_o[:, :, rows], err_msg=f"{topk} {flags}")
            assert stats[2] == 0
