"""CPU: which kernel of the dense stage a problem runs, on both sides of each line of the rules.  All of them give the same
bits, so that no comparison of outputs would notice a rule that sends everything to one of them."""
import ctypes as C

import pytest

from baselinebenchmark_b200 import _lib, build

ROWS_256, SHORT, ONE_TILE, FEW, WIDE, WIDE_SHORT = (
    _lib.KERNEL_ROWS_256, _lib.KERNEL_SHORT, _lib.KERNEL_ONE_TILE, _lib.KERNEL_FEW_ROWS, _lib.KERNEL_WIDE,
    _lib.KERNEL_WIDE_SHORT)


@pytest.fixture(scope="module")
def lib():
    build.build()
    return _lib.lib()


def _kernel(lib, lens, hq, hkv, dim, chunk, topk, new=0, impl=0, q_strides=None):
    """`lens`: tokens of one sequence or of each of a batch; `new`: the last tokens of the call are the queries."""
    lens = lens if isinstance(lens, tuple) else (lens,)
    total = sum(lens)
    sq = q_strides or (hq * dim, dim)
    p = _lib.Problem(total, len(lens), hq, hkv, dim, max(lens), chunk, topk, impl, *sq, hkv * dim, dim, hkv * dim, dim,
                     hq * dim, dim, total - new if new else 0, new, 0, 0)
    return lib.moba_problem_attend_kernel(C.byref(p))


@pytest.mark.parametrize("dim", [64, 96, 128])
def test_long_sequences_by_chunk(lib, dim):
    one = lambda chunk, topk=8: _kernel(lib, 20000, 16, 4, dim, chunk, topk)
    assert [one(c) for c in (95, 96, 127, 128, 129)] == [ONE_TILE if dim == 64 else SHORT, ONE_TILE, ONE_TILE, ONE_TILE, SHORT]
    assert one(64) == (ONE_TILE if dim == 64 else SHORT) and one(64, 7) == SHORT and one(63, 9) == SHORT
    assert one(512) == SHORT and one(4096) == ROWS_256
    # three tiles a list: ranks x chunk x heads of a group
    lists = lambda topk, hkv: _kernel(lib, 20000, 16, hkv, dim, 128, topk)
    assert [lists(k, 16) for k in (3, 4)] == [SHORT, ONE_TILE] and lists(2, 4) == ONE_TILE


def test_the_other_implementations(lib):
    assert _kernel(lib, 20000, 16, 4, 128, 128, 8, impl=1) == _lib.KERNEL_MMA_SYNC
    assert [_kernel(lib, 20000, 16, 4, 256, c, 8) for c in (256, 257)] == [WIDE_SHORT, WIDE]
    assert _kernel(lib, 20000, 16, 4, 256, 128, 8, new=1) == WIDE_SHORT
    assert _kernel(lib, 0, 16, 4, 128, 128, 8) < 0                       # refused, like by every entry point


def test_small_windows(lib):
    for dim in (96, 128):
        assert [_kernel(lib, 50000, 16, 4, dim, 128, 8, new=n) for n in (1, 2, 3)] == [FEW, FEW, SHORT]
        assert [_kernel(lib, 50000, 8, 1, dim, 4096, 8, new=n) for n in (1, 2, 16, 17)] == [FEW, SHORT, SHORT, ROWS_256]
    assert _kernel(lib, 50000, 16, 4, 64, 128, 8, new=1) == SHORT
    # a window of more than one tile of rows per kv head, on a prefix short enough for full lists
    assert [_kernel(lib, 1000, 16, 2, 128, 128, 8, new=n) for n in (16, 200)] == [SHORT, ONE_TILE]


@pytest.mark.parametrize("lens,hq,hkv,dim,chunk,topk,new", [
    (51000, 16, 16, 128, 128, 8, 1000), (50300, 16, 4, 128, 128, 8, 300), (25502, 8, 8, 128, 128, 4, 1254),
    (20800, 16, 8, 128, 128, 16, 1195), (36099, 16, 2, 128, 128, 2, 283), (6772, 16, 4, 128, 128, 6, 61)])
def test_windows_behind_a_long_prefix_have_few_rows_a_list(lib, lens, hq, hkv, dim, chunk, topk, new):
    assert _kernel(lib, lens, hq, hkv, dim, chunk, topk, new) == SHORT
    assert _kernel(lib, lens, hq, hkv, dim, chunk, topk) == ONE_TILE     # all tokens queries


def test_batches_of_short_sequences_have_few_rows_a_list(lib):
    assert _kernel(lib, (100,) * 30, 8, 2, 128, 96, 8) == SHORT
    assert _kernel(lib, (410,) * 50, 16, 16, 128, 96, 8) == SHORT
    assert _kernel(lib, (146,) * 42, 32, 8, 128, 96, 3) == SHORT
    assert _kernel(lib, (800,) * 45, 16, 16, 128, 96, 12) == ONE_TILE
    assert _kernel(lib, (563,) * 9, 32, 16, 128, 128, 4) == ONE_TILE
    # so few items that an SM has one or none: whatever the lists
    assert [_kernel(lib, 512, h, h, 128, 128, 4) for h in (4, 8, 9, 16)] == [ONE_TILE, ONE_TILE, SHORT, SHORT]
    # head dim 64, chunks of 64 keys with seven ranks
    assert _kernel(lib, 20000, 16, 16, 64, 64, 8) == ONE_TILE and _kernel(lib, (400,) * 50, 16, 16, 64, 64, 8) == SHORT
    # the workloads of the benchmark list
    assert _kernel(lib, (4096, 4096), 16, 16, 128, 128, 8) == ONE_TILE
    assert _kernel(lib, (1023, 4097, 8191), 16, 4, 64, 128, 8) == ONE_TILE
    assert _kernel(lib, 32768, 32, 8, 128, 128, 8) == ONE_TILE


def test_row_offsets_of_32_bits(lib):
    """The one-tile kernel keeps row offsets in 16-byte pieces of 32 bits: 2^35 elements of q at most."""
    edge = lambda stride: _kernel(lib, 20001, 16, 4, 128, 128, 8, q_strides=(stride, 128))
    most = ((1 << 35) - 15 * 128 - 1) // 20000 // 8 * 8
    assert edge(most) == ONE_TILE and edge(most + 8) == SHORT
