"""CPU: which rows IncrementalMoba.append hands to the native copy.  (The rule looks at the tensors only, so a cache
on the CPU stands in for one on the device.)"""
import pytest
import torch

from baselinebenchmark_b200.incremental import IncrementalMoba

N, HKV, DIM = 4, 2, 64


def _cache(store=None):
    inc = IncrementalMoba(64, HKV, DIM, 16, 3, device=torch.device("cpu"))
    if store is not None:                    # caches that are parts of one larger buffer
        inc.k, inc.v = store[:64], store[64:128]
    return inc


def _rows():
    return torch.zeros(N, HKV, DIM, dtype=torch.bfloat16)


def test_rows_of_their_own_are_copied_natively():
    inc = _cache()
    assert inc._plain(_rows(), _rows())
    fused = torch.zeros(N, 2 * HKV, DIM, dtype=torch.bfloat16)
    assert inc._plain(fused[:, :HKV], fused[:, HKV:])


@pytest.mark.parametrize("cache", ["k", "v"])
@pytest.mark.parametrize("side", ["k", "v"])
@pytest.mark.parametrize("start", [0, 9, 10, 11])
def test_rows_of_either_cache_are_not(side, cache, start):
    """The native copy reads the rows of both sides while it writes both caches (here at rows 10-13)."""
    inc = _cache()
    inc.length = 10
    rows = getattr(inc, cache)[start:start + N]
    assert not inc._plain(rows, _rows()) if side == "k" else not inc._plain(_rows(), rows)


def test_rows_that_start_before_the_cache_and_run_into_it_are_not():
    store = torch.zeros(130, HKV, DIM, dtype=torch.bfloat16)
    inc = _cache(store[2:])
    assert not inc._plain(store[:N], _rows()) and not inc._plain(_rows(), store[:N])


@pytest.mark.parametrize("part", ["k", "v", "cu"])
def test_inference_tensors_outside_inference_mode_are_left_to_torch(part):
    """torch's in-place copy refuses them there; inside inference mode it does not."""
    inc = _cache()
    with torch.inference_mode():
        setattr(inc, part, torch.zeros_like(getattr(inc, part)))
        assert inc._plain(_rows(), _rows())
    assert not inc._plain(_rows(), _rows())
    with pytest.raises(RuntimeError, match="[Ii]nference"):
        inc.append(torch.zeros(N, HKV, DIM, dtype=torch.bfloat16), _rows(), _rows())
    assert inc.length == 0
