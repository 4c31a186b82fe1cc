"""GPU: IncrementalMoba.append takes K and V rows in any layout, whichever way they reach the cache - copied by
the native call (same type, rows of 16-byte pieces) or by torch (everything else): the caches and the
results are the same bits."""
import pytest
import torch

from baselinebenchmark_b200.incremental import IncrementalMoba

pytestmark = pytest.mark.gpu


def _rows(t, how):
    n, h, d = t.shape
    if how == "fused":                       # heads of a fused projection: native, with strides
        return torch.cat([t, t], 1)[:, :h], True
    if how == "odd_stride":                  # token stride of no whole 16-byte pieces: torch
        store = torch.zeros(n * (h * d + 4), dtype=t.dtype, device=t.device)
        view = store.as_strided((n, h, d), (h * d + 4, d, 1))
        return view.copy_(t), False
    if how == "float32":                     # converted on the way: torch
        return t.float(), False
    if how == "expanded":                    # one head for all: torch (the row shape differs)
        return t[:, :1], False
    return t, True


@pytest.mark.parametrize("n", [1, 3, 200])
@pytest.mark.parametrize("how", ["contiguous", "fused", "odd_stride", "float32", "expanded"])
def test_rows_of_any_layout_reach_the_cache(how, n):
    hq, hkv, d, chunk, topk, prefix = 8, 2, 128, 256, 3, 1000
    g = torch.Generator(device="cuda").manual_seed(5)
    q, k, v = (torch.randn(prefix + n, h, d, device="cuda", dtype=torch.bfloat16, generator=g) for h in (hq, hkv, hkv))
    if how == "expanded":
        k[prefix:] = k[prefix:, :1]
        v[prefix:] = v[prefix:, :1]
    caches = []
    for layout in ("contiguous", how):
        inc = IncrementalMoba(prefix + 300, hkv, d, chunk, topk)
        inc.append(q[:prefix], k[:prefix], v[:prefix])
        (kn, native), (vn, _) = _rows(k[prefix:], layout), _rows(v[prefix:], layout)
        assert inc._plain(kn, vn) == native
        out, sel = inc.append(q[prefix:], kn, vn, return_selected=True)
        caches.append((out, sel, inc.k[:prefix + n].clone(), inc.v[:prefix + n].clone(), inc.means.clone(), inc.cu.clone()))
        assert inc.length == prefix + n
    for a, b in zip(*caches):
        assert torch.equal(a, b)


@pytest.mark.parametrize("native", [True, False])
def test_append_counts_as_an_in_place_write(native):
    """Autograd must notice that what it saved of the caches has been overwritten, whichever way the rows went."""
    inc = IncrementalMoba(64, 2, 64, 16, 3)
    rows = torch.randn(4, 2, 64, device="cuda", dtype=torch.bfloat16 if native else torch.float32)
    q = torch.randn(4, 4, 64, device="cuda", dtype=torch.bfloat16)
    assert inc._plain(rows, rows) == native
    scale = torch.ones(1, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    sums = [(scale * c).sum() for c in (inc.k, inc.v)]       # saves the cache for the gradient of `scale`
    inc.append(q, rows, rows)
    for s in sums:
        with pytest.raises(RuntimeError, match="modified by an inplace operation"):
            s.backward()
