"""GPU: a caller of the C ABI that makes another context of the device current.

A kernel's shared memory limit belongs to the context its module is loaded in.  The child process (no torch in it: nothing else
holds contexts there) runs forwards and backwards over the kernels of each stage in the primary context, in a second context and in the
first again, on fp16 data, and prints one JSON line of return codes and of whether the results agree."""
import json
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parent.parent

CHILD = r'''
import ctypes as C, json
import numpy as np
from baselinebenchmark_b200 import _lib

cuda, lib = C.CDLL("libcuda.so.1"), _lib.lib()
def cu(name, *args):
    rc = getattr(cuda, name)(*args)
    if rc != 0:
        raise RuntimeError(f"{name}: {rc}")

# head dim, chunk, implementation: every kernel of the dense stage, of dq and of dk/dv
CASES = [(128, 128, 0), (128, 512, 0), (128, 2048, 0), (64, 256, 0), (256, 128, 0), (256, 512, 0), (128, 512, 1), (256, 512, 1)]
TOKENS, HQ, HKV, TOPK = 3000, 8, 2, 4

def run(dim, chunk, impl):
    rng = np.random.default_rng(chunk + dim)
    q, k, v, dout = (rng.standard_normal((TOKENS, h, dim)).astype(np.float16) for h in (HQ, HKV, HKV, HQ))
    hist = min(TOPK - 1, -(-TOKENS // chunk) - 1)
    p = _lib.Problem(TOKENS, 1, HQ, HKV, dim, TOKENS, chunk, TOPK, impl, *[HQ * dim, dim], *[HKV * dim, dim] * 2, HQ * dim, dim,
                     0, 0, 1, 0)
    held = []
    def dev(x=None, nbytes=0):
        ptr = C.c_uint64(0)
        cu("cuMemAlloc_v2", C.byref(ptr), C.c_size_t(x.nbytes if x is not None else max(nbytes, 16)))
        if x is not None:
            cu("cuMemcpyHtoD_v2", ptr, x.ctypes.data_as(C.c_void_p), C.c_size_t(x.nbytes))
        held.append(ptr)
        return ptr.value
    def host(ptr, like):
        x = np.empty_like(like)
        cu("cuMemcpyDtoH_v2", x.ctypes.data_as(C.c_void_p), C.c_uint64(ptr), C.c_size_t(x.nbytes))
        return x
    need, back = C.c_size_t(0), C.c_size_t(0)
    codes = [lib.moba_workspace_size(C.byref(p), C.byref(need)), lib.moba_backward_workspace_size(C.byref(p), C.byref(back))]
    dq, dk, dv, dd = (dev(x) for x in (q, k, v, dout))
    cu_seqlens = dev(np.array([0, TOKENS], dtype=np.int32))
    out, lse, sel = dev(nbytes=q.nbytes), dev(nbytes=4 * HQ * TOKENS), dev(nbytes=4 * hist * HQ * TOKENS)
    ws, wb = dev(nbytes=need.value), dev(nbytes=back.value)
    codes.append(lib.moba_forward(C.byref(p), dq, dk, dv, cu_seqlens, out, lse, sel, ws, need.value, None))
    grads = [dev(nbytes=x.nbytes) for x in (q, k, v)]
    codes.append(lib.moba_backward(C.byref(p), dq, dk, dv, cu_seqlens, out, lse, sel, dd, *grads, wb, back.value, None))
    cu("cuCtxSynchronize")
    results = [host(out, q)] + [host(g, x) for g, x in zip(grads, (q, k, v))]
    for ptr in held:
        cu("cuMemFree_v2", ptr)
    return codes, results

cu("cuInit", 0)
device, first, second = C.c_int(0), C.c_void_p(), C.c_void_p()
cu("cuDeviceGet", C.byref(device), 0)
cu("cuDevicePrimaryCtxRetain", C.byref(first), device)
cu("cuCtxSetCurrent", first)
want = [run(*c) for c in CASES]
cu("cuCtxCreate_v2", C.byref(second), 0, device)
got = [run(*c) for c in CASES]
cu("cuCtxDestroy_v2", second)
cu("cuCtxSetCurrent", first)
again = [run(*c) for c in CASES]

def close(a, b):
    a, b = a.astype(np.float64), b.astype(np.float64)
    return bool(np.linalg.norm(a - b) <= 2e-3 * np.linalg.norm(b))   # order of the rows of a list: sums in another order
report = []
for case, (c0, r0), (c1, r1), (c2, r2) in zip(CASES, want, got, again):
    report.append({"case": case, "codes": [c0, c1, c2], "out": bool(np.array_equal(r0[0], r1[0]) and np.array_equal(r0[0], r2[0])),
                   "grads": all(close(x, y) for r in (r1, r2) for x, y in zip(r[1:], r0[1:]))})
print(json.dumps(report))
'''


def test_calls_in_a_second_context():
    res = subprocess.run([sys.executable, "-c", CHILD], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert res.returncode == 0, res.stderr[-2000:]
    for r in json.loads(res.stdout.splitlines()[-1]):
        assert r["codes"] == [[0] * 4] * 3, r
        assert r["out"] and r["grads"], r
