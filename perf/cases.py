"""Workloads of the MoBA operator, for timing and for comparing outputs.

A case is one call that a program using this package makes: a prefill of a packed batch
(`parallel_moba`), a training step of the operator (forward and backward through autograd), or an
append to a growing sequence (`IncrementalMoba`: a block of a chunked prefill, or one decode token).
Shapes are those of the package's configurations and benchmark list, and ragged variants of them.
"""
import math

import torch

from baselinebenchmark_b200.incremental import IncrementalMoba
from baselinebenchmark_b200.parallel import parallel_moba


def _case(name, kind, lens, hq, hkv, dim, chunk, topk, dtype="bfloat16", offsets=False, new=0):
    """`lens`: sequence lengths of the batch, as a text; for an append the one prefix length.
    `offsets`: keys carry a per-chunk offset, so that chunks differ in their means.
    `new`: tokens appended behind the prefix."""
    c = {"kind": kind, "lens": lens, "hq": hq, "hkv": hkv, "dim": dim, "chunk": chunk, "topk": topk, "dtype": dtype,
         "offsets": offsets, "new": new}
    return c if name is None else {"name": name, **c}


def listed():
    return [
        # one decode token on a long context (one sequence of the 128K-token serving configuration)
        _case("decode-128k", "append", "131072", 32, 8, 128, 4096, 8, offsets=True, new=1),
        # one decode token of a small head_dim-64 fp16 model, position not on any boundary
        _case("decode-20011-d64", "append", "20011", 16, 4, 64, 512, 8, "float16", True, new=1),
        # one block of a chunked prefill: 700 new tokens behind a ragged prefix
        _case("block-700", "append", "50021", 32, 8, 128, 1024, 8, offsets=True, new=700),
        # a few short requests packed together: latency of one call
        _case("varlen-gqa", "prefill", "200,400,648", 8, 2, 128, 128, 8),
        # the shape most of the benchmark list is built around
        _case("length-4096", "prefill", "4096,4096", 16, 16, 128, 128, 8),
        # ragged batch, fp16, head_dim 64, GQA
        _case("varlen-d64", "prefill", "1023,4097,8191", 16, 4, 64, 128, 8, "float16"),
        # the largest head_dim
        _case("dim-256", "prefill", "4096,4096", 16, 16, 256, 128, 8),
        # long GQA prefill with short chunks
        _case("long-gqa", "prefill", "32768", 32, 8, 128, 128, 8),
        # 32K GQA prefill with long chunks (headline configuration)
        _case("prefill-32k", "prefill", "32768", 32, 8, 128, 4096, 12, offsets=True),
        # one whole sequence of the 128K-token configuration: the largest call
        _case("prefill-128k", "prefill", "131072", 32, 8, 128, 4096, 8, offsets=True),
        # training step on a ragged batch, multi-head, 512-key chunks
        _case("train-varlen", "train", "6144,2560,7168,3584", 32, 32, 128, 512, 3, offsets=True),
        # training step with short chunks, GQA, ragged
        _case("train-c128", "train", "1023,4097,3071", 16, 4, 128, 128, 8),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["decode", "append", "prefill", "prefill", "prefill", "train"])
    hkv = rng.choice([1, 2, 4, 8, 16])
    hq = hkv * rng.choice([1, 2, 4, 8] if hkv <= 4 else [1, 4] if hkv == 8 else [1])
    dim = rng.choice([64, 96, 128, 128, 128, 256])
    dtype = rng.choice(["bfloat16", "bfloat16", "float16"])
    offsets = rng.random() < 0.5
    if kind in ("decode", "append"):
        prefix = _log(rng, 700, 131072)
        chunk = rng.choice([128, 512, 1024, 4096])
        new = 1 if kind == "decode" else _log(rng, 2, 4096)
        return _case(None, "append", str(prefix), hq, hkv, dim, chunk, rng.choice([4, 8, 12, 16]), dtype, offsets, new)
    total = _log(rng, 1000, 65536 if kind == "prefill" else 16384)
    parts = rng.choice([1, 1, 2, 3, 5])
    cuts = sorted(rng.sample(range(1, total), parts - 1))
    lens = ",".join(str(b - a) for a, b in zip([0] + cuts, cuts + [total]))
    chunk = rng.choice([64, 128, 128, 256, 512, 1024, 4096])
    topk = rng.choice([2, 3, 4, 8, 8, 12, 16])
    return _case(None, kind, lens, hq, hkv, dim, chunk, topk, dtype, offsets)


def _lens(case):
    return [int(x) for x in case["lens"].split(",")]


def _tensors(case, seed):
    """q, k, v (and the output gradient of a training step) of all tokens of the case."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    dtype = getattr(torch, case["dtype"])
    lens = _lens(case)
    if case["kind"] == "append":
        lens = [lens[0] + case["new"]]
    total = sum(lens)

    def rand(heads):
        return torch.randn(total, heads, case["dim"], device="cuda", dtype=dtype, generator=g)

    q, k, v = rand(case["hq"]), rand(case["hkv"]), rand(case["hkv"])
    if case["offsets"]:
        at = 0
        for n in lens:
            chunks = -(-n // case["chunk"])
            off = torch.randn(chunks, case["hkv"], case["dim"], device="cuda", generator=g) * 0.5
            k[at:at + n] += off.to(dtype).repeat_interleave(case["chunk"], 0)[:n]
            at += n
    dout = rand(case["hq"]) if case["kind"] == "train" else None
    return lens, q, k, v, dout


def prepare(case, seed):
    lens, q, k, v, dout = _tensors(case, seed)
    if case["kind"] == "append":
        # a sequence whose prefix has been prefilled: K, V and chunk means in the cache
        prefix, new = _lens(case)[0], case["new"]
        cache = IncrementalMoba(prefix + new, case["hkv"], case["dim"], case["chunk"], case["topk"], dtype=q.dtype)
        cache.append(q[:prefix], k[:prefix], v[:prefix])
        return {"kind": "append", "cache": cache, "prefix": prefix,
                "step": tuple(x[prefix:].clone() for x in (q, k, v))}
    cu = torch.tensor([0] + [sum(lens[:i + 1]) for i in range(len(lens))], dtype=torch.int32, device="cuda")
    state = {"kind": case["kind"], "args": (cu, max(lens), case["chunk"], case["topk"]), "dout": dout}
    if case["kind"] == "train":
        q, k, v = (x.requires_grad_() for x in (q, k, v))
    state["qkv"] = (q, k, v)
    return state


def run(state):
    if state["kind"] == "append":
        cache = state["cache"]
        cache.length = state["prefix"]            # back to the end of the prefix: the pass appends the same tokens again
        return cache.append(*state["step"])
    if state["kind"] == "prefill":
        with torch.inference_mode():
            return parallel_moba(*state["qkv"], *state["args"])
    out = parallel_moba(*state["qkv"], *state["args"])
    grads = torch.autograd.grad(out, state["qkv"], state["dout"])
    return (out.detach(), *grads)


def _query_range(case):
    """(sequence lengths, first query position of each sequence)."""
    lens = _lens(case)
    if case["kind"] == "append":
        return [lens[0] + case["new"]], lens[0]
    return lens, 0


def _pairs(n, first, chunk, hist):
    """Visible (query, key) pairs of one head for the queries [first, n) of a sequence of n tokens."""
    total, pos = 0, first
    while pos < n:
        j = pos // chunk
        end = min(n, (j + 1) * chunk)
        a, b = pos - j * chunk + 1, end - j * chunk            # own keys of the first and last query
        total += (a + b) * (end - pos) // 2 + min(hist, j) * chunk * (end - pos)
        pos = end
    return total


def work(case):
    """K and V rows that no query can see, or that no head is expected to select, are not counted."""
    lens, first = _query_range(case)
    hq, hkv, dim, chunk = case["hq"], case["hkv"], case["dim"], case["chunk"]
    hist = case["topk"] - 1
    pairs = sum(_pairs(n, first, chunk, hist) for n in lens)
    queries = sum(n - first for n in lens)
    flops = 4.0 * dim * hq * pairs
    keys = float(sum(lens))
    if case["kind"] == "append":
        # a group's queries pick `hist` of the earlier chunks each, independently of one another
        chunks = first // chunk
        if chunks > 0:
            missed = (1.0 - min(1.0, hist / chunks)) ** (queries * hq // hkv)
            keys = (1.0 - missed) * chunks * chunk + (lens[0] - chunks * chunk)
    moved = 2.0 * dim * (2 * queries * hq + 2 * keys * hkv)    # q, out, k, v
    if case["kind"] == "append":
        moved += 2.0 * dim * hkv * (first // chunk + 2 * queries)          # chunk means, the new K and V rows stored
    if case["kind"] == "train":
        flops *= 3.5
        moved += 2.0 * dim * (4 * queries * hq + 4 * keys * hkv)           # q, out, dout in, dq out; k, v in, dk, dv out
    return {"bytes": moved, "flops": flops}


def tolerance(case):
    # Another implementation of the attention stage at the same precision (P in 16 bits, another summation
    # order) was seen to differ by up to rel 3.1e-3 / max 0.26 in bf16 (one rounding of P and of the output;
    # the largest single difference on a gradient or on an output near zero) and 3.9e-4 / 0.0065 in fp16.
    if case["dtype"] == "bfloat16":
        return {"rel": 1.2e-2, "max": 0.8}
    return {"rel": 1.6e-3, "max": 0.05}


def _select(q, means, own, hist):
    """[tokens, heads, chunks] truth values: the chunks before the own one with the highest scores."""
    hq, hkv = q.shape[1], means.shape[1]
    s = torch.einsum("tghd,cgd->tghc", q.view(q.shape[0], hkv, hq // hkv, -1), means).reshape(q.shape[0], hq, -1)
    s = s.masked_fill(torch.arange(s.shape[2], device=s.device) >= own[:, None, None], -math.inf)
    top = s.topk(min(hist, s.shape[2]), dim=2)
    mask = torch.zeros(s.shape, dtype=torch.bool, device=s.device)
    return mask.scatter_(2, top.indices, top.values > -math.inf)


def exact(case, seed):
    lens, first = _query_range(case)
    hq, hkv, dim, chunk = case["hq"], case["hkv"], case["dim"], case["chunk"]
    if sum(hq * float(n - first) * n for n in lens) > 4e10:   # the dense 64-bit evaluation would take too long
        return None
    train = case["kind"] == "train"
    _, q, k, v, dout = _tensors(case, seed)
    out = torch.empty(sum(n - first for n in lens), hq, dim, dtype=torch.float64, device="cuda")
    dq = torch.zeros_like(out) if train else None
    dk = torch.zeros(k.shape, dtype=torch.float64, device="cuda") if train else None
    dv = torch.zeros_like(dk) if train else None
    at = row = 0
    for n in lens:
        kd, vd = k[at:at + n].double(), v[at:at + n].double()
        whole = max(0, (n - 1) // chunk)                       # chunks that end before the sequence does
        hist = min(case["topk"] - 1, -(-max(lens) // chunk) - 1)
        means = kd[:whole * chunk].view(whole, chunk, hkv, dim).mean(1).to(k.dtype).double() if whole else None
        key = torch.arange(n, device="cuda")
        step = max(1, min(2048, int(3e7) // n))
        for lo in range(first, n, step):
            hi = min(n, lo + step)
            pos = torch.arange(lo, hi, device="cuda")
            qd = q[at + lo:at + hi].double()
            picked = _select(qd, means, pos // chunk, hist) if whole and hist > 0 else None
            span = (pos[:, None] // chunk == key[None, :hi] // chunk) & (key[None, :hi] <= pos[:, None])
            for h in range(hq):
                see = span
                if picked is not None:
                    near = key[:hi] // chunk
                    see = span | (picked[:, h][:, near.clamp(max=whole - 1)] & (near < whole))
                kh, vh = kd[:hi, h // (hq // hkv)], vd[:hi, h // (hq // hkv)]
                p = torch.softmax((qd[:, h] @ kh.T * dim ** -0.5).masked_fill(~see, -math.inf), dim=1)
                o = p @ vh
                out[row + lo - first:row + hi - first, h] = o
                if train:
                    g = dout[at + lo:at + hi, h].double()
                    ds = p * (g @ vh.T - (g * o).sum(1, keepdim=True)) * dim ** -0.5
                    dq[at + lo:at + hi, h] = ds @ kh
                    dk[at:at + hi, h // (hq // hkv)] += ds.T @ qd[:, h]
                    dv[at:at + hi, h // (hq // hkv)] += p.T @ g
        at += n
        row += n - first
    return (out, dq, dk, dv) if train else out
