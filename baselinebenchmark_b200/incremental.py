"""Incremental prefill and decode of ONE growing sequence on top of `moba_forward_cached`.

The reference's MoBA operator has no incremental mode: `parallel_moba` takes whole sequences
and recomputes every chunk mean on each call (backends/_mthreads/ops/moba/parallel.py:306-311).
Here the K/V rows, the chunk means and the position live on the device between calls; a call
appends any number of tokens - a prefill block or a single decode token - and returns their
attention rows, which equal the rows of a one-shot run over the final sequence bit for bit
(a query only sees keys at or before its own position, and a chunk's mean only its own keys).
"""
import ctypes as C
from typing import Optional

import torch

from . import _lib, parallel


class IncrementalMoba:
    """K/V cache of one sequence with cached chunk means.

    `capacity` tokens of K and V ([capacity, Hkv, D]) and ceil(capacity / chunk) chunk means are
    allocated once.  `append(q, k, v)` stores the new K/V rows behind the `length` tokens already
    there and runs the operator on the query window [length, length + n) over the prefix; the
    means of chunks completed by earlier calls are read from the cache, the others recomputed.
    Nothing is read back to the host: the position is kept on both sides."""

    def __init__(self, capacity: int, num_kv_heads: int, head_dim: int, moba_chunk_size: int, moba_topk: int,
                 dtype: torch.dtype = torch.bfloat16, device: Optional[torch.device] = None,
                 attend_impl: Optional[int] = None):
        if capacity <= 0:
            raise ValueError(f"capacity must be positive, got {capacity}")
        device = torch.device("cuda", torch.cuda.current_device()) if device is None else torch.device(device)
        self.capacity, self.chunk, self.topk, self.attend_impl = capacity, moba_chunk_size, moba_topk, attend_impl
        self.k = torch.empty(capacity, num_kv_heads, head_dim, dtype=dtype, device=device)
        self.v = torch.empty_like(self.k)
        slots = (capacity + moba_chunk_size - 1) // moba_chunk_size
        self.means = torch.zeros(slots, num_kv_heads, head_dim, dtype=dtype, device=device)
        self.cu = torch.zeros(2, dtype=torch.int32, device=device)
        self.length = 0

    def reset(self) -> None:
        self.length = 0

    def append(self, q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, return_selected: bool = False):
        """q [n, Hq, D], k / v [n, Hkv, D]: the next n >= 1 tokens.  Returns their rows [n, Hq, D];
        with `return_selected` also the chunks they selected, (out, selected[hist, Hq, n] int32)."""
        n, begin = q.shape[0], self.length
        if k.shape[0] != n or v.shape[0] != n:
            raise ValueError(f"q, k and v must hold the same number of new tokens, got {n}, {k.shape[0]}, {v.shape[0]}")
        if n == 0 or begin + n > self.capacity:
            raise ValueError(f"cannot append {n} tokens at position {begin} of a cache of {self.capacity}")
        end = begin + n
        # a call on a prefix of `begin` tokens left final means in the slots of all chunks but the
        # prefix's last one (the last chunk of a sequence is no candidate and is not computed)
        cached = (begin - 1) // self.chunk if begin > 0 else 0
        if self._plain(k, v):
            out, sel = self._append(q, k, v, begin, end, cached, return_selected)
        else:
            self.k[begin:end].copy_(k)
            self.v[begin:end].copy_(v)
            self.cu[1:].fill_(end)
            out, _, sel = parallel.moba_forward(q, self.k[:end], self.v[:end], self.cu, self.capacity, self.chunk,
                                                self.topk, attend_impl=self.attend_impl, q_token_begin=begin,
                                                means_cache=self.means, cached_slots=cached,
                                                return_selected=return_selected)
        self.length = end
        return (out, sel) if return_selected else out

    def _plain(self, k: torch.Tensor, v: torch.Tensor) -> bool:
        """Rows that moba_append copies as they are: the caches' type, device and row shape, 16-byte pieces, memory
        of their own, and nothing for autograd to record.  Everything else goes through torch's copy."""
        kc, vc, cu = self.k, self.v, self.cu               # each attribute read once: this runs on every call
        if kc.requires_grad or vc.requires_grad:
            return False
        # torch refuses to write an inference tensor outside inference mode: leave that to its copy
        if (kc.is_inference() or vc.is_inference() or cu.is_inference()) and not torch.is_inference_mode_enabled():
            return False
        (size, heads, dim), dtype, device = kc.shape, kc.dtype, kc.device
        (k0, k1, _), (v0, v1, _), k_at, v_at = kc.stride(), vc.stride(), kc.data_ptr(), vc.data_ptr()
        k_end = k_at + 2 * ((size - 1) * k0 + (heads - 1) * k1 + dim)
        v_end = v_at + 2 * ((size - 1) * v0 + (heads - 1) * v1 + dim)
        for t in (k, v):
            shape = t.shape
            if len(shape) != 3 or shape[1] != heads or shape[2] != dim or t.dtype != dtype or t.device != device or t.requires_grad:
                return False
            (s0, s1, s2), at = t.stride(), t.data_ptr()
            if s2 != 1 or s0 % 8 or s1 % 8 or at % 16:
                return False
            # One kernel reads the rows and writes both caches: rows that share memory with either of them go
            # through torch, one cache after the other.
            end = at + 2 * ((shape[0] - 1) * s0 + (heads - 1) * s1 + dim)
            if at < k_end and k_at < end or at < v_end and v_at < end:
                return False
        return True

    def _append(self, q, k, v, begin: int, end: int, cached: int, return_selected: bool):
        """One native call: rows into the caches, position, attention on the new tokens."""
        kc, vc = self.k, self.v
        parallel._validate(q, kc, vc, self.cu, self.capacity, self.chunk, self.topk, windowed=True)
        out = torch.empty(q.shape, dtype=q.dtype, device=q.device)
        prob = parallel.make_problem(q, kc, vc, out, self.cu, self.capacity, self.chunk, self.topk, self.attend_impl, begin)
        prob.total_tokens = end
        need = parallel.workspace_bytes(prob)
        ws = parallel._workspace(q.device, need)
        sel = None
        if return_selected:
            hist = parallel._hist(self.capacity, self.chunk, self.topk)
            sel = torch.empty((hist, q.shape[1], q.shape[0]), dtype=torch.int32, device=q.device)
        lib = _lib.lib()
        (kt, kh, _), (vt, vh, _) = k.stride(), v.stride()
        _lib.check(parallel._on_device(q.device, lambda stream: lib.moba_append(
            C.byref(prob), q.data_ptr(), k.data_ptr(), v.data_ptr(), kt, kh, vt, vh, kc.data_ptr(), vc.data_ptr(),
            self.cu.data_ptr(), out.data_ptr(), sel.data_ptr() if sel is not None and sel.numel() else None,
            self.means.data_ptr(), cached, ws.data_ptr(), need, stream)))
        # what autograd saved of the caches is stale now, as after an in-place torch operation
        torch.autograd.graph.increment_version((kc, vc, self.cu))
        return out, sel
