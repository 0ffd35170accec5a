"""Thin torch-tensor wrappers over the C ABI (one function per entry point)."""

import collections
import ctypes
import functools
import math

import torch

from . import _lib
from ._lib import check, ptr, stream_ptr


class DeviceStatus:
    """One int32 in device memory that kernels set when a bounded wait or capacity check
    fails.  ``raise_if_set`` synchronises and raises; call it where a sync is acceptable."""

    NAMES = {1: "TMA wait timed out", 2: "MMA wait timed out", 3: "consumer wait timed out",
             4: "sort scratch too small", 5: "segment pool exhausted", 6: "self-test timeout"}

    def __init__(self, device):
        self.word = torch.zeros(1, dtype=torch.int32, device=device)

    def read(self):
        return int(self.word.item())

    def clear(self):
        self.word.zero_()

    def raise_if_set(self, what="kernel"):
        code = self.read()
        if code != 0:
            self.clear()
            raise _lib.StacError(f"{what}: device error {code} ({self.NAMES.get(code, 'unknown')})")


class LaggedInts:
    """Device int32 values mirrored on the host WITHOUT a synchronisation at the producing call:
    ``push`` enqueues copies into pinned host memory on the current stream and records an event;
    ``pull`` is made by the NEXT call that needs the numbers, by which time that event lies a
    whole stream step in the past, so waiting for it does not stall a host that runs at most
    one step ahead of the GPU.  ``pull`` returns None when nothing is pending."""

    def __init__(self, n):
        _free_dropped()
        self.pin = torch.zeros(n, dtype=torch.int32).pin_memory()
        self.host, self.event, self.waiting = self.pin.data_ptr(), None, False      # one event, recorded again by every push

    def push(self, first, second=None, *more):
        """(Copies and event in one call of the library: 14 -> 5 us with two tensors against torch's.)"""
        if more or not self._plain(first) or not (second is None or self._plain(second)):
            tensors = (first, *((second,) if second is not None else ()), *more)
            first, second = torch.cat([t.reshape(-1).to("cuda", torch.int32) for t in tensors]), None
        n, m = first.numel(), 0 if second is None else second.numel()
        assert n + m <= self.pin.numel()
        if self.event is None:
            event = ctypes.c_void_p()
            check(_lib.lib().stac_event_create(ctypes.byref(event)), "stac_event_create")
            self.event = event.value
        check(_lib.lib().stac_ints_to_host(self.host, first.data_ptr(), n, ptr(second), m, self.event, stream_ptr()),
              "stac_ints_to_host")
        self.waiting = True

    @staticmethod
    def _plain(t):
        return t.is_cuda and t.dtype is torch.int32 and t.is_contiguous()

    def pending(self):
        return self.waiting

    def _arrive(self):
        if self.waiting and self.event is not None:
            check(_lib.lib().stac_event_wait(self.event), "stac_event_wait")

    def pull(self):
        if not self.waiting:
            return None
        self._arrive()
        self.waiting = False
        return self.pin.tolist()

    # A copy, or what is unpickled, has memory of its own and no event.
    def __getstate__(self):
        self._arrive()
        return self.pin.tolist(), self.waiting

    def __setstate__(self, state):
        values, waiting = state
        self.__init__(len(values))
        self.pin.copy_(torch.tensor(values, dtype=torch.int32))
        self.waiting = waiting

    def __del__(self):
        # Whoever drops it may be a step ahead of the GPU, or in the middle of a graph capture, which a wait would spoil.
        event = self.__dict__.pop("event", None)
        try:
            if event is not None and self.waiting:
                _dropped.append((self.pin, event))
            elif event is not None:
                _lib.lib().stac_event_destroy(event)
        except Exception:       # the process or its context is on the way out
            pass


# Page-locked memory (which may be handed to somebody else as soon as it is free) and events of mirrors that went away before their
# copies had arrived; given back when the next mirror is made, so that there are never more than the GPU is behind.
_dropped = collections.deque()


def _free_dropped():
    if not _dropped or torch.cuda.is_current_stream_capturing():      # (an event must not be asked during a capture)
        return
    for _ in range(len(_dropped)):
        try:
            pin, event = _dropped.popleft()
        except IndexError:      # another thread has it
            return
        done = ctypes.c_int(0)
        _lib.lib().stac_event_done(event, ctypes.byref(done))
        if done.value:
            _lib.lib().stac_event_destroy(event)
        else:
            _dropped.append((pin, event))


_workspaces = {}
ATTN_CTL_WORDS = 512      # leading words of an attention workspace that have to be zero


@functools.lru_cache(maxsize=256)      # asking for a capture added 1.0 us to a call of 23 us on the host; this takes it off again
def _attn_workspace_bytes(M, H):
    return _lib.lib().stac_attn_workspace_bytes(M, H)


def _attn_workspace(device, M, H):
    """Scratch of stac_attn_colsum_kept (arrival counters, row log-sum-exps, split partials), zeroed when
    it is made; every call leaves the counters zero.  One per (device, stream): calls on one stream
    are ordered and may share it, calls issued on different streams may overlap on the GPU and must
    not.  A call under graph capture takes one of its own: it comes from the graph's memory, is zeroed by
    the graph, and is used by that graph alone.  (One kept for eager calls may be gone when the graph is
    replayed, or in use by an eager call on the stream that the graph was captured on.)"""
    need = _attn_workspace_bytes(M, H)
    capturing = torch.cuda.is_current_stream_capturing()
    key = (device, stream_ptr(device=device))
    ws = None if capturing else _workspaces.get(key)
    if ws is None or ws.numel() * 4 < need:
        ws = torch.empty(max(need // 4, 1), dtype=torch.float32, device=device)
        ws[:ATTN_CTL_WORDS].zero_()
        if not capturing:
            _workspaces[key] = ws
    return ws


def _kv_strides(t, layout):
    """(row_stride, head_stride) in elements for a [H,T,D] ('htd') or [T,H,D] ('thd') tensor."""
    outer, inner, last = t.stride()
    assert last == 1
    return (inner, outer) if layout == "htd" else (outer, inner)


def _check_score_update(scores, counts, row_stride, H, T_hot, device):
    """The kernel writes [H, T_hot] fp32 scores and counts at ``row_stride`` and is given pointers only."""
    assert scores.dtype is counts.dtype is torch.float32 and scores.device == counts.device == device, \
        "running scores and counts: fp32 on the queries' device"
    assert scores.stride() == counts.stride() == (row_stride, 1) and (H == 1 or row_stride >= T_hot), \
        "running scores and counts: strides"
    (hs, ws), (hc, wc) = scores.shape, counts.shape
    assert hs == hc == H and ws >= T_hot and wc >= T_hot, "running scores and counts: [H, >= T_hot]"


def attn_colsum(q, k_hot, v_hot, T_hot, k_ret=None, v_ret=None, bias_ret=None, T_ret=0, *,
                layout="htd", scale=None, subsample_ratio=1.0, want_lse=False, want_colsum=True,
                out=None, colsum=None, status=None, score_update=None):
    """q [M,H,64] bf16 (row stride arbitrary); hot and retrieved keys/values in ``layout``;
    bias_ret [H, >=T_ret] fp32.  ``score_update``: (scores, counts, row stride, old_T, Tq, temperature), the
    running scores [H, >=T_hot] fp32 of the hot keys that the column sums go into.  Returns (out [M,H,64] bf16, lse [H,M] | None,
    colsum [H, T_hot+T_ret] fp32 | None)."""
    assert q.is_cuda and q.dtype == torch.bfloat16 and q.dim() == 3 and q.stride(2) == 1
    M, H, D = q.shape
    assert q.stride(1) == D, "heads of a query row must be contiguous"
    dev = q.device
    if out is None:
        out = torch.empty((M, H, D), dtype=torch.bfloat16, device=dev)
    lse = torch.empty((H, M), dtype=torch.float32, device=dev) if want_lse else None
    N = T_hot + T_ret
    if want_colsum and colsum is None:
        colsum = torch.empty((H, N), dtype=torch.float32, device=dev)
    if not want_colsum:
        colsum = None
    ws = _attn_workspace(dev, M, H)
    hr, hh = _kv_strides(k_hot, layout) if T_hot > 0 else (D, D)
    if T_hot > 0:
        assert _kv_strides(v_hot, layout) == (hr, hh)
    rr, rh = (D, D)
    if T_ret > 0:
        rr, rh = _kv_strides(k_ret, layout)
        assert _kv_strides(v_ret, layout) == (rr, rh)
        assert bias_ret.dtype == torch.float32 and bias_ret.stride(1) == 1
    if scale is None:
        scale = 1.0 / math.sqrt(D)
    call = [ptr(q), q.stride(0),
            ptr(k_hot) if T_hot > 0 else None, ptr(v_hot) if T_hot > 0 else None, hr, hh, T_hot,
            ptr(k_ret) if T_ret > 0 else None, ptr(v_ret) if T_ret > 0 else None, rr, rh, T_ret,
            ptr(bias_ret) if T_ret > 0 else None, bias_ret.stride(0) if T_ret > 0 else 0,
            ptr(out), out.stride(0), ptr(lse), ptr(colsum), colsum.stride(0) if colsum is not None else 0,
            M, H, D, float(scale), float(subsample_ratio)]
    name = "stac_attn_colsum_kept"
    if score_update is not None:
        scores, counts, row_stride, old_T, Tq, temperature = score_update
        _check_score_update(scores, counts, row_stride, H, T_hot, dev)
        call += [ptr(scores), ptr(counts), row_stride, old_T, Tq, float(temperature)]
        name = "stac_attn_colsum_scored"
    check(getattr(_lib.lib(), name)(*call, ptr(ws), ws.numel() * 4, ptr(status.word) if status is not None else None,
                                    stream_ptr()), name)
    return out, lse, colsum


def flash_attn_bias_colsum(q, k, v, bias=None, softmax_scale=None, return_colsum=False,
                           subsample_ratio=1.0):
    """Same call as the reference's attn_cuda.flash_attn_bias_colsum
    (attn-cuda/attn_cuda/__init__.py:6-43): q [B,M,H,D], k/v [B,N,H,D] bf16 with B == 1,
    bias [B,H,1,N] or [B,H,N] (per-key).  Returns (out [B,M,H,D], lse [B,H,M][, colsum [B,H,N]])."""
    if q.dim() != 4 or q.shape[0] != 1:
        raise ValueError("batch size 1 only")
    if q.shape[-1] != 64:
        raise ValueError("Only head_dim=64 is supported")
    if not (0.0 < subsample_ratio <= 1.0):
        raise ValueError("subsample_ratio must be in (0, 1]")
    q3, k3, v3 = q[0].contiguous(), k[0].contiguous(), v[0].contiguous()
    N = k3.shape[0]
    if bias is None:
        o, lse, cs = attn_colsum(q3, k3, v3, N, layout="thd", scale=softmax_scale,
                                 subsample_ratio=subsample_ratio, want_lse=True,
                                 want_colsum=return_colsum)
    else:
        b = bias
        if b.dim() == 4:
            if b.shape[2] != 1:
                raise ValueError("4D bias must have shape [B, H, 1, N]")
            b = b.squeeze(2)
        b = b[0].to(torch.float32).contiguous()
        # every key carries a bias: treat all of them as the biased segment
        o, lse, cs = attn_colsum(q3, None, None, 0, k3, v3, b, N, layout="thd", scale=softmax_scale,
                                 subsample_ratio=subsample_ratio, want_lse=True,
                                 want_colsum=return_colsum)
    res = (o.unsqueeze(0), lse.unsqueeze(0))
    if return_colsum:
        res = res + (cs.unsqueeze(0),)
    return res
