"""ctypes binding of libstac_b200.so.  There is no fallback: if the library is missing or a
call fails, an exception is raised."""

import ctypes
import functools
import os

HERE = os.path.dirname(os.path.abspath(__file__))
LIB_PATH = os.path.join(HERE, "libstac_b200.so")

c_void_p, c_int, c_i64, c_f32, c_size_t = (ctypes.c_void_p, ctypes.c_int, ctypes.c_int64,
                                           ctypes.c_float, ctypes.c_size_t)



class StacPool(ctypes.Structure):
    """Mirror of `struct stac_pool` (include/stac_b200.h)."""
    _fields_ = [
        ("heads", c_int), ("head_dim", c_int), ("elem_bytes", c_int),
        ("pivot_cap", c_int), ("budget_cap", c_int),
        ("voxel_cap", c_int), ("voxel_used", c_int),
        ("sim_thresh", c_f32), ("replace_thresh", c_f32), ("score_thresh", c_f32),
        ("buf_K", c_void_p), ("buf_V", c_void_p), ("buf_S", c_void_p),
        ("buf_row_seg", c_void_p), ("buf_row_cnt", c_void_p), ("buf_free", c_void_p), ("buf_cap", c_int),
        ("piv_K", c_void_p), ("piv_V", c_void_p), ("piv_W", c_void_p), ("piv_S", c_void_p), ("piv_C", c_void_p),
        ("piv_row_seg", c_void_p), ("piv_row_cnt", c_void_p), ("piv_cap", c_int),
        ("over_K_in", c_void_p), ("over_V_in", c_void_p), ("over_S_in", c_void_p),
        ("over_hv_in", c_void_p), ("over_start_in", c_void_p),
        ("over_K_out", c_void_p), ("over_V_out", c_void_p), ("over_S_out", c_void_p),
        ("over_hv_out", c_void_p), ("over_start_out", c_void_p),
        ("over_cap", c_int),
        ("meta", c_void_p),
        ("voxel_count", c_void_p),
    ]


class StacEvicted(ctypes.Structure):
    """Mirror of `struct stac_evicted` (include/stac_b200.h)."""
    _fields_ = [
        ("k", c_void_p), ("v", c_void_p),
        ("kv_head_stride", c_i64), ("kv_row_stride", c_i64),
        ("scores", c_void_p), ("voxel_ids", c_void_p),
        ("meta_head_stride", c_i64),
        ("positions", c_void_p),
        ("tokens_per_head", c_int),
    ]


(META_BUF_TOP, META_BUF_FREE_LEN, META_PIV_TOP, META_OVER_COUNT, META_BUF_USED, META_PIV_USED, META_DROPPED,
 META_VOXELS) = range(8)
META_SIZE = 8
VOXEL_MAX_POINTS = 131072
ERR_CAPACITY = 3           # STAC_ERR_CAPACITY

# name -> (restype, argtypes); must list every function declared in include/stac_b200.h
SIGNATURES = {
    "stac_status_string": (ctypes.c_char_p, [c_int]),
    "stac_abi_version": (c_int, []),
    "stac_kernel_launches": (ctypes.c_uint64, []),
    "stac_attn_workspace_bytes": (c_size_t, [c_int, c_int]),
    "stac_attn_forward_plan": (c_int, [c_int, c_int, c_int, c_int, c_int, c_int, ctypes.POINTER(c_int), ctypes.POINTER(c_int)]),
    "stac_attn_colsum": (c_int, [c_void_p, c_i64, c_void_p, c_void_p, c_i64, c_i64, c_int, c_void_p, c_void_p,
                                 c_i64, c_i64, c_int, c_void_p, c_i64, c_void_p, c_i64, c_void_p, c_void_p, c_i64,
                                 c_int, c_int, c_int, c_f32, c_f32, c_void_p, c_size_t, c_void_p, c_void_p]),
    "stac_attn_colsum_kept": (c_int, [c_void_p, c_i64, c_void_p, c_void_p, c_i64, c_i64, c_int, c_void_p, c_void_p,
                                      c_i64, c_i64, c_int, c_void_p, c_i64, c_void_p, c_i64, c_void_p, c_void_p, c_i64,
                                      c_int, c_int, c_int, c_f32, c_f32, c_void_p, c_size_t, c_void_p, c_void_p]),
    "stac_attn_colsum_noalloc": (c_int, [c_void_p, c_i64, c_void_p, c_void_p, c_i64, c_i64, c_int, c_void_p,
                                         c_void_p, c_i64, c_i64, c_int, c_void_p, c_i64, c_void_p, c_i64, c_void_p,
                                         c_void_p, c_i64, c_int, c_int, c_int, c_f32, c_f32, c_void_p, c_void_p]),
    "stac_attn_colsum_scored": (c_int, [c_void_p, c_i64, c_void_p, c_void_p, c_i64, c_i64, c_int, c_void_p, c_void_p,
                                        c_i64, c_i64, c_int, c_void_p, c_i64, c_void_p, c_i64, c_void_p, c_void_p, c_i64,
                                        c_int, c_int, c_int, c_f32, c_f32, c_void_p, c_void_p, c_i64, c_int, c_int,
                                        c_f32, c_void_p, c_size_t, c_void_p, c_void_p]),
    "stac_selftest_bounded_wait": (c_int, [c_int, c_void_p, c_void_p]),
    "stac_voxel_scratch_bytes": (c_size_t, [c_int]),
    "stac_voxel_hash_clear": (c_int, [c_void_p, c_i64, c_void_p]),
    "stac_voxel_rehash": (c_int, [c_void_p, c_void_p, c_int, c_void_p, c_void_p, c_i64, c_void_p]),
    "stac_voxel_upsert": (c_int, [c_void_p, c_void_p, c_void_p, c_int, c_f32, c_void_p, c_int, c_void_p, c_void_p, c_i64,
                                  c_void_p, c_void_p, c_void_p, c_size_t, c_void_p, c_void_p]),
    "stac_pointmap_to_positions": (c_int, [c_void_p, c_void_p, c_int, c_int, c_int, c_int, c_int, c_f32, c_void_p,
                                           c_void_p, c_void_p]),
    "stac_voxel_neighbors": (c_int, [c_void_p, c_int, c_int, c_int, c_void_p, c_void_p, c_int, c_void_p, c_void_p,
                                     c_i64, c_void_p, c_void_p, c_void_p, c_void_p]),
    "stac_append_kv": (c_int, [c_void_p, c_void_p, c_i64, c_i64, c_i64, c_i64, c_void_p, c_void_p, c_i64, c_void_p,
                               c_i64, c_int, c_int, c_int, c_i64, c_int, c_int, c_void_p]),
    "stac_qkv_epilogue_append": (c_int, [c_void_p, c_i64, c_void_p, c_void_p, c_void_p, c_void_p, c_f32, c_void_p,
                                         c_void_p, c_void_p, c_int, c_void_p, c_i64, c_void_p, c_void_p, c_i64,
                                         c_void_p, c_i64, c_int, c_int, c_int, c_i64, c_void_p]),
    "stac_qkv_epilogue_append_tables": (c_int, [c_void_p, c_i64, c_void_p, c_void_p, c_void_p, c_void_p, c_f32, c_void_p,
                                                c_void_p, c_void_p, c_i64, c_int, c_void_p, c_i64, c_void_p, c_void_p,
                                                c_i64, c_void_p, c_i64, c_int, c_int, c_int, c_i64, c_void_p]),
    "stac_scores_update": (c_int, [c_void_p, c_i64, c_void_p, c_void_p, c_i64, c_int, c_int, c_int, c_int, c_f32,
                                   c_void_p]),
    "stac_h2o_select": (c_int, [c_void_p, c_i64, c_int, c_void_p, c_int, c_int, c_void_p, c_void_p, c_void_p]),
    "stac_compact": (c_int, [c_void_p, c_int, c_int, c_int, c_int, c_int, c_void_p, c_void_p, c_void_p, c_void_p,
                             c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p, c_void_p,
                             c_void_p]),
    "stac_compact_window": (c_int, [c_void_p, c_int, c_int, c_int, c_int, c_int, c_void_p, c_void_p, c_void_p, c_void_p,
                                    c_void_p, c_void_p, c_void_p]),
    "stac_event_create": (c_int, [ctypes.POINTER(c_void_p)]),
    "stac_event_destroy": (c_int, [c_void_p]),
    "stac_event_wait": (c_int, [c_void_p]),
    "stac_event_done": (c_int, [c_void_p, ctypes.POINTER(c_int)]),
    "stac_ints_to_host": (c_int, [c_void_p, c_void_p, c_int, c_void_p, c_int, c_void_p, c_void_p]),
    "stac_merge_scratch_bytes": (c_size_t, [c_int, c_int, c_int]),
    "stac_merge_insert": (c_int, [ctypes.POINTER(StacPool), ctypes.POINTER(StacEvicted), c_void_p, c_size_t, c_int,
                                  c_void_p, c_void_p]),
    "stac_retrieve": (c_int, [ctypes.POINTER(StacPool), c_void_p, c_void_p, c_int, c_void_p, c_void_p, c_void_p,
                              c_void_p, c_void_p, c_void_p, c_void_p]),
}


def kernel_launches():
    """Kernels that the library has launched so far, counted where they are launched."""
    return lib().stac_kernel_launches()


_lib = None


class StacError(RuntimeError):
    pass


def lib():
    """Load the shared library once; raise if it is absent (the product has no CPU path)."""
    global _lib
    if _lib is None:
        if not os.path.exists(LIB_PATH):
            raise StacError(f"{LIB_PATH} not found: build it with `python -m stac_b200.build`")
        handle = ctypes.CDLL(LIB_PATH)
        for name, (res, args) in SIGNATURES.items():
            fn = getattr(handle, name)
            fn.restype = res
            fn.argtypes = args
        _lib = handle
    return _lib


def check(status, what):
    if status != 0:
        msg = lib().stac_status_string(status).decode()
        raise StacError(f"{what} failed: {msg} (status {status})")


def ptr(t):
    """Device pointer of a torch tensor (or None -> NULL), as the plain int that ctypes converts itself."""
    return None if t is None else t.data_ptr()


_stream_calls = None


def _torch_stream_calls():
    """torch's functions for the raw handle of a stream and for the current device, looked up at the first
    use: this module is also imported without torch, and with a torch that has no CUDA."""
    global _stream_calls
    import torch
    if not hasattr(torch._C, "_cuda_getCurrentRawStream"):
        raise StacError("this torch has no CUDA: there is no stream to launch on")
    _stream_calls = torch._C._cuda_getCurrentRawStream, torch._C._cuda_getDevice
    return _stream_calls


def stream_ptr(stream=None, device=None):
    """Handle of `stream`, or of the stream that is current on `device` (default: the current device).
    The raw handle is asked for directly: a torch.cuda.Stream object per call costs 3.4 us, and a
    call of this library does little else on the host (a step of a small two-layer stream, all of it
    host time: 537 -> 440 us with the lighter calls of this file; points to voxel ids 82 -> 71 us)."""
    if stream is not None:
        return stream.cuda_stream
    raw_stream, current_device = _stream_calls or _torch_stream_calls()
    index = device.index if device is not None else None
    return raw_stream(current_device() if index is None else index)


def no_grad(fn):
    """torch.no_grad() around a plain function, for functions called several times per layer: nothing is
    done where gradients are off already (they call one another), and no context object is made."""
    import torch
    is_enabled, set_enabled = torch.is_grad_enabled, torch._C._set_grad_enabled

    @functools.wraps(fn)
    def wrapped(*args, **kwargs):
        if not is_enabled():
            return fn(*args, **kwargs)
        set_enabled(False)
        try:
            return fn(*args, **kwargs)
        finally:
            set_enabled(True)
    return wrapped
