"""Binding of ``csrc/libwcn_b200.so`` (declared in ``include/wcn_b200.h``).

The library is the only compute back-end of this package: when it is missing
or cannot be loaded, every operation raises; there is no CPU or eager fallback.
PyTorch is used for device memory and streams only.
"""
from __future__ import annotations

import ctypes
import functools
import importlib.util
import os
import threading
from collections import Counter
from typing import Optional

import torch

_HERE = os.path.dirname(os.path.abspath(__file__))
LIB_PATH = os.path.join(_HERE, "csrc", "libwcn_b200.so")
FASTCALL_PATH = os.path.join(_HERE, "csrc", "_fastcall.so")

WCN_F32, WCN_F16, WCN_BF16 = 0, 1, 2
CONV_AUTO, CONV_SIMT, CONV_TCGEN05 = 0, 1, 2
_DTYPE_CODE = {torch.float32: WCN_F32, torch.float16: WCN_F16, torch.bfloat16: WCN_BF16}

_c_i32, _c_i64, _c_vp = ctypes.c_int32, ctypes.c_int64, ctypes.c_void_p
_p_i64 = ctypes.POINTER(ctypes.c_int64)

# name -> argument types, exactly the prototypes of include/wcn_b200.h
SIGNATURES = {
    "wcn_version": [],
    "wcn_hash_table_bytes": [_c_i64, _p_i64],
    "wcn_hash_build": [_c_vp, _c_i64, _c_vp, _c_vp, _c_i64, _c_i32, _c_vp, _c_vp, _c_vp],
    "wcn_hash_search": [_c_vp, _c_i64, _c_i32, _c_vp, _c_i64, _c_vp, _c_vp],
    "wcn_unique_workspace_bytes": [_c_i64, _p_i64],
    "wcn_unique_mark": [_c_vp, _c_i64, _c_vp, _c_vp, _c_i64, _c_i32, _c_vp, _c_vp, _c_vp],
    "wcn_unique_emit": [_c_vp, _c_i64, _c_vp, _c_vp, _c_vp, _c_vp, _c_vp, _c_vp],
    "wcn_kmap_workspace_bytes": [_c_i64, _c_i32, _p_i64],
    "wcn_kmap_search": [_c_vp, _c_i64, _c_i32, _c_vp, _c_i64, _c_vp, _c_vp, _c_i32, _c_vp, _c_vp, _c_vp],
    "wcn_kmap_search_static": [_c_vp, _c_i64, _c_i32, _c_vp, _c_i64, _c_vp, _c_vp, _c_i32, _c_vp, _c_vp, _c_vp],
    "wcn_kmap_search_self": [_c_vp, _c_i64, _c_i32, _c_vp, _c_i64, _c_vp, _c_vp, _c_vp, _c_vp],
    "wcn_kmap_search_dilated": [_c_vp, _c_i64, _c_i32, _c_vp, _c_i64, _c_vp, _c_vp, _c_vp, _c_vp, _c_i32, _c_vp, _c_vp, _c_vp],
    "wcn_kmap_count": [_c_vp, _c_i64, _c_i32, _c_vp, _c_vp],
    "wcn_brick_table_bytes": [_c_i64, _p_i64],
    "wcn_brick_build": [_c_vp, _c_i64, _c_vp, _c_vp, _c_vp],
    "wcn_kmap_search_bricks": [_c_vp, _c_vp, _c_i64, _c_i32, _c_vp, _c_i64, _c_vp, _c_vp, _c_vp, _c_vp],
    "wcn_kmap_scan": [_c_vp, _c_i64, _c_i32, _c_vp, _c_vp],
    "wcn_kmap_compact": [_c_vp, _c_i64, _c_i32, _c_vp, _c_vp, _c_vp, _c_vp, _c_vp],
    "wcn_nbr_from_maps": [_c_vp, _c_vp, _c_vp, _c_i32, _c_i64, _c_i64, _c_vp, _c_vp],
    "wcn_nbr_transpose": [_c_vp, _c_i32, _c_i64, _c_i64, _c_vp, _c_vp],
    "wcn_morton20": [_c_vp, _c_i64, _c_i32, _c_i32, _c_vp, _c_vp, _c_vp],
    "wcn_gather_rows": [_c_vp, _c_i64, _c_vp, _c_vp, _c_i64, _c_i32, _c_i32, _c_vp, _c_vp],
    "wcn_scatter_add_rows": [_c_vp, _c_vp, _c_vp, _c_i64, _c_i64, _c_i32, _c_i32, _c_vp, _c_vp],
    "wcn_conv_packed_weight_bytes": [_c_i32, _c_i32, _c_i32, _c_i32, _c_i32, _p_i64],
    "wcn_conv_pack_weight": [_c_i32, _c_vp, _c_i32, _c_i32, _c_i32, _c_i32, _c_vp, _c_vp],
    "wcn_kmap_tile_order": [_c_vp, _c_i64, _c_i32, _c_vp, _c_vp, _c_vp],
    "wcn_row_reduce": [_c_vp, _c_i64, _c_vp, _c_i64, _c_i32, _c_i32, _c_i32, _c_i32, _c_vp, _c_vp, _c_vp],
    "wcn_row_reduce_train": [_c_vp, _c_i64, _c_vp, _c_i64, _c_i32, _c_i32, _c_i32, _c_i32, _c_vp, _c_vp, _c_i32, _c_vp, _c_vp, _c_vp],
    "wcn_row_reduce_backward": [_c_vp, _c_i64, _c_vp, _c_i64, _c_i32, _c_i32, _c_i32, _c_vp, _c_i32, _c_vp, _c_vp, _c_vp, _c_vp],
    "wcn_kmap_tile_masks": [_c_vp, _c_i64, _c_i32, _c_vp, _c_vp],
    "wcn_conv_wgrad": [_c_vp, _c_i64, _c_vp, _c_vp, _c_vp, _c_vp, _c_i64, _c_i32, _c_i32, _c_i32, _c_i32, _c_vp, _c_vp, _c_vp],
    "wcn_conv_wgrad_f32_workspace_bytes": [_c_i64, _c_i64, _c_i32, _c_i32, _c_i32, _p_i64],
    "wcn_conv_wgrad_f32": [_c_vp, _c_i64, _c_vp, _c_vp, _c_vp, _c_vp, _c_i64, _c_i32, _c_i32, _c_i32, _c_vp, _c_vp, _c_i64, _c_vp, _c_vp],
    "wcn_conv_wgrad_pairs_workspace_bytes": [_c_i64, _c_i32, _c_i32, _c_i32, _p_i64],
    "wcn_conv_wgrad_pairs": [_c_vp, _c_i64, _c_vp, _c_vp, _c_vp, _c_i64, _c_i32, _c_i32, _c_i32, _c_i32, _c_vp, _c_vp, _c_i64, _c_vp, _c_vp],
    "wcn_conv_workspace_bytes": [_c_i32, _c_i64, _c_i32, _c_i32, _c_i32, _c_i32, _c_i32, _c_i32, _p_i64],
    "wcn_conv_f32_launches": [],
    "wcn_conv_f32_workspace_bytes": [_c_i64, _c_i64, _c_i32, _c_i32, _c_i32, _p_i64],
    "wcn_conv_fwd": [_c_i32, _c_vp, _c_i64, _c_i64, _c_vp, _c_vp, _c_vp, _c_vp, _c_i64, _c_i32, _c_i32, _c_i32, _c_i32,
                     _c_vp, _c_vp, _c_vp, _c_i64, _c_i32, _c_vp, _c_i64, _c_i32, _c_i32, _c_vp, _c_i64, _c_vp, _c_vp],
    "wcn_column_sums_workspace_bytes": [_c_i64, _c_i32, _c_i32, _p_i64],
    "wcn_column_sums": [_c_vp, _c_i64, _c_i32, _c_i32, _c_vp, _c_vp, _c_vp],
    "wcn_batch_norm_workspace_bytes": [_c_i64, _c_i32, _c_i32, _p_i64],
    "wcn_batch_norm_train": [_c_vp, _c_i64, _c_i32, _c_i32, _c_vp, _c_vp, _c_i32, _c_i32, _c_vp, _c_vp, _c_vp, _c_vp, _c_i32,
                             _c_vp, _c_vp, _c_vp, _c_vp, _c_vp, _c_vp],
    "wcn_batch_norm_backward": [_c_vp, _c_vp, _c_vp, _c_i64, _c_i32, _c_i32, _c_vp, _c_vp, _c_vp, _c_vp, _c_i32, _c_vp, _c_vp,
                                _c_vp, _c_vp, _c_vp, _c_vp],
    "wcn_conv_pack_weight_from": [_c_vp, _c_i32, _c_i32, _c_i32, _c_i32, _c_i32, _c_i32, _c_i32, _c_vp, _c_vp],
    "wcn_cells_bytes": [_c_i64, _p_i64],
    "wcn_cells_build": [_c_vp, _c_i64, _c_vp, _c_vp],
    "wcn_kmap_search_cells": [_c_vp, _c_i64, _c_vp, _c_i64, _c_vp, _c_vp, _c_vp, _c_vp, _c_vp],
    "wcn_kmap_scan_host": [_c_vp, _c_i64, _c_i32, _c_vp, _c_vp, _c_vp, _c_vp],
    "wcn_unique_counts": [_c_vp, _c_i64, _c_vp, _c_i32, _c_vp, _c_vp, _c_vp, _c_vp],
    "wcn_morton_sort_workspace_bytes": [_c_i64, _p_i64],
    "wcn_morton_sort": [_c_vp, _c_i64, _c_vp, _c_i32, _c_vp, _c_vp, _c_vp, _c_vp, _c_vp, _c_vp, _c_i32, _c_vp, _c_vp, _c_vp],
    "wcn_pyramid_workspace_bytes": [_c_i64, _p_i64],
    "wcn_pyramid": [_c_vp, _c_i64, _c_vp, _c_vp, _c_i32, _c_i32, _c_vp, _c_vp, _c_vp, _c_vp, _c_vp, _c_vp, _c_vp],
    "wcn_level_brick_bytes": [_c_i64, _p_i64],
    "wcn_level_maps": [_c_vp, _c_i32, _c_vp, _c_vp, _c_i32, _c_vp],
    "wcn_net_run": [_c_vp, _c_i32, _c_vp, _c_vp, _c_vp, _c_i32, _c_vp, _c_vp],
    "wcn_selftest_bounded_wait": [_c_i64, _c_vp, _c_vp, _c_vp],
    "wcn_conv_rows_supported": [_c_i32, _c_i32, _c_i32, _c_i32, _c_i32, _c_vp],
    "wcn_conv_rows_fwd": [_c_vp, _c_i64, _c_i64, _c_vp, _c_vp, _c_i64, _c_i32, _c_i32, _c_i32, _c_i32, _c_i32, _c_vp, _c_vp,
                          _c_vp, _c_i64, _c_i32, _c_vp, _c_i64, _c_i32, _c_vp, _c_vp],
}



class Level(ctypes.Structure):
    """``wcn_level``"""
    _fields_ = [("rows", _c_vp), ("n", _c_i64), ("bricks", _c_vp), ("order", _c_vp), ("nbr", _c_vp), ("child", _c_vp),
                ("first_child", _c_vp), ("rows_below", _c_vp), ("n_below", _c_i64), ("level", _c_i64)]


class NetOp(ctypes.Structure):
    """``wcn_net_op``"""
    _fields_ = [(f, _c_i32) for f in ("kind", "table", "level_in", "level_out", "num_offsets", "c_in", "c_out", "c_out_packed",
                                      "relu", "src", "src_col", "dst", "dst_col", "res", "res_col", "reserved")] + [
        (f, _c_vp) for f in ("weight", "packed", "scale", "shift")]


_lib = None

# Kernels launched by one call of each entry point (0: host-only query).  Used to
# count this library's launches, e.g. by the benchmark harness.
KERNELS_PER_CALL = {
    "wcn_hash_build": 2, "wcn_hash_search": 1, "wcn_unique_mark": 3, "wcn_unique_emit": 2, "wcn_kmap_search": 1, "wcn_kmap_search_static": 3,
    "wcn_kmap_scan": 2, "wcn_kmap_compact": 1, "wcn_nbr_from_maps": 1, "wcn_nbr_transpose": 1, "wcn_morton20": 1,
    "wcn_kmap_tile_order": 3, "wcn_conv_wgrad": 1, "wcn_conv_wgrad_pairs": 2, "wcn_conv_wgrad_f32": 3, "wcn_kmap_tile_masks": 1, "wcn_row_reduce": 1, "wcn_row_reduce_train": 1, "wcn_row_reduce_backward": 1, "wcn_kmap_search_self": 1, "wcn_kmap_search_dilated": 1, "wcn_kmap_count": 1,
    "wcn_gather_rows": 1, "wcn_scatter_add_rows": 1, "wcn_conv_pack_weight": 1, "wcn_conv_fwd": 1,
    "wcn_selftest_bounded_wait": 1, "wcn_brick_build": 3, "wcn_kmap_search_bricks": 1,
    "wcn_conv_rows_fwd": 1, "wcn_batch_norm_train": 2, "wcn_column_sums": 2, "wcn_batch_norm_backward": 2, "wcn_conv_pack_weight_from": 1, "wcn_cells_build": 4, "wcn_kmap_search_cells": 1, "wcn_kmap_scan_host": 2, "wcn_unique_counts": 2, "wcn_morton_sort": 1, "wcn_pyramid": 2, "wcn_level_maps": 5,
}
LAUNCH_COUNTS: Counter = Counter()


def _counted(raw, name: str, kernels: Optional[int]):
    """``raw`` through ctypes, counting the kernels it launches."""
    if not kernels:
        return raw

    def fn(*args):
        LAUNCH_COUNTS[name] += kernels
        return raw(*args)
    return fn


class _Library:
    """The C functions as attributes.  Those that take only integers and pointers go through the ``_fastcall``
    extension (csrc/fastcall.c): a 26-argument call costs 0.3 us there and 3.5 us through ctypes, which for a small
    layer is as much as its launch.  It also counts the kernels they launch.  The extension is a way of calling and no
    more: where it cannot be built (it knows the argument passing of x86-64 Linux and needs Python 3.12 with its headers)
    ``bind`` is None and ctypes makes the same calls."""

    def __init__(self, handle, bind):
        for name, argtypes in SIGNATURES.items():
            fn = getattr(handle, name)
            fn.argtypes, fn.restype = argtypes, ctypes.c_int
            if bind is None:
                fn = _counted(fn, name, KERNELS_PER_CALL.get(name))
            elif all(t in (_c_i32, _c_i64, _c_vp) for t in argtypes):
                fn = bind(ctypes.cast(fn, ctypes.c_void_p).value, len(argtypes), name, LAUNCH_COUNTS,
                          KERNELS_PER_CALL.get(name))
            setattr(self, name, fn)
        handle.wcn_status_string.argtypes, handle.wcn_status_string.restype = [ctypes.c_int], ctypes.c_char_p
        handle.wcn_brick_usable_flag.argtypes, handle.wcn_brick_usable_flag.restype = [ctypes.c_void_p], ctypes.c_void_p
        self.wcn_status_string, self.wcn_brick_usable_flag = handle.wcn_status_string, handle.wcn_brick_usable_flag


def count_f32_launches(name: str) -> None:
    """Corrects what the call just made was counted as: with a workspace ``wcn_conv_fwd`` launches one or two kernels,
    ``wcn_conv_wgrad_f32`` two or three."""
    LAUNCH_COUNTS[name] += lib().wcn_conv_f32_launches() - KERNELS_PER_CALL[name]


def launches_total() -> int:
    return sum(LAUNCH_COUNTS.values())


class NativeLibraryError(RuntimeError):
    pass


def lib():
    """The loaded library; raises NativeLibraryError when it is not built."""
    global _lib
    if _lib is None:
        if not os.path.isfile(LIB_PATH):
            raise NativeLibraryError(
                f"{LIB_PATH} is missing: build it with `python -m warpconvnet_b200.csrc.build` "
                "(nvcc, sm_100a). This package has no fallback path.")
        try:
            handle = ctypes.CDLL(LIB_PATH)
        except OSError as e:  # pragma: no cover
            raise NativeLibraryError(f"cannot load {LIB_PATH}: {e}") from e
        _lib = _Library(handle, _fastcall_bind())
    return _lib


def _fastcall_bind():
    """``bind`` of the extension, or None where it was not built or does not load."""
    if not os.path.isfile(FASTCALL_PATH):
        return None
    try:
        spec = importlib.util.spec_from_file_location("_fastcall", FASTCALL_PATH)
        fastcall = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(fastcall)
    except ImportError:
        return None
    return fastcall.bind


def status_string(status: int) -> str:
    return lib().wcn_status_string(int(status)).decode()


def check(status: int, what: str = "") -> None:
    if status != 0:
        raise RuntimeError(f"libwcn_b200 {what} failed: {status_string(status)} ({status})")


def ptr(t: Optional[torch.Tensor]) -> Optional[int]:
    return None if t is None else t.data_ptr()


def stream_ptr(device: torch.device) -> int:
    """Raw handle of torch's current stream on ``device`` (the launches go there)."""
    idx = device.index
    if idx is None:
        idx = torch.cuda.current_device()
    return torch._C._cuda_getCurrentRawStream(idx)


def small_to_device(t: torch.Tensor, device, dtype: Optional[torch.dtype] = None) -> torch.Tensor:
    """A small host tensor (batch offsets, a few sizes) on ``device`` WITHOUT synchronising the
    stream: staged through pinned memory and copied asynchronously.  (A plain ``.to(device)`` of
    pageable memory waits for everything queued on the stream before it returns.)"""
    if t.device.type != "cpu":
        return t.to(device=device, dtype=dtype)
    if dtype is not None and t.dtype != dtype:
        t = t.to(dtype)
    return t.pin_memory().to(device, non_blocking=True)


def dtype_code(dtype: torch.dtype) -> int:
    try:
        return _DTYPE_CODE[dtype]
    except KeyError:
        raise TypeError(f"unsupported feature dtype {dtype}; expected float32, float16 or bfloat16")


def require_cuda(t: torch.Tensor, name: str) -> None:
    if not t.is_cuda:
        raise ValueError(f"{name} must be on a CUDA device, got {t.device}")


_status_words = {}


def device_status(device: torch.device) -> torch.Tensor:
    """Per-device int32 status word shared by all kernels that can fail on the device."""
    device = torch.device(device)
    key = (device.type, device.index if device.index is not None else torch.cuda.current_device())
    if key not in _status_words:
        _status_words[key] = torch.zeros(1, dtype=torch.int32, device=device)
    return _status_words[key]


def raise_for_status(code: int, device: torch.device) -> None:
    """Raise for a status-word value the caller has already brought to the host; the word is
    zeroed so that the next launches run again."""
    if code != 0:
        device_status(device).zero_()
        raise RuntimeError(f"libwcn_b200 kernel reported: {status_string(int(code))} ({int(code)})")


def check_device_status(device: torch.device) -> None:
    """Read the status word (synchronises) and raise if a kernel recorded a failure.

    Kernels report hash-table overflow, an expired bounded wait and out-of-range indices only
    through this word, and the tensor-core kernels do no work while it is set (convolution
    outputs are then filled with NaN).  The package reads it wherever it synchronises with the
    host anyway (sizing strided coordinates, compacting a kernel map); a caller that never reaches
    such a point should call this after the work it wants checked."""
    device = torch.device(device)
    word = device_status(device)
    host = torch.empty(1, dtype=torch.int32, pin_memory=True)  # (a pageable read costs another 10 us)
    host.copy_(word, non_blocking=True)
    torch.cuda.current_stream(device).synchronize()
    raise_for_status(int(host[0]), device)


_written: list = []   # (event, pinned tensor): results of kernels that may still be running
_written_lock = threading.Lock()


def pinned_result(words: int, dtype: torch.dtype, device: torch.device, launch):
    """(pinned tensor of ``words``, event after the kernels that write it): ``launch(tensor)`` enqueues those on the
    current stream.  Torch's pinned allocator knows of copies, not of kernels, and would hand the memory to the next
    caller as soon as the tensor is dropped; so it is kept here until the event has passed, whether or not the caller
    waits for it.  (Not inside a stream capture: a graph's kernels write at every replay.)"""
    host = torch.empty(words, dtype=dtype, pin_memory=True)
    done = torch.cuda.Event()
    try:
        launch(host)
    finally:
        done.record(torch.cuda.current_stream(device))
        with _written_lock:
            if len(_written) >= 16:
                _written[:] = [w for w in _written if not w[0].query()]
            _written.append((done, host))
    return host, done


@functools.lru_cache(maxsize=1024)
def query_bytes(fn_name: str, *args) -> int:
    """The size that a ``wcn_*_bytes`` function gives for ``args`` (it depends on them alone)."""
    out = ctypes.c_int64(0)
    check(getattr(lib(), fn_name)(*args, ctypes.byref(out)), fn_name)
    return int(out.value)
