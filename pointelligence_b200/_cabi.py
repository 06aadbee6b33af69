"""ctypes binding of ``libpointelligence_b200.so`` (see
``include/pointelligence_b200.h``) and the marshalling helpers used by the
host-side mirrors of the reference modules.

The library is mandatory: if it cannot be loaded every operator raises
``RuntimeError`` -- there is no CPU or PyTorch fallback.  Tensors are passed as
raw device pointers; outputs and workspaces are allocated here with PyTorch so
the caching allocator and the caller's current stream stay in charge.
"""
from __future__ import annotations

import ctypes
import os
import threading
import time
from ctypes import c_double, c_int, c_int64, c_size_t, c_void_p

import torch

_HERE = os.path.dirname(os.path.abspath(__file__))
LIB_PATH = os.path.join(_HERE, "lib", "libpointelligence_b200.so")

PCX_F32, PCX_F16, PCX_BF16 = 0, 1, 2
ENGINE_AUTO, ENGINE_CUDA_CORE, ENGINE_TENSOR = 0, 1, 2
ENGINE_FLAG_FAN_IN_ONE = 0x100   # OR-ed into an engine: every output row occurs in exactly one triplet
PCX_E_CAPACITY = -4

_DTYPES = {torch.float32: PCX_F32, torch.float16: PCX_F16, torch.bfloat16: PCX_BF16}

_STATUS_EXC = {
    -1: ValueError,          # PCX_E_ARG
    -2: TypeError,           # PCX_E_DTYPE
    -3: ValueError,          # PCX_E_ALIGN
    -4: RuntimeError,        # PCX_E_CAPACITY
    -5: RuntimeError,        # PCX_E_LAUNCH
    -6: NotImplementedError, # PCX_E_UNSUPPORTED
    -7: RuntimeError,        # PCX_E_DEVICE
}

# name -> (restype, argtypes); every symbol declared in the header
SIGNATURES = {
    "pcx_version": (c_int, []),
    "pcx_last_error_string": (ctypes.c_char_p, []),
    "pcx_device_status": (c_int, [c_void_p, c_int, c_void_p]),
    "pcx_launch_count": (ctypes.c_longlong, [c_int]),
    "pcx_profile_enable": (c_int, [c_int]),
    "pcx_profile_count": (c_int, []),
    "pcx_profile_get": (c_int, [c_int, ctypes.POINTER(ctypes.c_char_p), ctypes.POINTER(ctypes.c_float)]),
    "pcx_mvmr_workspace_bytes": (c_size_t, [c_int64, c_int, c_int, c_int, c_int, c_int, c_int]),
    "pcx_mvmr": (c_int, [c_void_p] * 7 + [c_int64] * 3 + [c_int] * 7 + [c_void_p, c_size_t, c_void_p]),
    "pcx_mvmr_bias": (c_int, [c_void_p] * 8 + [c_int64] * 3 + [c_int] * 7 + [c_void_p, c_size_t, c_void_p]),
    "pcx_reshape16": (c_int, [c_void_p] * 2 + [c_int64] + [c_int] * 4 + [c_void_p]),
    "pcx_column_sums_workspace_bytes": (c_size_t, [c_int64, c_int]),
    "pcx_column_sums": (c_int, [c_void_p] * 2 + [c_int64, c_int, c_int, c_void_p, c_size_t, c_void_p]),
    "pcx_mvmr_plan_group_blocks": (c_int, [c_int]),
    "pcx_mvmr_plan_bytes": (c_size_t, [c_int64, c_int64, c_int, c_int]),
    "pcx_mvmr_plan_workspace_bytes": (c_size_t, [c_int64, c_int64, c_int, c_int]),
    "pcx_mvmr_plan_build": (c_int, [c_void_p] * 3 + [c_int64, c_int, c_int64, c_int, c_void_p, c_size_t, c_void_p,
                                    c_size_t, c_void_p]),
    "pcx_mvmr_plan_build_counted": (c_int, [c_void_p] * 3 + [c_int64, c_int, c_int64, c_int, c_void_p, c_size_t,
                                            c_void_p, c_size_t, ctypes.POINTER(c_int64), c_void_p]),
    "pcx_mvmr_plan_multi_buckets": (c_int, [c_void_p, ctypes.POINTER(c_int64), c_void_p]),
    "pcx_mvmr_planned_workspace_bytes": (c_size_t, [c_int64, c_int]),
    "pcx_mvmr_planned": (c_int, [c_void_p] * 3 + [c_size_t, c_void_p] + [c_int64] * 3 + [c_int] * 6
                         + [c_int64, c_void_p, c_size_t, c_void_p]),
    "pcx_mvmr_planned_scratch_bytes": (c_size_t, [c_int64, c_int, c_int64, c_int, c_int, c_int]),
    "pcx_mvmr_planned_bias": (c_int, [c_void_p] * 3 + [c_size_t] + [c_void_p] * 2 + [c_int64] * 3 + [c_int] * 7
                              + [c_int64, c_void_p, c_size_t, c_void_p]),
    "pcx_mvmr_thin_workspace_bytes": (c_size_t, [c_int64] * 2 + [c_int] * 4),
    "pcx_mvmr_thin": (c_int, [c_void_p] * 7 + [c_int64] * 3 + [c_int] * 5 + [c_void_p, c_size_t, c_void_p]),
    "pcx_mvmr_split_workspace_bytes": (c_size_t, [c_int64, c_int64] + [c_int] * 5),
    "pcx_mvmr_split": (c_int, [c_void_p] * 6 + [c_size_t] + [c_void_p] * 2 + [c_int64] * 3 + [c_int] * 6
                       + [c_int64, c_void_p, c_size_t, c_void_p]),
    "pcx_debug_wait_runs_out": (c_int, [ctypes.c_ulonglong, c_void_p]),
    "pcx_vvor_workspace_bytes": (c_size_t, [c_int64, c_int, c_int, c_int, c_int]),
    "pcx_vvor": (c_int, [c_void_p] * 7 + [c_int64] * 4 + [c_int] * 5 + [c_void_p, c_size_t, c_void_p]),
    "pcx_vvor_store_limit": (c_int64, [c_int64, c_int, c_int, c_int]),
    "pcx_vvor_known": (c_int, [c_void_p] * 7 + [c_int64] * 4 + [c_int] * 5 + [c_int64, c_void_p, c_size_t, c_void_p]),
    "pcx_vvor_static_scratch_max_elements": (c_size_t, []),
    "pcx_vvor_static_scratch": (c_int, [c_void_p] * 6 + [c_int64] * 4 + [c_int] * 4 + [c_void_p]),
    "pcx_segment_reduce_workspace_bytes": (c_size_t, [c_int64, c_int]),
    "pcx_segment_reduce": (c_int, [c_void_p] * 3 + [c_int64, c_int64, c_int, c_int, c_int, c_void_p, c_size_t,
                                                   c_void_p]),
    "pcx_segment_reduce_backward": (c_int, [c_void_p] * 5 + [c_int64, c_int64, c_int, c_int, c_int, c_void_p,
                                                            c_size_t, c_void_p]),
    "pcx_indexed_segment_reduce_workspace_bytes": (c_size_t, [c_int64, c_int64, c_int, c_int, c_int]),
    "pcx_indexed_segment_reduce": (c_int, [c_void_p] * 4 + [c_int64] * 3 + [c_int] * 3 + [c_void_p, c_size_t,
                                                                                         c_void_p]),
    "pcx_indexed_segment_reduce_backward": (c_int, [c_void_p] * 6 + [c_int64] * 3 + [c_int] * 3
                                            + [c_void_p, c_size_t, c_void_p]),
    "pcx_ragged_layer_norm_workspace_bytes": (c_size_t, [c_int64, c_int64]),
    "pcx_ragged_layer_norm": (c_int, [c_void_p] * 8 + [c_int64, c_int64, c_int, c_double, c_int, c_int, c_void_p,
                                                      c_size_t, c_void_p]),
    "pcx_ragged_layer_norm_backward": (c_int, [c_void_p] * 11 + [c_int64, c_int64, c_int, c_int, c_int, c_void_p,
                                                                c_size_t, c_void_p]),
    "pcx_ragged_group_norm_workspace_bytes": (c_size_t, [c_int64, c_int]),
    "pcx_ragged_group_norm": (c_int, [c_void_p] * 7 + [c_int64, c_int64, c_int, c_int, c_double, c_int, c_void_p,
                                                      c_size_t, c_void_p]),
    "pcx_ragged_group_norm_backward": (c_int, [c_void_p] * 9 + [c_int64, c_int64, c_int, c_int, c_int, c_void_p,
                                                               c_size_t, c_void_p]),
    "pcx_rnet_workspace_bytes": (c_size_t, [c_int64, c_int]),
    "pcx_rnet_far": (c_int, [c_void_p] * 3 + [c_int64, c_void_p, c_void_p]),
    "pcx_rnet_rounds": (c_int, [c_void_p] * 4 + [c_int64, c_int, c_void_p, c_void_p, ctypes.POINTER(ctypes.c_int32),
                                c_void_p, c_size_t, c_void_p]),
    "pcx_seg_offs": (c_int, [c_void_p, c_int64, c_int, c_void_p, c_void_p]),
    "pcx_expand_taps": (c_int, [c_void_p, c_int, c_int64, c_void_p, c_void_p]),
    "pcx_set_radius_predicate": (c_int, [c_int]),
    "pcx_get_radius_predicate": (c_int, []),
    "pcx_radius_workspace_bytes": (c_size_t, [c_int64, c_int64, c_int]),
    "pcx_radius_fill_workspace_bytes": (c_size_t, [c_int64, c_int]),
    "pcx_radius_count": (c_int, [c_void_p] * 4 + [c_int64, c_int64, c_double, c_int, c_int, c_double]
                         + [c_void_p] * 3 + [c_void_p, c_size_t, c_void_p]),
    "pcx_radius_fill": (c_int, [c_void_p, c_void_p, c_int64, c_int64, c_double, c_int, c_int, c_double,
                                c_int64] + [c_void_p] * 5 + [c_void_p, c_size_t, c_void_p, c_size_t, c_void_p]),
    "pcx_radius_taps_supported": (c_int, [c_int]),
    "pcx_radius_taps_workspace_bytes": (c_size_t, [c_int64, c_int64, c_int]),
    "pcx_radius_taps_count": (c_int, [c_void_p] * 4 + [c_int64, c_int64, c_double, c_int, c_int, c_double]
                              + [c_void_p] * 2 + [c_void_p, c_size_t, c_void_p]),
    "pcx_radius_taps_total": (c_int, [c_int64, c_int64, c_int, c_void_p, c_void_p, c_size_t, c_void_p]),
    "pcx_radius_taps_fill": (c_int, [c_void_p] * 3 + [c_int64, c_int64, c_double, c_int, c_int, c_double, c_int64]
                             + [c_void_p] * 4 + [c_void_p, c_size_t, c_void_p]),
    "pcx_grid_sample_workspace_bytes": (c_size_t, [c_int64]),
    "pcx_grid_sample_count": (c_int, [c_void_p, c_void_p, c_int64, c_double, c_void_p, c_void_p, c_size_t,
                                      c_void_p]),
    "pcx_grid_sample_count_samples": (c_int, [c_void_p, c_void_p, c_int64, c_double, ctypes.POINTER(c_int64), c_void_p,
                                              c_size_t, c_void_p]),
    "pcx_sample_sizes": (c_int, [c_void_p, c_int64, c_int64, c_void_p, c_void_p]),
    "pcx_grid_sample_count_ids": (c_int, [c_void_p, c_void_p, c_int64, c_double, ctypes.POINTER(c_int64), c_void_p, c_size_t, c_void_p]),
    "pcx_grid_sample_select_ids": (c_int, [c_void_p, c_void_p, c_int64, c_double, c_int64] + [c_void_p] * 5
                                   + [c_int64, c_void_p, c_size_t, c_void_p]),
    "pcx_grid_sample_select": (c_int, [c_void_p, c_void_p, c_int64, c_double, c_int64] + [c_void_p] * 4
                               + [c_void_p, c_size_t, c_void_p]),
}

_lib = None


def lib():
    """The loaded library; raises if it has not been built."""
    global _lib
    if _lib is None:
        if not os.path.exists(LIB_PATH):
            raise RuntimeError(
                f"{LIB_PATH} is missing: build it with `python -m pointelligence_b200.build` "
                "(the operators have no fallback implementation)")
        handle = ctypes.CDLL(LIB_PATH)
        for name, (res, args) in SIGNATURES.items():
            fn = getattr(handle, name)
            fn.restype = res
            fn.argtypes = args
        _lib = handle
    return _lib


_host = None


def host():
    """The compiled host path (``csrc/host.cpp``) of the hot operators; raises if it has not been built."""
    global _host
    if _host is None:
        lib()
        try:
            from .lib import _pcx_host
        except ImportError as exc:
            raise RuntimeError("pointelligence_b200/lib/_pcx_host.so is missing or does not load: build it with "
                               f"`python -m pointelligence_b200.build` ({exc})") from exc
        _pcx_host.set_hooks(_plan_hook, is_symmetric, _rows_ascend, fullest_tap, _differentiable_backward)
        from .sparse_engines._dispatch_override import current_engine

        _pcx_host.set_engine(current_engine())
        _host = _pcx_host
    return _host


def check(rc):
    if rc == 0:
        return
    msg = lib().pcx_last_error_string().decode("utf-8", "replace")
    raise _STATUS_EXC.get(rc, RuntimeError)(f"{msg} [pcx status {rc}]")


def dtype_code(dtype):
    try:
        return _DTYPES[dtype]
    except KeyError:
        raise TypeError(f"unsupported feature dtype {dtype}; expected float32, float16 or bfloat16")


def require_cuda(*tensors):
    for t in tensors:
        if t is not None and not t.is_cuda:
            raise RuntimeError(
                "pointelligence_b200 operators run on CUDA tensors only (no CPU fallback); "
                f"got a tensor on {t.device}")


def ptr(t):
    return None if t is None else c_void_p(t.data_ptr())


def stream_ptr():
    return c_void_p(torch.cuda.current_stream().cuda_stream)


def workspace(nbytes, device):
    return torch.empty(max(int(nbytes), 256), dtype=torch.uint8, device=device)


# ---------------------------------------------------- geometry beside the features ----
_SIDE_STREAMS = {}
_VALUES = frozenset((type(None), bool, int, float, str))
_overlap = threading.local()


class geometry_overlap:
    """Scope in which the index-building calls of this module (radius search, grid sampling, plan
    building) run on a stream of their own, so that their host hand-overs wait for the geometry
    kernels only and the feature kernels already queued on the caller's stream keep the GPU busy
    meanwhile.  Results are handed to the caller's stream with an event, never with a host wait.

    Contract: inside the scope, every tensor handed to those calls was either complete before the
    scope was entered or is itself the result of one of them (point clouds, sample ids, index
    arrays) -- true for a network that derives its geometry from the input cloud alone.  The side
    stream waits for the caller's stream once, on entry; the caller's stream waits for the side
    stream on exit.  Not re-entrant across devices; nested use on one device is a no-op."""

    def __init__(self, device=None):
        self.device = torch.device("cuda", torch.cuda.current_device()) if device is None else torch.device(device)
        self.owner = False

    def __enter__(self):
        if self.device.type != "cuda" or os.environ.get("PCX_GEOMETRY_OVERLAP", "1") == "0":
            return self
        index = self.device.index if self.device.index is not None else torch.cuda.current_device()
        active = getattr(_overlap, "devices", None)
        if active is None:
            active = _overlap.devices = set()
            _overlap.inside = False
            _overlap.known = {}
        if index in active:
            return self
        if index not in _SIDE_STREAMS:
            _SIDE_STREAMS[index] = torch.cuda.Stream(device=index, priority=-1)
        _SIDE_STREAMS[index].wait_stream(torch.cuda.current_stream(index))
        active.add(index)
        self.owner, self.index = True, index
        return self

    def __exit__(self, *exc):
        if self.owner:
            _overlap.devices.discard(self.index)
            _overlap.known.clear()
            torch.cuda.current_stream(self.index).wait_stream(_SIDE_STREAMS[self.index])
            self.owner = False
        return False


def on_geometry_stream(fn):
    """Decorator of an index-building function (no feature arithmetic inside): when its device is
    inside a ``geometry_overlap`` scope the whole body runs on the side stream, and every tensor it
    returns -- also inside tuples and geometry records such as ``MetaData`` and its parents -- is
    made known to the caller's stream (event wait, allocator bookkeeping)."""
    import functools

    def device_of(values):
        for v in values:
            if isinstance(v, torch.Tensor):
                if v.is_cuda:
                    return v.device
            elif hasattr(v, "points") and isinstance(getattr(v, "points"), torch.Tensor) and v.points.is_cuda:
                return v.points.device
        return None

    def collect(value, out, caller, depth=0):
        if isinstance(value, torch.Tensor):
            if (id(value), caller) not in _overlap.known:      # kept until the scope ends, so that ids stay unique
                _overlap.known[id(value), caller] = value
                out.append(value)
        elif isinstance(value, (tuple, list)):
            for v in value:
                if type(v) not in _VALUES:
                    collect(v, out, caller, depth)
        elif isinstance(value, MvmrPlan):
            out.append(value.buffer)
        elif hasattr(value, "__dataclass_fields__") and depth < 8:
            for v in vars(value).values():
                if type(v) not in _VALUES:
                    collect(v, out, caller, depth + 1)

    @functools.wraps(fn)
    def wrapper(*args, **kwargs):
        active = getattr(_overlap, "devices", None)
        if not active or _overlap.inside:            # no scope, or already on the geometry stream
            return fn(*args, **kwargs)
        dev = device_of(list(args) + list(kwargs.values()))
        if dev is None or dev.index not in active:
            return fn(*args, **kwargs)
        side = _SIDE_STREAMS[dev.index]
        before = host().side_begin(side.stream_id, side.device_index, side.device_type)
        _overlap.inside = True
        try:
            out = fn(*args, **kwargs)
        finally:
            _overlap.inside = False
            host().side_end(*before)
        fresh = []
        collect(out, fresh, before)
        host().record_streams(fresh)
        return out

    return wrapper


def as_i32(t):
    if t is None:
        return None
    return t.contiguous() if t.dtype == torch.int32 else t.to(torch.int32).contiguous()


def device_status(clear=True):
    """Status word set by kernels whose bounded waits ran out (0 = healthy)."""
    out = ctypes.c_uint(0)
    check(lib().pcx_device_status(ctypes.byref(out), 1 if clear else 0, stream_ptr()))
    return int(out.value)


def raise_if_device_reported():
    """Raise ``RuntimeError`` (PCX_E_DEVICE) if a kernel of the library gave up on one of its bounded
    waits since the last check; its result is incomplete.  Called where the host synchronises
    anyway (the geometry hand-overs), so that such a result cannot go unnoticed for long."""
    status = device_status(clear=True)
    if status:
        raise RuntimeError(f"a kernel of the library gave up on a bounded wait (device status word {status:#x}): "
                           "results computed since the last check are incomplete [pcx status -7]")


def launch_count(reset=False):
    """Kernels launched by the library so far (optionally resetting the counter)."""
    return int(lib().pcx_launch_count(1 if reset else 0))


def profile_enable(on=True):
    check(lib().pcx_profile_enable(1 if on else 0))


def profile_records():
    """[(kernel label, milliseconds)] recorded since ``profile_enable(True)``."""
    L = lib()
    out = []
    for i in range(L.pcx_profile_count()):
        name, ms = ctypes.c_char_p(), ctypes.c_float()
        check(L.pcx_profile_get(i, ctypes.byref(name), ctypes.byref(ms)))
        out.append((name.value.decode(), float(ms.value)))
    return out


# ---------------------------------------------------------------- sparse ----
# Engine choice of ``mvmr`` with the automatic engine.  The output-stationary kernel
# (``pcx_mvmr_planned``: accumulators in tensor memory across all taps, every output row written
# once) needs a plan of the rulebook, built once per rulebook and direction and remembered by the
# identity of the index tensors.  Rooms of the benchmark's kind on B200, 27 taps, us per forward
# pass on the scatter kernel / on this one (its plan):
#
#   triplets per row          16 -> 32        64 -> 64      128 -> 128     256 -> 256
#    6.5 (150 000 points)      63 /  31        84 /  49      209 /  96      490 / 212   (179)
#   10.1 (150 000)             85 /  38       114 /  72      295 / 132      705 / 293   (203)
#   13.5 (150 000)            110 /  44       149 /  87      381 / 162      924 / 351   (217)
#   21.9 (300 000)            321 /  97       403 / 215     1175 / 412                  (361)
#    6.3 (600 000)            210 /  89       402 / 158     1054 / 304                  (337)
#   15.3 (20 000)              32 /  27        37 /  35       78 /  51      163 / 105   (144)
#
# It is chosen
#   - from twelve triplets per output row on (the deeper levels of a U-Net, dense scans), and
#   - from four on once the scatter kernel's fp32 accumulator (n_out x width x 4 bytes) outgrows half
#     of the 126 MB L2 and its reductions start to go to HBM: wide layers and large clouds.
# Below that a pass gains less than the plan costs, and a rulebook may be used once.  The kernel also
# rounds the sums of (row, tap) buckets to 16 bits, which the scatter kernel does not: the lines are
# not moved for time alone.  Single-tap rulebooks (nothing to keep across taps) and rulebooks
# that are thin in tap space (fewer than 0.18 triplets per output row and tap: tiles mostly padding)
# stay on the scatter kernel.  125 taps, 130 000 points, the same pairs of widths:
#
#   17.5 per row, 0.14 per tap  123 / 119      157 / 250     413 / 497     1009 / 1215  (307)
#   39.6, 0.32                  264 / 158      306 / 327     878 / 652                  (442)
ENGINE_PLANNED = 3
_PLANNED_DENSE_RATIO = float(os.environ.get("PCX_PLANNED_DENSE_RATIO", "12"))   # triplets per output row: always planned
_PLANNED_MIN_RATIO = float(os.environ.get("PCX_PLANNED_MIN_RATIO", "4"))        # ... planned when the accumulator is large
_PLANNED_MIN_ACC_BYTES = int(os.environ.get("PCX_PLANNED_MIN_ACC_BYTES", str(64 << 20)))
_PLANNED_MIN_TAP_FILL = float(os.environ.get("PCX_PLANNED_MIN_TAP_FILL", "0.18"))  # triplets per output row and tap
_PLANNED_ENABLED = os.environ.get("PCX_PLANNED", "1") != "0"


def _planned_pays(T, n_out, outw, K):
    if not _PLANNED_ENABLED or K <= 1 or n_out <= 0:
        return False
    ratio = T / n_out
    if ratio / K < _PLANNED_MIN_TAP_FILL:
        return False
    return ratio >= _PLANNED_DENSE_RATIO or (ratio >= _PLANNED_MIN_RATIO and n_out * outw * 4 >= _PLANNED_MIN_ACC_BYTES)


# Grouped layers and rows wider than 256 channels go to the output-stationary kernel with its bucket sums in two parts
# (bf16 alone): as exact as the scatter kernels once a row is rounded (relative error against fp64 1.65e-3 on both over all
# shapes below; operands of one sign 1.6603e-3 on both at 64 -> 384, 1.6622e-3 and 1.6619e-3 at 1024 -> 384), for a
# contraction twice as long.  One pass on a built plan, scatter / split, and the plan, us:
#
#   triplets per row (rows)     512 -> 512    128 -> 384    32 -> 512    2 x 128 -> 128    plan
#   33.8 (942)                    81 /  50      35 / 30       38 / 27        30 /  27        74
#   11.4 (5000)                  123 / 122      54 / 48       62 / 35        42 /  42       128
#    7.3 (15 000)                217 / 291      82 / 83       96 / 43        57 /  78       135
#   25.4 (15 000)                672 / 350     232 / 95      277 / 49       150 / 100       139
#
# (these and below without the scatter kernels behind, which return at once where all operands are finite: 9 us more.)
# It is chosen where the scatter kernel's fp32 reductions (triplets x width x 4 bytes) are half a gigabyte and the two-part
# sums stay within 4 GB.  On a plan that exists it would pay far below that (the first line: 65 and 390 MB); the line is
# for rulebooks that are used once or twice.  At half a gigabyte a pass over a dense rulebook gains a quarter of a plan
# (2 x 64 -> 64, 22.5 triplets a row: 180 / 128, plan 190) to twice one (1024 -> 288, 15.7: 1074 / 777, plan 163).  Thin
# rulebooks gain less, and a contraction much longer than the row loses on a plan that exists, too, since the low parts are
# multiplied tile by tile whether or not a tile holds a sum.  Below six triplets a row, scatter / split / plan:
#
#   4.9 (60 000)     512 -> 512    514 /  462 / 163 (574 MB)    1024 -> 512   942 /  907     32 -> 512  260 /  75
#   5.0 (120 000)    512 -> 512   1037 /  858 / 182 (1182 MB)   1024 -> 512  1914 / 1683     1024 -> 288  1439 / 1498 (665 MB)
#   6.8 (60 000)     512 -> 512    679 /  519 / 168 (800 MB)    1024 -> 512  1274 / 1034     128 -> 384  273 / 145
#
# There it takes a gigabyte, and a contraction of at most twice the row.  The input gradient of an up-sampling layer 384 ->
# 128 with 134 triplets a row (18.9 M) took 10.1 ms on the scatter kernel; the training step around it went from 113.0 to
# 104.7 ms, its plan included.
_SPLIT_MIN_REDUCED_BYTES, _SPLIT_MAX_SCRATCH_BYTES = 512 << 20, 4 << 30


def _split_pays(T, n_out, outw, inw, K):
    thin = T < 6 * n_out
    if thin and inw > 2 * outw:
        return False
    return (T * outw * 4 >= _SPLIT_MIN_REDUCED_BYTES * (2 if thin else 1)
            and min(T // 2, n_out * K) * inw * 4 <= _SPLIT_MAX_SCRATCH_BYTES)


_PLAN_WAIT_SECONDS = 30.0   # for a plan that is being built on another stream


class MvmrPlan:
    """A rulebook regrouped for the output-stationary MVMR kernel (``pcx_mvmr_plan_build``).

    Holds the device buffer and the sizes it was built for.  A plan belongs to one rulebook,
    one direction (which index is scattered) and one ``group_blocks`` value.
    """

    __slots__ = ("buffer", "T", "K", "n_out", "group_blocks", "_multi", "_word", "_stream", "__weakref__")

    def __init__(self, buffer, T, K, n_out, group_blocks, multi, word=None, stream=None):
        self.buffer, self.T, self.K, self.n_out, self.group_blocks = buffer, T, K, n_out, group_blocks
        self._multi, self._word, self._stream = multi, word, stream

    @property
    def multi_buckets(self):
        """(row, tap) buckets with several triplets; a bound while the plan of an ordered rulebook is being built."""
        word = self._word                # threads may share the plan: one of them drops the word
        if word is not None:
            n = host().peek(word)
            if n == -1 and torch.cuda.current_stream(self.buffer.device) != self._stream:
                # another stream than the one the plan is built on: wait for the build, without a call that a stream
                # under capture refuses
                give_up = time.monotonic() + _PLAN_WAIT_SECONDS
                while n == -1:
                    if time.monotonic() > give_up:
                        raise RuntimeError("a plan was not ready after "
                                           f"{_PLAN_WAIT_SECONDS:g} s [pcx status -7]")
                    time.sleep(0)
                    n = host().peek(word)
            if n == -2:
                raise RuntimeError("a plan was built for rows that ascend inside every tap, and these do not")
            if n >= 0:
                self._multi, self._word = n, None
        return self._multi

    def views(self):
        """The plan's arrays as tensors (for tests): perm, tile_offs, entries (T, 2), group_order."""
        nblocks = (self.n_out + 127) // 128
        ngroups = (nblocks + self.group_blocks - 1) // self.group_blocks

        def up(n):
            return (n + 255) // 256 * 256

        buf, off, out = self.buffer, 0, {}
        for name, count, dtype, width in (("ctrl", 64, torch.int32, 4), ("perm", nblocks * 128, torch.int32, 4),
                                          ("tile_offs", nblocks * self.K + 1, torch.int32, 4),
                                          ("entries", max(self.T, 1) * 2, torch.int32, 4),
                                          ("group_order", max(ngroups, 1), torch.int32, 4),
                                          ("tile_rows", nblocks * self.K * 128, torch.int32, 4),
                                          ("buckets", (self.T // 2 + 1) * 2, torch.int32, 4)):
            out[name] = buf[off:off + count * width].view(dtype)
            off += up(count * width)
        out["entries"] = out["entries"][: self.T * 2].view(-1, 2)
        out["group_order"] = out["group_order"][:ngroups]
        out["tile_rows"] = out["tile_rows"].view(-1, 128)
        out["buckets"] = out["buckets"].view(-1, 2)[: self.multi_buckets]
        return out


def plan_group_blocks(out_width):
    """Blocks of 128 output rows that share the weight tiles they stream, for rows of ``out_width`` channels."""
    width = min(int(out_width), 256)
    blocks = _GROUP_BLOCKS.get(width)
    if blocks is None:
        blocks = _GROUP_BLOCKS[width] = int(lib().pcx_mvmr_plan_group_blocks(width))
    return blocks


_GROUP_BLOCKS = {}


def padded_width(width):
    """Channels the tensor engines work on for a row of ``width``: parts of at most 256, multiples of 16."""
    unit = 16 * ((width + 255) // 256)
    return (width + unit - 1) // unit * unit


def planned_supported(weight, feat, gather, scatter, seg_offs, n_out, transpose):
    """Whether the automatic choice may give this call to the output-stationary kernel (fp16 / bf16, one group,
    tap-sorted int32 triplets, channel counts that need no padding, output rows of at most 256 channels).  Asked for
    by name it takes grouped and wider layers too."""
    K, G, C, M = weight.shape
    inw, outw = (M, C) if transpose else (C, M)
    if G != 1 or seg_offs is None or feat.dtype not in (torch.float16, torch.bfloat16) or n_out <= 0:
        return False
    if inw != padded_width(inw) or outw != padded_width(outw) or outw > 256 or inw > 1024 or K > 512:
        return False
    T = gather.numel()
    nblocks = (int(n_out) + 127) // 128
    return T < 2 ** 31 and nblocks * K * 128 <= 2 ** 32


def _split_supported(weight, gather, seg_offs, n_out, transpose):
    """Whether the automatic choice may give this call to the output-stationary kernel with its sums in two parts."""
    K, G, C, M = weight.shape
    inw, outw = (M, C) if transpose else (C, M)
    if seg_offs is None or weight.dtype != torch.bfloat16 or K <= 1 or K > 512 or n_out <= 0 or not (G > 1 or outw > 256):
        return False
    if inw != padded_width(inw) or outw != padded_width(outw) or inw > 1024 or G * inw > 2048 or G * ((inw + 255) // 256) * ((outw + 255) // 256) > 64:
        return False
    return gather.numel() < 2 ** 31 and (int(n_out) + 127) // 128 * K * 128 <= 2 ** 32


@on_geometry_stream
def mvmr_plan(scatter, gather, seg_offs, K, n_out, group_blocks):
    """Build the plan of a tap-sorted rulebook: ``scatter`` indexes the rows that are summed
    into (n_out of them), ``gather`` the rows that are read."""
    require_cuda(scatter, gather, seg_offs)
    T = scatter.numel()
    ordered = T <= _NO_WAIT_TRIPLETS and _rows_ascend(scatter, gather, seg_offs, K)
    buf, multi, word = host().plan_build(scatter, gather, seg_offs, int(K), int(n_out), int(group_blocks), ordered)
    return MvmrPlan(buf, T, int(K), int(n_out), int(group_blocks), multi, word)


# Rulebooks of the geometry path up to this size get their plan without a wait (150 us each where a network of
# 40 000 points builds eleven per pass).  Until the count of multi-triplet buckets has arrived, passes reserve scratch
# for its bound, half the triplets: at 2^20 triplets and 256 channels 256 MB.
_NO_WAIT_TRIPLETS = 1 << 20

_PLAN_CACHE = {}
_PLAN_CACHE_MAX = 64
_BUILT = {}


def _stamp(*tensors):
    """What tells whether the tensors were written to since; None for tensors of inference mode, which do not say (and
    raise when they are asked): nothing is remembered about those."""
    try:
        return tuple([t._version for t in tensors])
    except RuntimeError:
        return None


def mark_built(i, j, seg_offs, K, symmetric, fullest=None):
    """Record that ``(i, j)`` cut into ``K`` taps by ``seg_offs`` come from the geometry path: i ascends inside every
    tap.  ``symmetric``: the rulebook is its own mirror image: with ``(i, j, k)`` it holds ``(j, i, K - 1 - k)``.
    True for a self-search (queries are the points): the distance is symmetric and the tap of the opposite offset is
    the mirrored tap.  The input gradient of such a layer is then a forward pass over the SAME rulebook with the taps
    of the weight reversed, so it needs no plan of its own (``tig_grad_input``).  ``fullest``: triplets of the fullest
    tap, where they were counted.  Remembered by tensor identity, like the plans."""
    import weakref

    for key in [key for key, (refs, *_) in _BUILT.items() if any(r() is None for r in refs)]:
        _BUILT.pop(key, None)
    stamp = _stamp(i, j, seg_offs)
    if stamp is not None:
        _BUILT[(i.data_ptr(), j.data_ptr(), i.numel())] = (tuple(weakref.ref(t) for t in (i, j, seg_offs)), stamp,
                                                           int(K), bool(symmetric), fullest)


def _built(i, j):
    """What ``mark_built`` recorded for these tensors (None: nothing, or they were written to since)."""
    hit = _BUILT.get((i.data_ptr(), j.data_ptr(), i.numel()))
    if hit is None:
        return None
    refs, stamp = hit[:2]
    return hit if refs[0]() is i and refs[1]() is j and stamp[:2] == _stamp(i, j) else None


def _rows_ascend(i, j, seg_offs, K):
    """Whether i is known to ascend inside every tap.  That is a property of the cut into taps too: where taps are
    merged, rows fall at the seams."""
    hit = _built(i, j)
    return hit is not None and hit[0][2]() is seg_offs and hit[1][2:] == _stamp(seg_offs) and hit[2] == int(K)


def fullest_tap(i, j, seg_offs, K):
    """Triplets of the fullest tap of a rulebook, or of the mirrored one of an up-sampling layer; None where nobody counted."""
    for a, b in ((i, j), (j, i)):
        hit = _built(a, b)
        if hit is not None and hit[0][2]() is seg_offs and hit[1][2:] == _stamp(seg_offs) and hit[2] == int(K):
            return hit[4]
    return None


def is_symmetric(i, j, K=None):
    hit = _built(i, j)
    return (hit is not None and hit[3] and (K is None or hit[2] == int(K))
            and os.environ.get("PCX_SYMMETRIC_DGRAD", "1") != "0")


def _plan_key(scatter, gather, seg_offs, K, n_out, group_blocks):
    return (scatter.data_ptr(), gather.data_ptr(), seg_offs.data_ptr(), scatter.numel(), int(K), int(n_out),
            int(group_blocks))


def _remembered_plan(key, scatter, gather, seg_offs):
    hit = _PLAN_CACHE.get(key)
    if hit is not None:
        (i, j, seg), stamp, value = hit
        if i() is scatter and j() is gather and seg() is seg_offs and stamp == _stamp(scatter, gather, seg_offs):
            return value
    return None


def cached_mvmr_plan(scatter, gather, seg_offs, K, n_out, group_blocks):
    """``mvmr_plan`` remembered by the identity (and version) of the index tensors, so that every
    layer and every step that shares a rulebook builds its plan once."""
    import weakref

    key = _plan_key(scatter, gather, seg_offs, K, n_out, group_blocks)
    value = _remembered_plan(key, scatter, gather, seg_offs)
    if value is not None:
        return value
    stamp = _stamp(scatter, gather, seg_offs)
    if stamp is None:
        return mvmr_plan(scatter, gather, seg_offs, K, n_out, group_blocks)
    value = mvmr_plan(scatter, gather, seg_offs, K, n_out, group_blocks)
    value._stream = torch.cuda.current_stream(scatter.device)
    for k in [k for k, (refs, _, _) in _PLAN_CACHE.items() if any(r() is None for r in refs)]:
        _PLAN_CACHE.pop(k, None)
    if len(_PLAN_CACHE) >= _PLAN_CACHE_MAX:
        for k in list(_PLAN_CACHE)[: _PLAN_CACHE_MAX // 2]:
            _PLAN_CACHE.pop(k, None)
    _PLAN_CACHE[key] = (tuple(weakref.ref(t) for t in (scatter, gather, seg_offs)), stamp, value)
    return value


_CAPTURED_PLANS = {}


def _keep_for_graph(plan, scatter):
    """A pass that is being captured reads the plan at every replay: it lives as long as the index tensor it was built
    from, which is what the owner of a graph keeps anyway, whatever becomes of it in the cache."""
    import weakref

    if plan not in _CAPTURED_PLANS:
        _CAPTURED_PLANS[plan] = weakref.ref(scatter, lambda _, kept=_CAPTURED_PLANS: kept.pop(plan, None))


def mvmr_planned(weight, feat, plan, transpose, split=False):
    """``out[scatter[t]] += feat[gather[t]] @ W[tap(t)]`` for the rulebook of ``plan``
    (``transpose``: use W^T; ``split``: bucket sums in two parts); returns (plan.n_out, G * out_width) in feat.dtype."""
    require_cuda(weight, feat)
    K, G, C, M = weight.shape
    assert K == plan.K and weight.dtype == feat.dtype, (weight.shape, plan.K, weight.dtype, feat.dtype)
    return host().planned(weight, feat, plan.buffer, plan.group_blocks, plan.multi_buckets, plan.T, plan.n_out,
                          bool(transpose), bool(split))


def debug_wait_runs_out(limit_ns=1_000_000):
    """Launch the test kernel whose bounded wait runs out after ``limit_ns``."""
    check(lib().pcx_debug_wait_runs_out(int(limit_ns), stream_ptr()))


def mvmr(weight, feat, gather, scatter, seg_offs, tap_idx, n_out, transpose, engine=ENGINE_AUTO):
    """``out[scatter[t]] += feat[gather[t]] @ W[tap(t)]`` (``transpose``: use W^T).

    weight (K,G,C,M); feat (n_feat, G*inw); returns (n_out, G*outw) in feat.dtype.  With the
    automatic engine, wide rows and dense neighbourhoods take the output-stationary kernel
    (``ENGINE_PLANNED`` forces it), everything else the scatter engines of ``pcx_mvmr``.
    """
    return host().mvmr(weight, feat, gather, scatter, seg_offs, tap_idx, int(n_out), bool(transpose), int(engine))


def _plan_hook(scatter, gather, seg_offs, K, n_out, outw, inw, forced, split=False, capturing=False):
    """Asked by the host path for every pass the output-stationary kernel could take: the plan to run
    (buffer, blocks per group, multi-triplet buckets) or None for the scatter engine."""
    T, blocks = gather.numel(), plan_group_blocks(outw)
    if not forced and not _planned_pays(T, n_out, outw, K):
        return None
    # Wide and grouped layers are captured on the scatter kernels, whether or not a plan exists: these read the caller's
    # tensors alone, so that a replay follows what is written into them.
    if split and (capturing or not _split_pays(T, n_out, outw, inw, K)):
        return None
    plan = _remembered_plan(_plan_key(scatter, gather, seg_offs, K, n_out, blocks), scatter, gather, seg_offs)
    if plan is None:
        if not forced and (scatter.is_inference() or gather.is_inference() or seg_offs.is_inference()):
            return None    # (a plan of inference tensors cannot be remembered, and one per pass does not pay)
        try:
            plan = cached_mvmr_plan(scatter, gather, seg_offs, K, n_out, blocks)
        except torch.OutOfMemoryError:
            if not split:
                raise
            return None    # wide and grouped layers fit without a plan
    if capturing:
        _keep_for_graph(plan, scatter)
    return plan.buffer, plan.group_blocks, plan.multi_buckets


def _differentiable_backward(weight, feat, grad, i, j, seg_offs, n_out, n_in, K, cover_out, cover_in, want_w, want_x,
                             want_b):
    """Gradients of a convolution as differentiable operators (``create_graph=True``)."""
    from .sparse_engines import tig

    index = tig.TigIndex.from_flat(i, j, seg_offs, n_out, n_in, K, cover_out, cover_in)
    gw = tig.tig_grad_weight(feat, grad, index, weight.shape).to(weight.dtype) if want_w else None
    gf = tig.tig_grad_input(weight, grad, index).to(feat.dtype) if want_x else None
    return gw, gf, (grad.sum(0) if want_b else None)


def prepare_mvmr(weight, gather, scatter, seg_offs, n_out, transpose=False):
    """Build (and cache) now what ``mvmr`` with the automatic engine would build on its first call
    for this rulebook -- the plan of the output-stationary kernel, whose construction may end with a
    host hand-over -- so that the feature pass itself is kernels only.  Returns True when a plan
    was prepared, False when the policy keeps the scatter engines (which need no preparation)."""
    K, G, C, M = weight.shape
    n_out = int(n_out)
    inw, outw = (G * M, G * C) if transpose else (G * C, G * M)
    if gather is None or not gather.is_cuda:
        return False
    if not planned_supported(weight, weight, gather, scatter, seg_offs, n_out, transpose) and not (
            _split_supported(weight, gather, seg_offs, n_out, transpose) and _split_pays(gather.numel(), n_out, outw, inw, K)):
        return False
    if not _planned_pays(gather.numel(), n_out, outw, K) or _stamp(scatter, gather, seg_offs) is None:
        return False
    cached_mvmr_plan(scatter, gather, seg_offs, K, n_out, plan_group_blocks(outw))
    return True


def vvor(a, a_idx, b, b_idx, seg_offs, o_idx, n_o, engine=ENGINE_AUTO):
    """``out[o[t], g, m, c] += a[a_idx[t], g, m] * b[b_idx[t], g, c]``.

    a (n_a, G, Ma); b (n_b, G, Cb); returns (n_o, G, Ma, Cb) in a.dtype.
    """
    return host().vvor(a, a_idx, b, b_idx, seg_offs, o_idx, int(n_o), int(engine))


def vvor_static_scratch(a, a_idx, b, b_idx, seg_offs, out):
    """VVOR into the caller's ``out`` (n_o, G, Ma, Cb) using the library's built-in
    scratch array: nothing is allocated by the call, here or in the library.
    For embedders that cannot allocate device memory at the call site; see
    ``pcx_vvor_static_scratch`` in the header for the size limits and for the
    rule that calls must not overlap on the GPU."""
    require_cuda(a, b, a_idx, b_idx, seg_offs, out)
    code = dtype_code(a.dtype)
    for t in (a, b, out):
        assert t.is_contiguous() and t.dtype == a.dtype
    assert a_idx.dtype == torch.int32 and b_idx.dtype == torch.int32 and seg_offs.dtype == torch.int64
    n_o, G, Ma, Cb = out.shape
    with torch.cuda.device(a.device):
        check(lib().pcx_vvor_static_scratch(ptr(a), ptr(a_idx), ptr(b), ptr(b_idx), ptr(seg_offs), ptr(out),
                                            a_idx.numel(), a.shape[0], b.shape[0], n_o, G, Ma, Cb, code,
                                            stream_ptr()))
    return out


REDUCE_OPS = {"sum": 0, "mean": 1, "max": 2, "min": 3}


def segment_reduce(x, lengths, op):
    """``out[s] = op`` over the ``lengths[s]`` consecutive rows of segment s; x (N, C) -> (S, C)."""
    require_cuda(x, lengths)
    x = x.contiguous()
    lengths = lengths.to(torch.int64).contiguous()
    N, C = x.shape
    S = lengths.numel()
    out = torch.empty((S, C), dtype=x.dtype, device=x.device)
    L = lib()
    with torch.cuda.device(x.device):
        ws = workspace(L.pcx_segment_reduce_workspace_bytes(S, C), x.device)
        check(L.pcx_segment_reduce(ptr(x), ptr(lengths), ptr(out), N, S, C, op, dtype_code(x.dtype), ptr(ws),
                                   ws.numel(), stream_ptr()))
    return out


def segment_reduce_backward(grad_out, x, out, lengths, op, n_rows):
    require_cuda(grad_out, lengths)
    grad_out = grad_out.contiguous()
    if op >= 2:   # max / min compare x with out: both are read row-major in the gradient's element type
        assert x.dtype == grad_out.dtype and out.dtype == grad_out.dtype, (x.dtype, out.dtype, grad_out.dtype)
        x, out = x.contiguous(), out.contiguous()
    lengths = lengths.to(torch.int64).contiguous()
    S, C = grad_out.shape
    grad_x = torch.empty((n_rows, C), dtype=grad_out.dtype, device=grad_out.device)
    L = lib()
    with torch.cuda.device(grad_out.device):
        ws = workspace(L.pcx_segment_reduce_workspace_bytes(S, 1), grad_out.device)
        check(L.pcx_segment_reduce_backward(ptr(grad_out), ptr(x), ptr(out), ptr(lengths), ptr(grad_x), n_rows, S, C,
                                            op, dtype_code(grad_out.dtype), ptr(ws), ws.numel(), stream_ptr()))
    return grad_x


def indexed_segment_reduce(x, indices, lengths, op):
    """``y[k] = op`` over ``x[indices[e]]`` for the ``lengths[k]`` consecutive entries of list k."""
    require_cuda(x, indices, lengths)
    x = x.contiguous()
    indices = as_i32(indices)
    lengths = lengths.to(torch.int64).contiguous()
    n_x, C = x.shape
    K = lengths.numel()
    y = torch.empty((K, C), dtype=x.dtype, device=x.device)
    L = lib()
    code = dtype_code(x.dtype)
    with torch.cuda.device(x.device):
        ws = workspace(L.pcx_indexed_segment_reduce_workspace_bytes(K, n_x, C, code, 0), x.device)
        check(L.pcx_indexed_segment_reduce(ptr(x), ptr(indices), ptr(lengths), ptr(y), n_x, indices.numel(), K, C, op,
                                           code, ptr(ws), ws.numel(), stream_ptr()))
    return y


def indexed_segment_reduce_backward(grad_y, x, y, indices, lengths, op, n_x):
    require_cuda(grad_y, indices, lengths)
    grad_y = grad_y.contiguous()
    indices = as_i32(indices)
    lengths = lengths.to(torch.int64).contiguous()
    K, C = grad_y.shape
    grad_x = torch.empty((n_x, C), dtype=grad_y.dtype, device=grad_y.device)
    L = lib()
    code = dtype_code(grad_y.dtype)
    with torch.cuda.device(grad_y.device):
        ws = workspace(L.pcx_indexed_segment_reduce_workspace_bytes(K, n_x, C, code, 1), grad_y.device)
        check(L.pcx_indexed_segment_reduce_backward(ptr(grad_y), ptr(x), ptr(y), ptr(indices), ptr(lengths),
                                                    ptr(grad_x), n_x, indices.numel(), K, C, op, code, ptr(ws),
                                                    ws.numel(), stream_ptr()))
    return grad_x


def _f32_or_none(t):
    return None if t is None else t.detach().to(torch.float32).contiguous()


def ragged_group_norm(x, lengths, weight, bias, groups, eps):
    """Group norm per sample (``groups`` blocks of consecutive channels; ``groups == C`` is the
    instance norm); returns ``(y, mean, rstd)`` with the statistics as (S * groups,) fp32."""
    require_cuda(x, lengths, weight, bias)
    x = x.contiguous()
    lengths = lengths.to(torch.int64).contiguous()
    weight, bias = _f32_or_none(weight), _f32_or_none(bias)
    N, C = x.shape
    S, G = lengths.numel(), int(groups)
    y = torch.empty_like(x)
    mean = torch.empty(S * G, dtype=torch.float32, device=x.device)
    rstd = torch.empty(S * G, dtype=torch.float32, device=x.device)
    L = lib()
    with torch.cuda.device(x.device):
        ws = workspace(L.pcx_ragged_group_norm_workspace_bytes(S, G), x.device)
        check(L.pcx_ragged_group_norm(ptr(x), ptr(lengths), ptr(weight), ptr(bias), ptr(y), ptr(mean), ptr(rstd),
                                      N, S, C, G, float(eps), dtype_code(x.dtype), ptr(ws), ws.numel(), stream_ptr()))
    return y, mean, rstd


def ragged_group_norm_backward(grad_y, x, lengths, weight, mean, rstd, groups, want_affine):
    """Returns ``(grad_x, grad_weight|None, grad_bias|None)`` (affine gradients in fp32)."""
    require_cuda(grad_y, x, lengths)
    grad_y, x = grad_y.contiguous(), x.contiguous()
    lengths = lengths.to(torch.int64).contiguous()
    weight = _f32_or_none(weight)
    N, C = x.shape
    S, G = lengths.numel(), int(groups)
    grad_x = torch.empty_like(x)
    gw = torch.empty(C, dtype=torch.float32, device=x.device) if want_affine else None
    gb = torch.empty(C, dtype=torch.float32, device=x.device) if want_affine else None
    L = lib()
    with torch.cuda.device(x.device):
        ws = workspace(L.pcx_ragged_group_norm_workspace_bytes(S, G), x.device)
        check(L.pcx_ragged_group_norm_backward(ptr(grad_y), ptr(x), ptr(lengths), ptr(weight), ptr(mean), ptr(rstd),
                                               ptr(grad_x), ptr(gw), ptr(gb), N, S, C, G, dtype_code(x.dtype), ptr(ws),
                                               ws.numel(), stream_ptr()))
    return grad_x, gw, gb


def seg_offs_from_sorted(idx_sorted, K):
    require_cuda(idx_sorted)
    idx = as_i32(idx_sorted)
    out = torch.empty(int(K) + 1, dtype=torch.int64, device=idx.device)
    with torch.cuda.device(idx.device):
        check(lib().pcx_seg_offs(ptr(idx), idx.numel(), int(K), ptr(out), stream_ptr()))
    return out


def expand_taps(seg_offs, K, T):
    require_cuda(seg_offs)
    out = torch.empty(int(T), dtype=torch.int32, device=seg_offs.device)
    with torch.cuda.device(seg_offs.device):
        check(lib().pcx_expand_taps(ptr(seg_offs), int(K), int(T), ptr(out), stream_ptr()))
    return out


def rnet_select(points, centres, centre_of, neighbors, offsets, source, rounds_per_call=4):
    """Residual R-net over ``points`` (n, 3): returns ``(chosen bool (n,), rounds)``.

    ``neighbors`` / ``offsets``: query-major neighbour lists within R (self included);
    ``centres[centre_of[v]]`` is the initial centre of v's stride cell; ``source`` breaks ties.
    The host sees the device once per ``rounds_per_call`` rounds."""
    require_cuda(points, centres, centre_of, neighbors, offsets, source)
    dev, n = points.device, points.shape[0]
    points, centres = points.contiguous().float(), centres.contiguous().float()
    centre_of, neighbors = centre_of.to(torch.int64).contiguous(), neighbors.to(torch.int64).contiguous()
    offsets, source = offsets.to(torch.int64).contiguous(), source.to(torch.int64).contiguous()
    far = torch.empty(n, dtype=torch.float32, device=dev)
    active = torch.ones(n, dtype=torch.uint8, device=dev)
    chosen = torch.zeros(n, dtype=torch.uint8, device=dev)
    L = lib()
    rounds = 0
    with torch.cuda.device(dev):
        check(L.pcx_rnet_far(ptr(points), ptr(centres), ptr(centre_of), n, ptr(far), stream_ptr()))
        ws = workspace(L.pcx_rnet_workspace_bytes(n, rounds_per_call), dev)
        remaining = (ctypes.c_int32 * rounds_per_call)()
        for _ in range(n + 1):           # every productive round retires at least one point
            check(L.pcx_rnet_rounds(ptr(neighbors), ptr(offsets), ptr(far), ptr(source), n, rounds_per_call,
                                    ptr(active), ptr(chosen), remaining, ptr(ws), ws.numel(), stream_ptr()))
            left = list(remaining)
            if 0 in left:
                rounds += left.index(0) + 1
                break
            rounds += rounds_per_call
        else:
            raise RuntimeError("full-cover R-net selector made no progress")
    return chosen.bool(), rounds


# -------------------------------------------------------------- geometry ----
@on_geometry_stream
def radius_search(points, queries, radius, point_sample, query_sample, distance_type,
                  kernel_size=0, kernel_grid_size=0.0, return_distances=False, want_k=False):
    """Sorted-grid fixed-radius search.

    ``kernel_size == 0``: returns ``(neighbors int64, num_neighbors int64, distances|None)``.
    ``kernel_size > 0``: returns ``(i int32, j int32, k int32|None, seg_offs int64, num_neighbors int64)``.
    Inputs must be non-empty fp32 (P,3)/(Q,3) CUDA tensors.
    """
    require_cuda(points, queries, point_sample, query_sample)
    dev = points.device
    if takes_taps(kernel_size):
        return radius_taps(points, queries, radius, point_sample, query_sample, distance_type, kernel_size, kernel_grid_size, want_k)
    points, queries = points.contiguous(), queries.contiguous()
    ps = as_i32(point_sample)
    qs = ps if query_sample is point_sample else as_i32(query_sample)
    P, Q = points.shape[0], queries.shape[0]
    L = lib()
    k3 = kernel_size ** 3
    with torch.cuda.device(dev):
        ws = workspace(L.pcx_radius_workspace_bytes(P, Q, kernel_size), dev)
        num_neighbors = torch.empty(Q, dtype=torch.int64, device=dev)
        seg = torch.empty(k3 + 1, dtype=torch.int64, device=dev) if kernel_size > 0 else None
        total = c_int64(0)
        check(L.pcx_radius_count(ptr(points), ptr(queries), ptr(ps), ptr(qs), P, Q, float(radius),
                                 distance_type, kernel_size, float(kernel_grid_size), ptr(num_neighbors),
                                 ptr(seg), ctypes.byref(total), ptr(ws), ws.numel(), stream_ptr()))
        total = int(total.value)
        raise_if_device_reported()   # the count above was a host hand-over: the stream is idle
        if kernel_size == 0:
            neighbors = torch.empty(total, dtype=torch.int64, device=dev)
            dist = torch.empty(total, dtype=torch.float32, device=dev) if return_distances else None
            check(L.pcx_radius_fill(ptr(points), ptr(queries), P, Q, float(radius), distance_type, 0, 0.0,
                                    total, ptr(neighbors), ptr(dist), None, None, None, ptr(ws), ws.numel(),
                                    None, 0, stream_ptr()))
            return neighbors, num_neighbors, dist
        if total > 2 ** 31 - 1:
            raise RuntimeError("prepared kernel-segment output currently requires fewer "
                               f"than 2^31 edges; got {total}")
        out_i = torch.empty(total, dtype=torch.int32, device=dev)
        out_j = torch.empty(total, dtype=torch.int32, device=dev)
        out_k = torch.empty(total, dtype=torch.int32, device=dev) if want_k else None
        ws2 = workspace(L.pcx_radius_fill_workspace_bytes(total, kernel_size), dev)
        check(L.pcx_radius_fill(ptr(points), ptr(queries), P, Q, float(radius), distance_type, kernel_size,
                                float(kernel_grid_size), total, None, None, ptr(out_i), ptr(out_j), ptr(out_k),
                                ptr(ws), ws.numel(), ptr(ws2), ws2.numel(), stream_ptr()))
    return out_i, out_j, out_k, seg, num_neighbors


# Largest pairs-per-query ratio seen per (kernel_size, distance_type, radius) -- one entry per level of a
# network: sizes the edge buffers of the next such search so that it needs one host hand-over, not two.
_TAPS_RATIO = {}


def takes_taps(kernel_size):
    """Whether the tap-segmented search serves this kernel (and is not switched off)."""
    return (kernel_size > 0 and lib().pcx_radius_taps_supported(kernel_size)
            and os.environ.get("PCX_RADIUS_TAPS", "1") != "0")


def radius_taps(points, queries, radius, ps, qs, distance_type, kernel_size, kernel_grid_size, want_k):
    """Tap-segmented search through ``pcx_radius_taps_*``: the pairs are written into buffers sized
    from the density of earlier searches (exactly sized after a counted first call or when the
    estimate turns out too small) and returned as views of the first ``total`` entries."""
    ratio_key = (kernel_size, distance_type, float(radius))
    ratio = _TAPS_RATIO.get(ratio_key)
    i, j, k, seg, num_neighbors, n, lonely, status, fullest = host().radius_taps(
        points, queries, float(radius), ps, qs, distance_type, kernel_size, float(kernel_grid_size), want_k,
        -1.0 if ratio is None else ratio)
    if status:                 # the hand-over of the fill pass brought the status word along
        raise_if_device_reported()
    if len(_TAPS_RATIO) > 256:
        _TAPS_RATIO.clear()
    _TAPS_RATIO[ratio_key] = max(ratio or 0.0, n / queries.shape[0])
    num_neighbors.pcx_counted = lonely, fullest   # queries without neighbour, pairs of the fullest tap: spares the caller passes over the pairs
    return i, j, k, seg, num_neighbors


@on_geometry_stream
def grid_sample_center_nearest(points, cell, sample, return_mapping):
    """Returns ``(indices int64 (S,), points_f (S,3), sample_f (S,)|None, mapping int64|None)``; ``sample_f`` in the type
    of int32 and int64 ids, in int32 for others."""
    require_cuda(points, sample)
    indices, out, out_sample, mapping, sizes = host().grid_sample(points, float(cell), sample, bool(return_mapping))
    if sizes is not None:
        out_sample.pcx_sample_sizes = sizes     # spares the caller a histogram and its hand-over
    return indices, out, out_sample, mapping
