"""Batched device entry points over torch CUDA tensors.

Thin wrappers that hand raw device pointers and the current CUDA stream to the
C ABI (include/habitat_b200.h).  torch is used for device memory and streams
only; all arithmetic happens in the library's sm_100a kernels.
"""
import ctypes
import math
import os
from dataclasses import dataclass
from typing import Optional, Sequence

import numpy as np
import torch

from habitat_b200 import _native


def _require_cuda(t, dtype, name):
    if not isinstance(t, torch.Tensor) or not t.is_cuda:
        raise TypeError("%s must be a CUDA tensor" % name)
    if t.dtype != dtype:
        raise TypeError("%s must have dtype %s, got %s" % (name, dtype, t.dtype))
    if not t.is_contiguous():
        raise ValueError("%s must be contiguous" % name)
    return t


# HABITAT_B200_NVTX=1 wraps every native call in an NVTX range named after it, so that a timeline
# shows which entry point a kernel belongs to.
_NVTX = os.environ.get("HABITAT_B200_NVTX", "") not in ("", "0")


def _call(name, fn, *args):
    if not _NVTX:
        return fn(*args)
    torch.cuda.nvtx.range_push(name)
    try:
        return fn(*args)
    finally:
        torch.cuda.nvtx.range_pop()


def _ptr(t):
    return ctypes.c_void_p(t.data_ptr()) if t is not None else ctypes.c_void_p(0)


@dataclass
class KernelBatch:
    """Structure-of-arrays view of K recorded kernels (device tensors).

    num_blocks int32, block_size uint16, regs_per_thread uint16, smem_bytes
    uint32 (static + dynamic), run_time_ns float32, gamma float32 in [0, 1].
    """
    num_blocks: torch.Tensor
    block_size: torch.Tensor
    regs_per_thread: torch.Tensor
    smem_bytes: torch.Tensor
    run_time_ns: torch.Tensor
    gamma: Optional[torch.Tensor] = None

    def __len__(self):
        return int(self.num_blocks.numel())

    @classmethod
    def from_numpy(cls, arrays, device="cuda"):
        """arrays: mapping with the six field names (numpy); uploads them."""
        def up(name, dt):
            a = np.ascontiguousarray(arrays[name]).astype(dt, copy=False)
            return torch.from_numpy(a.view(_NP_VIEW.get(dt, dt))).to(device).view(_TORCH_DT[dt])
        g = arrays.get("gamma")
        return cls(up("num_blocks", np.int32), up("block_size", np.uint16),
                   up("regs_per_thread", np.uint16), up("smem_bytes", np.uint32),
                   up("run_time_ns", np.float32),
                   up("gamma", np.float32) if g is not None else None)


_NP_VIEW = {np.uint16: np.int16, np.uint32: np.int32}
_TORCH_DT = {np.int32: torch.int32, np.uint16: torch.uint16, np.uint32: torch.uint32,
             np.float32: torch.float32}


@dataclass
class KernelMetricsBatch:
    """Raw metrics per kernel (float64 device tensors; has_metrics uint8)."""
    flop_efficiency_pct: torch.Tensor
    dram_read_bytes: torch.Tensor
    dram_write_bytes: torch.Tensor
    has_metrics: torch.Tensor


@dataclass
class WaveResult:
    """Destination-major planes: element (d, k) of a [D, K] tensor."""
    scaled_ns: torch.Tensor          # [D, K] float32, NaN where the reference raises
    dest_occupancy: torch.Tensor     # [D, K] uint8
    dest_waves: torch.Tensor         # [D, K] uint32
    origin_occupancy: torch.Tensor   # [K] uint8
    origin_waves: torch.Tensor       # [K] uint32
    status: Optional[torch.Tensor] = None   # [D, K] uint8
    limits: Optional[torch.Tensor] = None   # [D + 1, 4, K] int32


class WavePartials:
    """Room for the first stage of the per-destination totals of a wave_scale call over up to K
    kernels and D destinations (hb_wave_scale_partials): pass it as `partials=`, then `totals()`
    (or PeerTotals.partials_sum across GPUs) gives the D float64 totals without a second pass over
    the [D, K] results when the launch takes the table kernel."""

    def __init__(self, K, D, device="cuda"):
        self.K, self.D = int(K), int(D)
        n = int(_native.load().hb_wave_scale_partials_len(self.K))
        self.buffer = torch.empty((self.D * n,), dtype=torch.float64, device=device)
        self.per_plane = 0      # first-stage sums per destination left by the last call
        self.n_planes = 0

    def totals(self, out=None):
        """[D] float64 totals of the last wave_scale call that was given this object."""
        res = _call("hb_partials_sum", _native.binding().partials_sum, self.buffer, self.per_plane, self.n_planes,
                    out)
        if res is None:
            _require_cuda(out, torch.float64, "out")
            raise ValueError("out must have one entry per destination")
        return res


def wave_scale(kernels: KernelBatch, origin, dests: Sequence, dest_regs=None, metrics=None,
               want_status=False, want_limits=False, out: Optional[WaveResult] = None,
               partials: Optional[WavePartials] = None):
    """Wave-scales K kernels measured on `origin` to every device in `dests`.

    origin / dests are DeviceProperties.  dest_regs is an optional [D, K] int16
    tensor of per-destination register counts (-1: use the kernel's own).
    With `metrics`, gamma is computed on the device per (kernel, destination).
    With `partials` the call also leaves the first stage of the per-destination totals there.
    Queued on the current stream; does not synchronise.
    """
    name = ("hb_wave_scale_partials" if partials is not None else
            "hb_wave_scale" if metrics is None else "hb_wave_scale_metrics")
    res = _call(name, _native.binding().wave_scale, kernels, origin, dests, dest_regs, metrics,
                want_status, want_limits, out, partials)
    if res is None:
        _check_wave_arguments(kernels, dests, dest_regs, metrics, out, partials)
    return res


def _check_result(t, size, count, name):
    """A given result: contiguous memory that the GPU can write, of `size`-byte elements, at least `count`."""
    if not isinstance(t, torch.Tensor) or not (t.is_cuda or t.is_pinned()):
        raise TypeError("%s must be a CUDA tensor" % name)
    if t.element_size() != size:
        raise TypeError("%s must have elements of %d bytes" % (name, size))
    if not t.is_contiguous() or t.numel() < count:
        raise ValueError("%s must be contiguous, of at least %d elements" % (name, count))


def _check_wave_arguments(kernels, dests, dest_regs, metrics, out, partials):
    """Says what is wrong with arguments the binding did not take."""
    K, D = len(kernels), len(dests)
    _require_cuda(kernels.num_blocks, torch.int32, "num_blocks")
    _require_cuda(kernels.block_size, torch.uint16, "block_size")
    _require_cuda(kernels.regs_per_thread, torch.uint16, "regs_per_thread")
    _require_cuda(kernels.smem_bytes, torch.uint32, "smem_bytes")
    _require_cuda(kernels.run_time_ns, torch.float32, "run_time_ns")
    for name in ("block_size", "regs_per_thread", "smem_bytes", "run_time_ns"):
        if getattr(kernels, name).numel() != K:
            raise ValueError("%s has a different length" % name)
    if metrics is None:
        if kernels.gamma is None:
            raise ValueError("gamma is required unless metrics are given")
        _require_cuda(kernels.gamma, torch.float32, "gamma")
        if kernels.gamma.numel() < K:
            raise ValueError("gamma has a different length")
    if dest_regs is not None:
        _require_cuda(dest_regs, torch.int16, "dest_regs")
        if tuple(dest_regs.shape) != (D, K):
            raise ValueError("dest_regs must be [D, K]")
    if partials is not None:
        if metrics is not None:
            raise ValueError("partials are not available together with metrics")
        if K > partials.K or D > partials.D:
            raise ValueError("partials were sized for fewer kernels or destinations")
    if metrics is not None:
        for name, dtype in (("flop_efficiency_pct", torch.float64), ("dram_read_bytes", torch.float64),
                            ("dram_write_bytes", torch.float64), ("has_metrics", torch.uint8)):
            _require_cuda(getattr(metrics, name), dtype, name)
            if getattr(metrics, name).numel() < K:
                raise ValueError("%s has a different length" % name)
    if out is not None:
        for name, size, count in (("scaled_ns", 4, D * K), ("dest_occupancy", 1, D * K), ("dest_waves", 4, D * K),
                                  ("origin_occupancy", 1, K), ("origin_waves", 4, K), ("status", 1, D * K),
                                  ("limits", 4, (D + 1) * 4 * K)):
            if getattr(out, name) is not None:
                _check_result(getattr(out, name), size, count, name)
    raise ValueError("wave_scale: unsupported arguments (at most %d destinations)" % _native.HB_MAX_DEVICES)


WAVE_PATHS = {0: "none", 1: "wave_scale_kernel", 2: "wave_scale_fast_kernel", 4: "wave_scale_lut_kernel"}


def wave_scale_path():
    """Name of the kernel the calling thread's last wave_scale call launched."""
    return WAVE_PATHS[int(_native.load().hb_wave_scale_path())]


def wave_scale_host(arrays, origin, dests, want_status=False, want_limits=False):
    """Host-buffer path: numpy in, numpy out, transfers inside the native call.  Results of up to a
    few megabytes lie in one block of page-locked memory that the kernel writes directly."""
    binding = _native.binding()
    ins = [np.ascontiguousarray(arrays[name], dtype=dt) for name, dt in _HOST_IN]
    K, D = ins[0].shape[0], len(dests)
    names = ("scaled_ns", "dest_occupancy", "dest_waves", "origin_occupancy", "origin_waves", "status", "limits")
    pairs = (D, K)
    planes = [(names[0], np.float32, pairs, 4), (names[1], np.uint8, pairs, 1), (names[2], np.uint32, pairs, 4),
              (names[3], np.uint8, (K,), 1), (names[4], np.uint32, (K,), 4),
              (names[5], np.uint8, pairs, 1) if want_status else None,
              (names[6], np.int32, (D + 1, 4, K), 4) if want_limits else None]
    at, total = [], 0
    for p in planes:
        at.append(total)
        if p is not None:
            total += (math.prod(p[2]) * p[3] + 255) & ~255
    block = binding.host_block(total) if total and not want_limits else None
    if block is not None:
        outs = [None if p is None else np.ndarray(p[2], p[1], block, o) for p, o in zip(planes, at)]
    else:
        outs = [None if p is None else np.empty(p[2], p[1]) for p in planes]
    if binding.wave_scale_host(*ins, origin, dests, tuple(outs)) is None:
        raise ValueError("the kernel arrays must cover the entries of num_blocks (at most %d destinations)"
                         % _native.HB_MAX_DEVICES)
    return dict(zip(names, outs))


_HOST_IN = (("num_blocks", np.int32), ("block_size", np.uint16), ("regs_per_thread", np.uint16),
            ("smem_bytes", np.uint32), ("run_time_ns", np.float32), ("gamma", np.float32))


class MLPHandle:
    """Device-side weight pack of one runtime predictor (hb_mlp)."""

    def __init__(self, n_op_features, fc1_w, fc1_b, hidden_w, hidden_b, fc2_w, fc2_b, mu, sigma,
                 device_features, precision="bf16"):
        lib = _native.load()
        f32 = lambda a: np.ascontiguousarray(a, dtype=np.float32)
        f64 = lambda a: np.ascontiguousarray(a, dtype=np.float64)
        fc1_w, fc1_b, hidden_w, hidden_b = f32(fc1_w), f32(fc1_b), f32(hidden_w), f32(hidden_b)
        fc2_w, fc2_b = f32(fc2_w).reshape(-1), f32(fc2_b).reshape(-1)
        mu, sigma, device_features = f64(mu), f64(sigma), f64(device_features)
        layers, width = hidden_w.shape[0], hidden_w.shape[1]
        if fc1_w.shape != (width, n_op_features + 4):
            raise ValueError("fc1 weight must be [width, F + 4]")
        if mu.shape != (n_op_features + 4,) or sigma.shape != (n_op_features + 4,):
            raise ValueError("mu and sigma must have F + 4 entries")
        if device_features.ndim != 2 or device_features.shape[1] != 4:
            raise ValueError("device_features must be [n, 4]")
        prec = {"bf16": _native.HB_PRECISION_BF16, "bf16x3": _native.HB_PRECISION_BF16X3}[precision]
        self.n_op_features = n_op_features
        self.precision = precision
        self.n_device_rows = device_features.shape[0]
        self._handle = ctypes.c_void_p(0)
        p = lambda a: ctypes.c_void_p(a.ctypes.data)
        _native.check(lib.hb_mlp_create(
            ctypes.byref(self._handle), n_op_features, layers, width, p(fc1_w), p(fc1_b),
            p(hidden_w), p(hidden_b), p(fc2_w), p(fc2_b), p(mu), p(sigma), p(device_features),
            device_features.shape[0], prec))

    def predict(self, op_features, device_row, out=None):
        """op_features [Q, F] float32 CUDA, device_row [Q] uint8 CUDA -> [Q] float32."""
        res = _call("hb_mlp_predict", _native.binding().mlp_predict, self._handle.value or 0, self.n_op_features,
                    op_features, device_row, out)
        if res is None:
            _require_cuda(op_features, torch.float32, "op_features")
            _require_cuda(device_row, torch.uint8, "device_row")
            if op_features.ndim != 2 or op_features.shape[1] != self.n_op_features:
                raise ValueError("op_features must be [Q, %d]" % self.n_op_features)
            if device_row.numel() != op_features.shape[0]:
                raise ValueError("device_row must have Q entries")
            _check_result(out, 4, op_features.shape[0], "out")
        return res

    def predict_one(self, op_features, device_row):
        """One query, a sequence of F numbers and a device row; returns a float.  The query travels as a
        kernel parameter and the result comes back through page-locked memory."""
        value = _call("hb_mlp_predict_host", _native.binding().mlp_predict_one, self._handle.value or 0,
                      self.n_op_features, op_features, device_row)
        if value is None:
            raise ValueError("op_features must be [Q, %d]" % self.n_op_features)
        return value

    def predict_host(self, op_features, device_row):
        """numpy in / numpy out; transfers and the status check inside the native call."""
        lib = _native.load()
        f = np.ascontiguousarray(op_features, dtype=np.float32)
        r = np.ascontiguousarray(device_row, dtype=np.uint8)
        out = np.empty((f.shape[0],), np.float32)
        _native.check(lib.hb_mlp_predict_host(
            self._handle, ctypes.c_void_p(f.ctypes.data), ctypes.c_void_p(r.ctypes.data),
            f.shape[0], ctypes.c_void_p(out.ctypes.data)))
        return out

    def check_status(self):
        """Synchronises and raises if a launch gave up on a bounded device wait (reported once:
        the next call judges the launches after this one)."""
        code = ctypes.c_int32(0)
        _native.check(_native.load().hb_mlp_status(self._handle, ctypes.byref(code)))

    def inject_status(self, code):
        """Writes the device status word from the host (tests of the error path)."""
        _native.check(_native.load().hb_mlp_inject_status(self._handle, int(code)))

    def inject_mark(self, block=None):
        """Leaves, from the host, the mark of a small-batch launch that gave up (tests of the error path): the next
        such launch on this GPU reports an error instead of results.  With `block` only the block of that rank in each
        cluster heeds it."""
        lib = _native.load()
        _native.check(lib.hb_mlp_inject_mark(self._handle) if block is None
                      else lib.hb_mlp_inject_mark_at(self._handle, int(block)))

    def inject_stale(self, layer=None, feature=0, word=0):
        """Makes the next launch on clusters of SM pairs (43 to 4,224 queries; split precision 15 to 2,112) of each stream on
        this GPU take what its blocks exchange for stale (tests), or, in the library with index checks, send one 32-bit
        word of one feature of a layer's output as if it were.  The network runs once more, and the predictions are the same."""
        lib = _native.load()
        _native.check(lib.hb_mlp_inject_stale(self._handle) if layer is None
                      else lib.hb_mlp_inject_stale_at(self._handle, int(layer), int(feature), int(word)))

    def second_runs(self):
        """How often a cluster of SM pairs has had to run the network once more (synchronises)."""
        runs = ctypes.c_int64()
        _native.check(_native.load().hb_mlp_second_runs(self._handle, ctypes.byref(runs)))
        return runs.value

    def phase_cycles(self):
        """Cycle counters of the first cluster in the last launch of the two-SM kernel (synchronises): epilogue
        group 0 (wait, epilogue, fc2, layers, epi_publish, epi_remote), the MMA issuer (mma_wait_act,
        mma_wait_weights, mma_wait_tmem, mma_issue, slots of 16 KB; mma_total_cycles and mma_total_ns over the
        same interval, whose ratio is the SM clock under load) and the first of three producers
        (producer_wait_slot: waiting for its slots and requesting copies, copies: how many of them;
        producer_copy: the launch's first copy alone, not a sum over `copies`)."""
        out = (ctypes.c_int64 * 16)()
        _native.check(_native.load().hb_mlp_phase_cycles(self._handle, out))
        names = ("wait", "epilogue", "fc2", "layers", "mma_wait_act", "mma_wait_weights", "mma_wait_tmem",
                 "mma_issue", "slots", "producer_wait_slot", "producer_copy", "copies", "mma_total_cycles",
                 "mma_total_ns", "epi_publish", "epi_remote")
        return dict(zip(names, [int(x) for x in out]))

    def close(self):
        if self._handle:
            _native.load().hb_mlp_destroy(self._handle)
            self._handle = ctypes.c_void_p(0)

    def __del__(self):
        try:
            self.close()
        except Exception:
            pass


def special_scale(run_time_ms, pred_dest, pred_orig, negative_count=None):
    """max(0, run_time_ms * pred_dest / pred_orig) elementwise (float32 CUDA tensors)."""
    lib = _native.load()
    for name, t in (("run_time_ms", run_time_ms), ("pred_dest", pred_dest), ("pred_orig", pred_orig)):
        _require_cuda(t, torch.float32, name)
    n = run_time_ms.numel()
    out = torch.empty_like(run_time_ms)
    if negative_count is not None:
        _require_cuda(negative_count, torch.uint32, "negative_count")
    _native.check(lib.hb_special_scale(_ptr(run_time_ms), _ptr(pred_dest), _ptr(pred_orig), n,
                                       _ptr(out), _ptr(negative_count), _native.current_stream_ptr()))
    return out


def segment_sum(values, offsets):
    """float64 sums of values[offsets[s]:offsets[s+1]] (float32 / int64 CUDA tensors)."""
    res = _native.binding().segment_sum(values, offsets)
    if res is None:
        _require_cuda(values, torch.float32, "values")
        _require_cuda(offsets, torch.int64, "offsets")
    return res


def plane_sum(values, out=None):
    """float64 sum of each row of a [P, L] float32 CUDA tensor, NaN entries skipped."""
    res = _native.binding().plane_sum(values, out)
    if res is None:
        _require_cuda(values, torch.float32, "values")
        if values.ndim != 2:
            raise ValueError("values must be [planes, length]")
        _require_cuda(out, torch.float64, "out")
        raise ValueError("out must have one entry per plane")
    return res


def group_sum(values, keys, n_groups, out=None):
    """float64 sums of a float32 CUDA vector grouped by a uint8 key per element (keys at or above
    n_groups and NaN values are skipped): per-device totals of a batch of MLP predictions."""
    res = _native.binding().group_sum(values, keys, n_groups, out)
    if res is None:
        _require_cuda(values, torch.float32, "values")
        _require_cuda(keys, torch.uint8, "keys")
        if values.numel() != keys.numel():
            raise ValueError("values and keys must have the same length")
        if out is not None:
            _require_cuda(out, torch.float64, "out")
        raise ValueError("out must have one entry per group")
    return res
