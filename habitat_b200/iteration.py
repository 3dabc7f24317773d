"""Per-iteration predicted times for many training iterations at once.

The array form of what Trace.to_device(...).run_time_ms computes per trace in the
reference (analyzer/habitat/analysis/trace.py:26-51 over predictor.py:84-148):
every iteration is a list of wave-scaled kernels (one operation each, with its
launch overhead) and of MLP-predicted operations; the result is the predicted
iteration time on every destination.  Everything between the inputs and the
[iterations, destinations] totals stays on the device: the wave-scale kernel,
the fused MLP chain of every operation kind side by side, and one kernel that forms
the ratios and adds everything up in a fixed order (float64).
"""
from dataclasses import dataclass
from typing import Dict, Sequence

import torch

from habitat_b200 import _native, batched


@dataclass
class SpecialOps:
    """MLP-predicted operations of one kind, ordered by iteration.

    handle: batched.MLPHandle; features [n, F] float32 CUDA; run_time_ms [n]
    float32 CUDA (measured on the origin); offsets [I + 1] int64 CUDA."""
    handle: "batched.MLPHandle"
    features: torch.Tensor
    run_time_ms: torch.Tensor
    offsets: torch.Tensor


def predict_iteration_totals(kernels: batched.KernelBatch, overhead_ns: torch.Tensor,
                             kernel_offsets: torch.Tensor, special: Dict[str, SpecialOps],
                             origin, dests: Sequence, origin_mlp_row: int,
                             dest_mlp_rows: Sequence[int]):
    """-> ([I, D] float64 CUDA tensor of predicted ms per iteration and destination,
    the batched.WaveResult of the wave-scaled kernels: its scaled_ns is NaN for the pairs the
    reference would raise ZeroDivisionError on, and so are the totals of their iterations).

    A destination with the origin's name keeps the measured times, as
    MeasuredOperation.to_device does (analysis/operation.py:82-85)."""
    same = bytes(d.name == origin.name for d in dests)
    rows = bytes([origin_mlp_row] + [r for r, s in zip(dest_mlp_rows, same) if not s])
    if len(rows) != 1 + same.count(0):
        raise ValueError("dest_mlp_rows must have an entry per destination")
    kinds, own = [], []                       # own: handles with a predict of their own
    for ops in special.values():
        if ops.features.shape[0] == 0:
            continue
        if getattr(ops.handle.predict, "__func__", None) is not batched.MLPHandle.predict:
            own.append(ops)
            continue
        if ops.features.ndim != 2 or (len(rows) > 1 and ops.features.shape[1] != ops.handle.n_op_features):
            raise ValueError("op_features must be [Q, %d]" % ops.handle.n_op_features)
        kinds.append((ops.handle._handle.value or 0, ops.features.contiguous(), ops.run_time_ms, ops.offsets, rows))
    res = batched.wave_scale(kernels, origin, dests)
    totals = batched._call("iteration_totals", _native.binding().iteration_totals, kernels, res.scaled_ns, overhead_ns,
                           kernel_offsets, same, kinds)
    if totals is None:
        batched._require_cuda(overhead_ns, torch.float32, "overhead_ns")
        batched._require_cuda(kernel_offsets, torch.int64, "kernel_offsets")
        for ops in special.values():
            batched._require_cuda(ops.features.contiguous(), torch.float32, "features")
            batched._require_cuda(ops.run_time_ms, torch.float32, "run_time_ms")
            batched._require_cuda(ops.offsets, torch.int64, "offsets")
        raise ValueError("overheads, features, measured times and offsets have to fit the kernels and iterations")
    for ops in own:
        _add_special(totals, ops, rows, same)
    return totals, res


def _add_special(totals, ops, rows, same):
    """Adds the operations of one kind from the predictions of ops.handle.predict."""
    n, T = ops.features.shape[0], len(rows) - 1
    if T:
        pred = ops.handle.predict(ops.features.repeat(T + 1, 1), torch.tensor(
            list(rows), dtype=torch.uint8, device=totals.device).repeat_interleave(n))
        ms = batched.special_scale(ops.run_time_ms.repeat(T), pred[n:], pred[:n].repeat(T)).view(T, n)
    t = 0
    for d, measured in enumerate(same):
        totals[:, d] += batched.segment_sum(ops.run_time_ms if measured else ms[t], ops.offsets)
        t += not measured
