"""Cross-device prediction of operations and whole traces.

Reference: analyzer/habitat/analysis/predictor.py.  Same constructor, the same
four predictor attributes and the same predict_operation(); what differs is the
inside: instead of one Python call per kernel and two CPU forwards per special
operation, a trace is flattened once and goes through three device launches
(wave scaling, the fused MLP chain per operation kind, the ratio/clamp), for
any number of destination devices at a time (predict_trace).
"""
import collections.abc
import functools
import logging
import operator
import os

import numpy as np
import torch

from habitat_b200 import _native, batched
from habitat_b200.analysis import SPECIAL_OPERATIONS
from habitat_b200.analysis.kernels import MeasuredKernel, PredictedKernel
from habitat_b200.analysis.mlp.mlp import FEATURES, RuntimePredictor
from habitat_b200.analysis.operation import MeasuredOperation, PredictedOperation
from habitat_b200.analysis.run_time import RunTimeMeasurement, RunTimePrediction, RunTimePurePrediction
from habitat_b200.analysis.wave_scaling import batch as wave_batch
from habitat_b200.analysis.wave_scaling.metadata import MetadataManager
from habitat_b200.analysis.wave_scaling.unified import unified_wave_scaling
from habitat_b200.data import path_to_data
from habitat_b200.habitat_cuda import KernelInstance
from habitat_b200.utils import name_all_arguments

logger = logging.getLogger(__name__)

# positional parameter names of the torch callables whose arguments were recorded
CONV2D_PARAMS = ["input", "weight", "bias", "stride", "padding", "dilation", "groups"]
LINEAR_PARAMS = ["input", "weight", "bias"]
BMM_PARAMS = ["input", "mat2", "out"]
LSTM_PARAMS_NO_BATCH_SIZES = ["input", "hx", "flat_weights", "bias", "num_layers", "dropout",
                              "training", "bidirectional", "batch_first"]
LSTM_PARAMS = ["input", "batch_sizes", "hx", "flat_weights", "bias", "num_layers", "dropout",
               "training", "bidirectional"]
MATMUL_PARAMS = ["input", "other", "out"]

_MLP_OPS = ("conv2d", "linear", "bmm", "lstm")


def _first(value):
    return value[0] if isinstance(value, tuple) else value


def conv2d_features(operation):
    """predictor.py:150-176 of the reference."""
    a = name_all_arguments(CONV2D_PARAMS, operation.arguments.args, operation.arguments.kwargs)
    return dict(batch=a["input"][0], image_size=a["input"][2], in_channels=a["input"][1],
                out_channels=a["weight"][0], kernel_size=a["weight"][2], stride=_first(a["stride"]),
                padding=_first(a["padding"]), bias=0 if a["bias"] is None else 1)


def linear_features(operation):
    """predictor.py:184-213: every leading input dimension counts towards the batch."""
    a = name_all_arguments(LINEAR_PARAMS, operation.arguments.args, operation.arguments.kwargs)
    return dict(batch=functools.reduce(operator.mul, a["input"][:-1]), in_features=a["weight"][1],
                out_features=a["weight"][0], bias=0 if a["bias"] is None else 1)


def bmm_features(operation):
    """predictor.py:220-232."""
    a = name_all_arguments(BMM_PARAMS, operation.arguments.args, operation.arguments.kwargs)
    return dict(batch=a["input"][0], left=a["input"][1], middle=a["input"][2], right=a["mat2"][2])


def lstm_features(operation):
    """predictor.py:240-277: the two torch LSTM overloads are told apart by the
    type of the fifth positional argument."""
    args, kwargs = operation.arguments.args, operation.arguments.kwargs
    if not isinstance(args[4], bool):
        a = name_all_arguments(LSTM_PARAMS_NO_BATCH_SIZES, args, kwargs)
        batch, seq_len, input_size = a["input"][1], a["input"][0], a["input"][2]
    else:
        a = name_all_arguments(LSTM_PARAMS, args, kwargs)
        batch = max(operation.arguments.special["batch_sizes"])
        seq_len, input_size = a["input"][0] // batch, a["input"][1]
    return dict(bias=0 if a["bias"] is None else 1, bidirectional=1 if a["bidirectional"] else 0,
                batch=batch, seq_len=seq_len, input_size=input_size, hidden_size=a["hx"][0][2],
                num_layers=a["num_layers"])


_EXTRACTORS = {"conv2d": conv2d_features, "linear": linear_features, "bmm": bmm_features,
               "lstm": lstm_features}


# Batched form of the extractors above for the common recording (every argument positional,
# as torch passes them): one tuple per operation, no dictionaries.  Operations recorded with
# keyword arguments, and the LSTM overloads, go through the named path.
def _conv2d_row(a):
    x, w = a[0], a[1]
    return (x[0], x[2], x[1], w[0], w[2], _first(a[3]), _first(a[4]), 0 if a[2] is None else 1)


def _linear_row(a):
    x, w = a[0], a[1]
    batch = 1
    for v in x[:-1]:
        batch *= v
    return (batch, w[1], w[0], 0 if a[2] is None else 1)


def _bmm_row(a):
    x = a[0]
    return (x[0], x[1], x[2], a[1][2])


_FAST_ROWS = {
    "conv2d": (_conv2d_row, 5, ("batch", "image_size", "in_channels", "out_channels", "kernel_size",
                                "stride", "padding", "bias")),
    "linear": (_linear_row, 3, ("batch", "in_features", "out_features", "bias")),
    "bmm": (_bmm_row, 2, ("batch", "left", "middle", "right")),
}


def feature_matrix(name, operations, order):
    """[n, F] float32 features of `operations` (all of kind `name`) in the column order `order`."""
    fast = _FAST_ROWS.get(name)
    if fast is not None:
        row, arity, columns = fast
        try:
            rows = [row(op.arguments.args) if len(op.arguments.args) >= arity and not op.arguments.kwargs
                    else None for op in operations]
        except (TypeError, IndexError):
            rows = [None]
        if None not in rows:
            m = np.array(rows, dtype=np.float32).reshape(len(rows), len(columns))
            return np.ascontiguousarray(m[:, [columns.index(f) for f in order]])
    extract = _EXTRACTORS[name]
    return np.array([[extract(op)[f] for f in order] for op in operations], dtype=np.float32)


class _LazyRunTimePrediction(RunTimePrediction):
    """A predicted pass whose time is known (summed on the device) and whose
    PredictedKernel objects are only built when somebody asks for them."""

    def __init__(self, overhead_ns, measured_kernels, times_ns, total_kernel_ns, device):
        super().__init__(overhead_ns=overhead_ns, predicted_kernels=None, device=device)
        self._measured_kernels = measured_kernels
        self._times_ns = times_ns
        self._run_time_ms = (overhead_ns + total_kernel_ns) / 1e6

    @property
    def kernels(self):
        if self._predicted_kernels is None:
            self._predicted_kernels = [PredictedKernel(k, float(t))
                                       for k, t in zip(self._measured_kernels, self._times_ns)]
        return self._predicted_kernels


_METRIC_KEYS = tuple((m, m.value.cupti_name, m.value.legacy_cupti_name) for m in wave_batch._NEEDED)
# the kinds whose features the native walk extracts, and the columns it fills: those of the predictors' classes
_FAST_KINDS = ("conv2d", "linear", "bmm")
_FAST_ORDERS = tuple(tuple(_FAST_ROWS[k][2].index(f) for f in FEATURES[k]) for k in _FAST_KINDS)


def _trace_types():
    return MeasuredOperation, RunTimeMeasurement, MeasuredKernel, KernelInstance


class _GroupPlan:
    """Everything about the operations of one origin device that does not depend on the
    destination: which operation is predicted how, the flattened kernels of the wave-scaled
    passes, launch overheads, MLP feature matrices.  Built by the first prediction of a trace
    and kept with it."""

    def __init__(self, operations, indices, mode, flat=None):
        self.mode = mode
        self.mlp_inputs = {}      # op kind -> (features, measured ms) on the GPU, measured ms, columns; filled on first use
        self._layout = None
        if flat is None:
            self._flatten(operations, indices, mode)
        else:
            self._take(operations, flat)

    @classmethod
    def of_whole_trace(cls, operations, mode, with_names, early=None, first=None):
        """The plan of a trace recorded on one device, walked by the native binding; None when the
        operations are not all of this package's ordinary classes (any object with their surface
        takes the Python walk), or when a missing metric has to raise (the roofline strategy).
        early(inputs of the MLP kinds, indices of their operations) is called before the kernels are walked, with None
        for the inputs when some kind's are not known by then.
        What belongs to the prediction that asks and not to the plan goes into the list `first`: what `early`
        returned, and memory to be kept until that prediction has ended."""
        if mode == wave_batch.ROOFLINE:
            return None
        flat = _native.binding().flatten_trace(operations, _trace_types(), SPECIAL_OPERATIONS, _MLP_OPS, _METRIC_KEYS,
                                               mode != wave_batch.RESIMPLIFIED, _FAST_ORDERS, with_names, early)
        if flat is None:
            return None
        if first is not None:
            first.extend(flat[-2:])
        return cls(operations, None, mode, flat[:-2])

    def _take(self, operations, flat):
        (self.n_kernels, self.n_runs, self._names, wave_idx, fwd, bwd, offsets, overheads, kind_idx, self.passthrough_idx,
         records, metrics, self.offsets_dev, special) = flat
        self._kernels, self._operations = None, operations
        self.indices = None                      # all operations
        self.wave_idx, self.fwd_run, self.bwd_run, self.offsets = (
            np.frombuffer(x, np.int64) for x in (wave_idx, fwd, bwd, offsets))
        self.overheads = np.frombuffer(overheads, np.float64)
        self.mlp_idx = {name: np.frombuffer(x, np.int64) for name, x in zip(_MLP_OPS, kind_idx)}
        for name, got in zip(_FAST_KINDS, special):
            if got is not None:
                self.mlp_inputs[name] = (got[0], got[1], np.frombuffer(got[2], np.float32), FEATURES[name])
        for i in self.passthrough_idx:
            logger.warning("Unhandled special operation: %s", operations[i].name)
        self.flat = (wave_batch.FlatKernels.from_device(self.mode, self.n_kernels, self._names, records, metrics)
                     if self.n_kernels else None)

    # The recorded kernels and their names, in the order of the flattened records: only the register table and
    # user-supplied strategies ask for them.
    @property
    def kernels(self):
        if self._kernels is None:
            self._kernels = [k for i in self.wave_idx for run in (self._operations[i].forward, self._operations[i].backward)
                             if run is not None for k in run.kernels]
        return self._kernels

    @property
    def names(self):
        if self._names is None:
            self._names = [k.name for k in self.kernels]
        return self._names

    def _flatten(self, operations, indices, mode):
        self.indices = np.asarray(indices, np.int64)
        wave_idx, fwd_run, bwd_run, runs = [], [], [], []
        self.mlp_idx = {op: [] for op in _MLP_OPS}
        self.passthrough_idx = []
        for i in indices:
            op = operations[i]
            name = op.name
            if name not in SPECIAL_OPERATIONS:
                wave_idx.append(i)
                fwd_run.append(len(runs))
                runs.append(op.forward)
                if op.backward is not None:
                    bwd_run.append(len(runs))
                    runs.append(op.backward)
                else:
                    bwd_run.append(-1)
            elif name in self.mlp_idx:
                self.mlp_idx[name].append(i)
            else:
                logger.warning("Unhandled special operation: %s", name)
                self.passthrough_idx.append(i)
        self.mlp_idx = {op: np.asarray(idx, np.int64) for op, idx in self.mlp_idx.items()}
        self.wave_idx = np.asarray(wave_idx, np.int64)
        self.fwd_run = np.asarray(fwd_run, np.int64)
        self.bwd_run = np.asarray(bwd_run, np.int64)
        self._kernels, self._names = [], None
        offsets = [0]
        for run in runs:
            self._kernels.extend(run.kernels)
            offsets.append(len(self._kernels))
        self.n_kernels, self.n_runs = len(self._kernels), len(runs)
        self.offsets = np.asarray(offsets, np.int64)
        self.flat = wave_batch.FlatKernels(self.kernels, mode) if (self.kernels and mode is not None) else None
        if self.flat is not None:
            self._names = self.flat.names
        # launch overhead of a pass (predictor.py:113-116 of the reference): wall time minus kernel time
        measured = np.array([k.run_time_ns for k in self.kernels], np.float64)
        per_run = np.add.reduceat(np.concatenate([measured, [0.0]]), self.offsets[:-1]) if runs else np.zeros(0)
        per_run = np.where(self.offsets[1:] > self.offsets[:-1], per_run, 0.0) if runs else per_run
        wall_ns = np.array([run.run_time_ms for run in runs], np.float64) * 1e6
        self.overheads = np.maximum(wall_ns - per_run, 0.0)
        self.offsets_dev = torch.from_numpy(self.offsets).cuda() if self.flat is not None else None

    def layout(self, n):
        """(kind, a, b) of the n operations of the trace for a destination that predicts this group
        alone, shared by every such destination (PredictedOperations)."""
        if self._layout is None:
            kind, a, b = np.zeros(n, np.int8), np.full(n, -1, np.int64), np.full(n, -1, np.int64)
            kind[self.wave_idx] = 1
            a[self.wave_idx], b[self.wave_idx] = self.fwd_run, self.bwd_run
            for idx in self.mlp_idx.values():
                kind[idx] = 2
            if self.passthrough_idx:
                kind[self.passthrough_idx] = 3
            self._layout = kind, a, b
        return self._layout

    def special_inputs(self, name, operations, order):
        """Features and measured times of the operations of one MLP kind, on the GPU."""
        got = self.mlp_inputs.get(name)
        if got is None or got[3] != order:
            ops = [operations[i] for i in self.mlp_idx[name]]
            rt = np.array([op.run_time_ms for op in ops], np.float32)
            got = torch.from_numpy(feature_matrix(name, ops, order)).cuda(), torch.from_numpy(rt).cuda(), rt, order
            self.mlp_inputs[name] = got
        return got


class PredictedOperations(collections.abc.Sequence):
    """The operations of a trace as predicted for one destination.  Behaves like the list the
    reference builds (len, indexing, iteration); PredictedOperation, RunTimePrediction and
    PredictedKernel objects are created when an element is first touched, the per-operation
    times (`run_times_ms`) and their sum (`total_run_time_ms`) are there from the start."""

    def __init__(self, operations, dest, group=None, run_times_ms=None, total_ms=None):
        self._operations = operations
        self._dest = dest
        self._made = None                           # elements, once one has been touched
        self._groups = [group] if group else []     # per origin group: dict(plan, times, totals)
        self._total = total_ms
        self._group = None                          # which group an operation is of; None: the first
        n = len(operations)
        if group is not None:                       # all of one group: its layout, when an element is touched
            self._kind = None
            self.run_times_ms = run_times_ms
        else:
            self._kind = np.zeros(n, np.int8)       # 0 as measured, 1 wave-scaled, 2 MLP, 3 special passed through
            self._a = np.full(n, -1, np.int64)      # wave: forward run
            self._b = np.full(n, -1, np.int64)      # wave: backward run or -1
            self._group = np.zeros(n, np.int32)
            self.run_times_ms = np.zeros(n, np.float64)

    def __len__(self):
        return len(self._operations)

    def __getitem__(self, i):
        if isinstance(i, slice):
            return [self[j] for j in range(*i.indices(len(self)))]
        if i < 0:
            i += len(self)
        if self._made is None:
            self._made = [None] * len(self._operations)
        made = self._made[i]
        if made is None:
            made = self._made[i] = self._make(i)
        return made

    @property
    def total_run_time_ms(self):
        if self._total is None:
            self._total = float(self.run_times_ms.sum())
        return self._total

    def _make(self, i):
        op = self._operations[i]
        if self._kind is None:
            self._kind, self._a, self._b = self._groups[0]["plan"].layout(len(self._operations))
        kind = self._kind[i]
        if kind == 0:
            return op
        if kind == 3:
            return PredictedOperation(op, op.forward, op.backward, self._dest)
        g = self._groups[self._group[i] if self._group is not None else 0]
        if kind == 2:
            return PredictedOperation(op, RunTimePurePrediction(float(self.run_times_ms[i]), self._dest),
                                      None, self._dest)
        plan = g["plan"]

        def run(r, measured):
            lo, hi = plan.offsets[r], plan.offsets[r + 1]
            return _LazyRunTimePrediction(float(plan.overheads[r]), measured.kernels, g["times"][lo:hi],
                                          float(g["totals"][r]), self._dest)
        b = self._b[i]
        return PredictedOperation(op, run(self._a[i], op.forward), run(b, op.backward) if b >= 0 else None, self._dest)


class Predictor:
    def __init__(self, kernel_metadata_file=None, wave_scaling_strategy=unified_wave_scaling, *,
                 model_paths=None, precision=None):
        if kernel_metadata_file is None:
            default = path_to_data("kernels.sqlite")
            kernel_metadata_file = default if os.path.exists(default) else None
        self._kernel_metadata = MetadataManager(kernel_metadata_file)
        self._wave_scaling_strategy = wave_scaling_strategy
        # "bf16" (2e-2 relative against the float32 reference) or "bf16x3" (1e-4); the environment
        # variable HABITAT_B200_PRECISION chooses for callers that keep the reference's constructor call
        self._precision = precision or os.environ.get("HABITAT_B200_PRECISION", "bf16")
        if self._precision not in ("bf16", "bf16x3"):
            raise ValueError("precision must be 'bf16' or 'bf16x3', got %r" % (self._precision,))
        self._model_paths = dict(model_paths or {})
        self._predictors = {}

    # The four predictors load on first use: their checkpoints are large and,
    # unlike the reference, most traces do not need all of them.
    def _predictor(self, op):
        if op not in self._predictors:
            path = self._model_paths.get(op, path_to_data("%s/model.pth" % op))
            if not os.path.exists(path):
                raise FileNotFoundError(
                    "no checkpoint for the %s predictor at %s (pass model_paths= or assign "
                    "Predictor.%s_pred)" % (op, path, op))
            self._predictors[op] = RuntimePredictor(op, 8, 1024, path, precision=self._precision)
        return self._predictors[op]

    linear_pred = property(lambda self: self._predictor("linear"),
                           lambda self, v: self._predictors.__setitem__("linear", v))
    lstm_pred = property(lambda self: self._predictor("lstm"),
                         lambda self, v: self._predictors.__setitem__("lstm", v))
    conv2d_pred = property(lambda self: self._predictor("conv2d"),
                           lambda self, v: self._predictors.__setitem__("conv2d", v))
    bmm_pred = property(lambda self: self._predictor("bmm"),
                        lambda self, v: self._predictors.__setitem__("bmm", v))

    # ------------------------------------------------------------------
    def predict_operation(self, operation, dest_device):
        return self.predict_trace([operation], [dest_device])[0][0]

    def predict_trace(self, operations, dest_devices, cache=None):
        """Predicts every operation on every destination.

        Returns one sequence of operations per destination, in order (PredictedOperations:
        list-like, elements built on first access); operations measured on a device of the
        same name as the destination are returned as they are (analysis/trace.py:40-41 and
        operation.py:82-85).  `cache` is a dict the caller keeps with the operations (Trace
        does): the destination-independent plan of the trace (flattened, GPU-resident kernel
        records, overheads, MLP features) is stored there and reused by later calls."""
        if not isinstance(operations, (list, tuple)):
            operations = list(operations)
        whole = self._predict_whole(operations, dest_devices, cache)
        if whole is not None:
            return whole
        D = len(dest_devices)
        results = [PredictedOperations(operations, dest) for dest in dest_devices]
        key = ("origins", len(operations))
        by_origin = cache.get(key) if cache is not None else None
        if by_origin is None:
            by_origin = {}
            for i, op in enumerate(operations):
                by_origin.setdefault(op.device.name, []).append(i)
            if cache is not None:
                cache[key] = by_origin
        for origin_name, indices in by_origin.items():
            origin = operations[indices[0]].device
            targets = [d for d in range(D) if dest_devices[d].name != origin_name]
            same = [d for d in range(D) if dest_devices[d].name == origin_name]
            if same:
                ms = np.array([operations[i].run_time_ms for i in indices], np.float64)
                for d in same:
                    results[d].run_times_ms[indices] = ms      # kind 0: the measured operation itself
            if targets:
                self._predict_group(operations, indices, origin, dest_devices, targets, results, cache)
        return results

    def _predict_whole(self, operations, dest_devices, cache):
        """predict_trace for a trace recorded on one device and predicted for others (what a Trace
        is); None for anything else."""
        if not operations or not dest_devices:
            return None
        mode = getattr(self._wave_scaling_strategy, "batch_mode", None)
        origin = operations[0].device
        key = ("whole", mode, len(operations))
        known = cache.get(key) if cache is not None else None
        plan, first = known, [None]              # first: of this prediction alone, whoever else finds the plan
        if mode is None or any(d.name == origin.name for d in dest_devices):
            return None
        if plan is None:
            first = []
            plan = _GroupPlan.of_whole_trace(
                operations, mode, self._has_registers(),
                lambda special, indices: self._start_kinds(special, indices, origin, dest_devices, len(operations)),
                first)
            if plan is None:
                return None
        ms = np.empty((len(dest_devices), len(operations)), np.float64)
        for i in plan.passthrough_idx:
            ms[:, i] = operations[i].run_time_ms
        times, totals, sums = self._run_plan(plan, operations, origin, dest_devices, ms, first[0])
        if known is None and cache is not None:
            cache[key] = plan                    # not before its records are on the GPU, for other streams as well
        return [PredictedOperations(operations, dest, dict(plan=plan, times=times[t], totals=totals[t]), ms[t], sums[t])
                for t, dest in enumerate(dest_devices)]

    def _start_kinds(self, special, indices, origin, dests, n_operations):
        """Starts the predictors of a trace whose kernels are still being walked: what run_group takes as their
        results, with the kinds it is for, or None when they cannot be started now (`_run_plan`
        then prepares them again and raises what there is to raise).  What a launch raises is raised here."""
        if special is None or len(dests) > _native.HB_MAX_DEVICES:
            return None
        try:
            kinds, held = [], []
            for name, idx in zip(_MLP_OPS, indices):
                if not idx:
                    continue
                got = special[_FAST_KINDS.index(name)]
                pred = self._predictor(name)
                if FEATURES[name] != pred.model.features or not self._is_plain(pred):
                    return None
                rows = bytes([pred.device_row(origin.name)] + [pred.device_row(d.name) for d in dests])
                held.append(pred._handle)
                kinds.append((held[-1]._handle.value or 0, got[0], got[1], rows, idx))
        except Exception:
            return None
        return batched._call("start_kinds", _native.binding().start_kinds, kinds, len(dests), n_operations, held), kinds

    @staticmethod
    def _is_plain(pred):
        return getattr(pred.predict_batch, "__func__", None) is RuntimePredictor.predict_batch

    def _has_registers(self):
        return self._kernel_metadata is not None and not getattr(self._kernel_metadata, "empty", False)

    # ------------------------------------------------------------------
    def _predict_group(self, operations, indices, origin, dest_devices, targets, results, cache=None):
        dests = [dest_devices[d] for d in targets]
        mode = getattr(self._wave_scaling_strategy, "batch_mode", None)
        whole = len(indices) == len(operations)
        key = ("whole", mode, len(operations)) if whole else ("plan", origin.name, mode, len(indices))
        plan = cache.get(key) if cache is not None else None
        if plan is None:
            if whole and mode is not None:
                plan = _GroupPlan.of_whole_trace(operations, mode, self._has_registers())
            plan = plan or _GroupPlan(operations, indices, mode)
        ms = np.zeros((len(dests), len(operations)), np.float64)
        for i in plan.passthrough_idx:
            ms[:, i] = operations[i].run_time_ms
        times, totals, _ = self._run_plan(plan, operations, origin, dests, ms)
        if cache is not None:
            cache[key] = plan                    # as in _predict_whole
        for t, d in enumerate(targets):
            res = results[d]
            g = len(res._groups)
            res._groups.append(dict(plan=plan, times=times[t], totals=totals[t]))
            if len(plan.wave_idx):
                res._kind[plan.wave_idx] = 1
                res._group[plan.wave_idx] = g
                res._a[plan.wave_idx] = plan.fwd_run
                res._b[plan.wave_idx] = plan.bwd_run
            for i in plan.passthrough_idx:
                res._kind[i] = 3
            for idx in plan.mlp_idx.values():
                res._kind[idx] = 2
            res.run_times_ms[indices] = ms[t, indices]

    def _run_plan(self, plan, operations, origin, dests, ms, started=None):
        """One prediction of a flattened group: fills `ms` [T, operations] for its operations and returns
        (scaled kernel times [T, K], per-pass kernel totals [T, runs], sums of the rows of `ms`), all on
        the host (predictor.py:111-148 of the reference for every pass, special operation and destination
        at once).  `started`: what _start_kinds returned for these operations and destinations."""
        T, K, n_runs = len(dests), plan.n_kernels, plan.n_runs
        names = [name for name in _MLP_OPS if len(plan.mlp_idx[name])]
        kinds, native, held = [], [], []
        if started is not None:
            kinds, native, names = started[1], names, []
        for name in names:
            pred = self._predictor(name)
            rows = bytes([pred.device_row(origin.name)] + [pred.device_row(d.name) for d in dests])
            feats, rt, rt_host, _ = plan.special_inputs(name, operations, pred.model.features)
            if self._is_plain(pred):
                held.append(pred._handle)        # the call below knows its address only
                kinds.append((held[-1]._handle.value or 0, feats, rt, rows, plan.mlp_idx[name]))
                native.append(name)
            else:
                ms[:, plan.mlp_idx[name]] = self._special_scale_ops(name, pred, rows, feats, rt, rt_host, T)
        flat = plan.flat                         # None: no kernels, or a user-supplied strategy
        times = np.empty((T, K), np.float32 if flat is not None else np.float64)
        totals = (np.empty if flat is not None else np.zeros)((T, n_runs), np.float64)
        if flat is None and K:
            # the reference's per-kernel protocol
            for t, dest in enumerate(dests):
                times[t] = [self._wave_scaling_strategy(k, origin, dest, self._kernel_metadata).run_time_ns
                            for k in plan.kernels]
            for r in range(n_runs):
                totals[:, r] = times[:, plan.offsets[r]:plan.offsets[r + 1]].sum(axis=1)
        if flat is None and len(plan.wave_idx):
            run_ms = (plan.overheads + totals) / 1e6
            ms[:, plan.wave_idx] = run_ms[:, plan.fwd_run] + np.where(plan.bwd_run >= 0, run_ms[:, plan.bwd_run], 0.0)
        if flat is None and not kinds:           # nothing for the GPU, and none needed
            return times, totals, ms.sum(axis=1).tolist()
        regs = None
        if flat is not None and self._has_registers():
            regs = wave_batch.destination_registers(plan.kernels, plan.names, dests, self._kernel_metadata)
        nan, sums, clamped = batched._call(
            "run_group", _native.binding().run_group, flat.batch if flat is not None else None,
            flat.metrics if flat is not None else None, origin, dests, regs,
            plan.offsets_dev if flat is not None else None, kinds,
            (plan.overheads, plan.wave_idx, plan.fwd_run, plan.bwd_run), times, totals, ms,
            *(() if started is None else started[:1]))
        if nan:
            wave_batch.raise_zero_wave()
        for name, raw in zip(native, clamped):
            if raw is not None:
                self._warn_negative(name, plan.mlp_inputs[name][2], np.frombuffer(raw, np.float32).astype(np.float64), T)
        return times, totals, sums

    def _special_scale_ops(self, name, pred, rows, feats, rt, rt_host, T):
        """-> [T, n] predicted ms of the operations of one kind (predictor.py:132-148 of the reference) from a
        predictor with a predict_batch of its own."""
        n = len(rt_host)
        p = pred.predict_batch(feats.repeat(T + 1, 1), torch.tensor(list(rows), dtype=torch.uint8,
                                                                    device="cuda").repeat_interleave(n))
        neg = torch.zeros(1, dtype=torch.int32, device="cuda")
        ms = batched.special_scale(rt.repeat(T), p[n:], p[:n].repeat(T), neg.view(torch.uint32)).view(T, n).cpu().numpy()
        if getattr(pred, "_handle", None) is not None:
            pred._handle.check_status()
        if int(neg.cpu()[0]):
            self._warn_negative(name, rt_host, p.cpu().numpy().astype(np.float64), T)
        return ms

    @staticmethod
    def _warn_negative(name, run_time_ms, pred_ms, T):
        n = len(run_time_ms)
        for t in range(T):
            raw = run_time_ms.astype(np.float64) * pred_ms[(t + 1) * n:(t + 2) * n] / pred_ms[:n]
            for j in np.nonzero(raw < 0)[0]:
                logger.warning("Operation %s predicted run time %.2f ms", name, raw[j])
