"""Workloads of the prediction path, from one query to the scale sweep's batch.

A case is a dict of plain values; its "kind" says which public entry point it goes through:

  predict     RuntimePredictor.predict, one query per call: what the analyzer's scalar API does
  mlp         batched.MLPHandle.predict (or predict_host) over a batch of queries, and with
              "totals" the per-device sums of the predictions (batched.group_sum)
  wave        batched.wave_scale of K recorded kernels to D devices; "variant" is plain (gamma
              given), metrics (gamma from raw metrics, per-destination register counts: the
              analyzer's inputs), status (the per-pair status plane) or totals (the
              per-destination sums started inside the call)
  host        batched.wave_scale_host: numpy arrays in, numpy arrays out
  pipeline    hostio.WaveScaleHost: three pinned record blocks through the host pipeline
  trace       Trace.to_devices of recorded operations to five devices, for the first time or again
  iterations  iteration.predict_iteration_totals over the mixed iteration trace

Value ranges are those of habitat_b200/workloads.py; weights are random, with a gain that keeps
the outputs moving with the inputs and an output bias that keeps predicted times positive, as
trained predictors have them.  Everything is made from the seed, on the GPU where it is large.
"""
import math

import numpy as np
import torch

from habitat_b200 import batched, device_table, hostio, iteration, workloads
from habitat_b200.analysis.arguments import Arguments
from habitat_b200.analysis.kernels import MeasuredKernel
from habitat_b200.analysis.metrics import Metric
from habitat_b200.analysis.mlp.mlp import RuntimePredictor, state_to_arrays
from habitat_b200.analysis.operation import MeasuredOperation
from habitat_b200.analysis.predictor import Predictor
from habitat_b200.analysis.run_time import RunTimeMeasurement
from habitat_b200.analysis.trace import Trace
from habitat_b200.habitat_cuda import KernelInstance

OPS = ("conv2d", "linear", "bmm", "lstm")
LAYERS, WIDTH = 8, 1024                       # every shipped predictor
MAX_PAIRS = workloads.SWEEP_KERNELS * 6       # the scale sweep's (kernel, device) pairs
MAX_QUERIES = workloads.SWEEP_QUERIES
MLP_SHARE = ("conv2d", "linear", "bmm")       # predictors of the mixed iteration trace


def listed():
    return [
        # One operation through the reference's scalar API: what Operation.to_device pays per query.
        {"name": "predict one", "kind": "predict", "op": "conv2d", "precision": "bf16", "calls": 1},
        # The conv2d operations of one recorded iteration, on the origin and six destinations.
        {"name": "mlp iteration", "kind": "mlp", "op": "conv2d", "precision": "bf16", "queries": 371,
         "totals": False, "host": False},
        # A design-space study in the 1e-4 mode: the linear predictor's benchmark batch.
        {"name": "mlp split 65536", "kind": "mlp", "op": "linear", "precision": "bf16x3", "queries": 65536,
         "totals": False, "host": False},
        # One predictor's share of the scale sweep, with the per-device totals.
        {"name": "mlp sweep", "kind": "mlp", "op": "lstm", "precision": "bf16", "queries": MAX_QUERIES,
         "totals": True, "host": False},
        # The kernels of one small recorded trace to three candidate GPUs.
        {"name": "wave 333", "kind": "wave", "kernels": 333, "dests": 3, "variant": "plain"},
        # The synthetic trace of the wave-scaling benchmark.
        {"name": "wave 1M", "kind": "wave", "kernels": 1 << 20, "dests": 6, "variant": "plain"},
        # The analyzer's inputs (raw metrics, register table) over many traces; an odd kernel count.
        {"name": "wave metrics 250001", "kind": "wave", "kernels": 250001, "dests": 6, "variant": "metrics"},
        # The scale sweep's batch with its per-destination totals.
        {"name": "wave sweep totals", "kind": "wave", "kernels": workloads.SWEEP_KERNELS, "dests": 6,
         "variant": "totals"},
        # A program that keeps its records in numpy and calls the host-buffer entry point.
        {"name": "host 65536", "kind": "host", "kernels": 65536, "dests": 6},
        # A freshly recorded iteration of a model (160 operations) predicted for five GPUs.
        {"name": "trace first", "kind": "trace", "iterations": 1, "again": False},
        # The same question asked again about a longer trace, as a what-if session does.
        {"name": "trace again", "kind": "trace", "iterations": 64, "again": True},
        # The mixed iteration trace, device-resident: per-iteration totals on six GPUs.
        {"name": "iterations 512", "kind": "iterations", "iterations": 512},
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))))


def draw(rng):
    kind = rng.choice(("mlp", "mlp", "mlp", "wave", "wave", "wave", "predict", "host", "pipeline", "trace",
                       "iterations"))
    precision = rng.choice(("bf16", "bf16", "bf16x3"))
    if kind == "predict":
        return {"kind": kind, "op": rng.choice(OPS), "precision": precision, "calls": rng.randint(2, 16)}
    if kind == "mlp":
        host = rng.random() < 0.2
        top = MAX_QUERIES if precision == "bf16" else MAX_QUERIES // 8
        return {"kind": kind, "op": rng.choice(OPS), "precision": precision,
                "queries": _log_int(rng, 1, 65536 if host else top),
                "totals": not host and rng.random() < 0.3, "host": host}
    if kind == "wave":
        dests = rng.randint(1, 13)
        return {"kind": kind, "kernels": _log_int(rng, 1, MAX_PAIRS // max(dests, 6)), "dests": dests,
                "variant": rng.choice(("plain", "plain", "metrics", "status", "totals"))}
    if kind in ("host", "pipeline"):
        return {"kind": kind, "kernels": _log_int(rng, 64, 1 << 20), "dests": rng.randint(1, 8)}
    if kind == "trace":
        return {"kind": kind, "iterations": _log_int(rng, 1, 64), "again": rng.random() < 0.5}
    return {"kind": kind, "iterations": _log_int(rng, 1, 512)}


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _devices(n):
    """(origin, n destinations): the benchmark's six rows, then the other rows of the device table."""
    table = device_table.load_device_file()
    names = list(workloads.BENCH_DEVICES) + [d for d in sorted(table) if d not in workloads.BENCH_DEVICES]
    return table[names[0]], [table[d] for d in names[:n]]


def _uniform(g, lo, hi, n):
    return torch.rand(n, generator=g, device="cuda", dtype=torch.float64) * (hi - lo) + lo


def _log_uniform(g, lo, hi, n):
    """Integers in [lo, hi] with log-uniform density (float64)."""
    return torch.exp(_uniform(g, math.log(lo), math.log(hi + 1), n)).floor().clamp(lo, hi)


def _randint(g, lo, hi, n):
    return torch.randint(lo, hi, (n,), generator=g, device="cuda", dtype=torch.int32)


def _choice(g, values, n):
    return torch.tensor(values, dtype=torch.int32, device="cuda")[_randint(g, 0, len(values), n).long()]


def _kernels(g, n, launchable=False):
    """Recorded kernels as device tensors.  `launchable` keeps to launches that every device can
    run (what a recorded trace holds); otherwise the whole range, some of it not runnable."""
    block = _choice(g, [32, 64, 128, 256, 512, 1024], n)
    regs = _randint(g, 16, 256, n)
    smem = 256 * _randint(g, 0, 385, n)
    if launchable:
        regs = torch.minimum(regs, 32768 // block)
        smem = smem % (47 * 1024)
    return batched.KernelBatch(
        num_blocks=_log_uniform(g, 1, 1 << 20, n).to(torch.int32),
        block_size=block.to(torch.int16).view(torch.uint16),
        regs_per_thread=regs.to(torch.int16).view(torch.uint16),
        smem_bytes=smem.view(torch.uint32),
        run_time_ns=_log_uniform(g, 2000, 50_000_000, n).float(),
        gamma=torch.rand(n, generator=g, device="cuda"))


def _metrics(g, n):
    """Raw metrics; one kernel in eight has none, a few have no FLOPs or no traffic."""
    kind = _randint(g, 0, 32, n)
    eff = _uniform(g, 0.0, 80.0, n)
    rd, wr = _log_uniform(g, 1e3, 1e10, n), _log_uniform(g, 1e3, 1e10, n)
    eff[kind == 0] = 0.0
    rd[kind == 1] = 0.0
    wr[kind == 1] = 0.0
    return batched.KernelMetricsBatch(eff, rd, wr, (_randint(g, 0, 8, n) != 0).to(torch.uint8))


def _host_arrays(kb):
    return {f: getattr(kb, f).cpu().numpy() for f in ("num_blocks", "block_size", "regs_per_thread", "smem_bytes",
                                                      "run_time_ns", "gamma")}


def _queries(g, op, n):
    """[n, F] float32 features in the predictor's column order and [n] uint8 device rows."""
    if op == "linear":
        cols = [_randint(g, 0, 2, n), _log_uniform(g, 1, 3500, n), _log_uniform(g, 1, 32768, n),
                _log_uniform(g, 1, 32768, n)]
    elif op == "conv2d":
        cols = [_randint(g, 0, 2, n), _log_uniform(g, 1, 64, n), _log_uniform(g, 1, 256, n),
                _log_uniform(g, 3, 2048, n), _log_uniform(g, 3, 2048, n), _choice(g, [1, 3, 5, 7], n),
                _choice(g, [1, 2, 4], n), _randint(g, 0, 4, n)]
    elif op == "bmm":
        cols = [_log_uniform(g, 1, 512, n)] + [_log_uniform(g, 1, 4096, n) for _ in range(3)]
    else:
        cols = [_randint(g, 0, 2, n), _randint(g, 0, 2, n), _log_uniform(g, 1, 128, n), _log_uniform(g, 1, 512, n),
                _log_uniform(g, 32, 4096, n), _log_uniform(g, 32, 4096, n), _randint(g, 1, 5, n)]
    feats = torch.stack([c.float() for c in cols], dim=1).contiguous()
    return feats, _randint(g, 0, len(workloads.BENCH_DEVICES), n).to(torch.uint8)


def _predictor(g, op, precision):
    """A RuntimePredictor with weights, mu and sigma as a checkpoint would bring them."""
    pred = RuntimePredictor(op, LAYERS, WIDTH, precision=precision)
    gain = 2.0
    with torch.no_grad():
        for name, p in pred.model.named_parameters():
            layer = pred.model.get_submodule(name.rpartition(".")[0])
            bound = 1.0 / math.sqrt(layer.in_features)
            scale = gain if p.ndim == 2 and not name.startswith("fc2") else 1.0
            p.copy_((_uniform(g, -bound, bound, p.numel()) * scale).view_as(p).float())
        pred.model.fc2.bias.fill_(1.0)
    feats, rows = _queries(g, op, 1 << 14)
    pred.mu, pred.sigma = workloads.batch_mu_sigma(feats.cpu().numpy(), rows.cpu().numpy())
    return pred


def _handle(pred):
    return batched.MLPHandle(len(pred.model.features), mu=pred.mu, sigma=pred.sigma,
                             device_features=workloads.BENCH_DEVICE_FEATURES, precision=pred.precision,
                             **state_to_arrays(pred.model))


def _op_args(op, f):
    """The positional arguments torch would have been called with, from one feature row."""
    if op == "conv2d":
        bias, batch, image, cin, cout, ksz, stride, pad = f
        return ((batch, cin, image, image), (cout, cin, ksz, ksz), (cout,) if bias else None, (stride, stride),
                (pad, pad), (1, 1), 1)
    if op == "linear":
        bias, batch, fin, fout = f
        return ((batch, fin), (fout, fin), (fout,) if bias else None)
    batch, left, middle, right = f
    return ((batch, left, middle), (batch, middle, right))


def _operations(g, iterations, origin):
    """A recorded trace: per iteration 53 conv2d, 1 linear and 32 bmm operations and 74 others of
    one forward and one backward kernel each, seven in eight kernels with metrics."""
    n = iterations * workloads.ITER_KERNELS
    k = _host_arrays(_kernels(g, 2 * n, launchable=True))
    m = _metrics(g, 2 * n)
    eff, rd, wr, has = (getattr(m, f).tolist() for f in ("flop_efficiency_pct", "dram_read_bytes",
                                                         "dram_write_bytes", "has_metrics"))
    nb, bs, rg, sm, tm = (k[f].tolist() for f in ("num_blocks", "block_size", "regs_per_thread", "smem_bytes",
                                                  "run_time_ns"))
    overhead = _uniform(g, 0, 10_000, 2 * n).tolist()
    names = tuple(x.value.cupti_name for x in (Metric.SinglePrecisionFLOPEfficiency, Metric.DRAMReadBytes,
                                               Metric.DRAMWriteBytes))

    def run(i):
        metrics = list(zip(names, (eff[i], rd[i], wr[i]))) if has[i] else []
        c = KernelInstance("kernel_%d" % (i % 97), nb[i], bs[i], 0, sm[i], rg[i], int(tm[i]), metrics)
        return RunTimeMeasurement((tm[i] + overhead[i]) / 1e6, [MeasuredKernel(c, [c] if metrics else [], origin)],
                                  origin)

    special = {}
    for op in MLP_SHARE:
        count = iterations * workloads.ITER_SPECIAL[op]
        feats, _ = _queries(g, op, count)
        special[op] = feats.int().tolist(), torch.exp(_uniform(g, math.log(0.02), math.log(50.0), count)).tolist()
    out = []
    for it in range(iterations):
        for i in range(it * workloads.ITER_KERNELS, (it + 1) * workloads.ITER_KERNELS):
            out.append(MeasuredOperation("relu", Arguments((), {}), run(2 * i), run(2 * i + 1), origin))
        for op in MLP_SHARE:
            feats, ms = special[op]
            for j in range(it * workloads.ITER_SPECIAL[op], (it + 1) * workloads.ITER_SPECIAL[op]):
                out.append(MeasuredOperation(op, Arguments(_op_args(op, feats[j]), {}),
                                             RunTimeMeasurement(ms[j], [], origin), None, origin))
    return out


def prepare(case, seed):
    g = _generator(seed)
    kind = case["kind"]
    s = {"case": case, "kind": kind}
    if kind == "predict":
        s["pred"] = _predictor(g, case["op"], case["precision"])
        s["pred"].device_row(workloads.BENCH_DEVICES[0])
        feats, rows = _queries(g, case["op"], case["calls"])
        s["queries"] = [(f, workloads.BENCH_DEVICES[r]) for f, r in zip(feats.tolist(), rows.tolist())]
    elif kind == "mlp":
        s["handle"] = _handle(_predictor(g, case["op"], case["precision"]))
        s["feats"], s["rows"] = _queries(g, case["op"], case["queries"])
        if case["host"]:
            s["feats"], s["rows"] = s["feats"].cpu().numpy(), s["rows"].cpu().numpy()
    elif kind in ("wave", "host", "pipeline"):
        K, D = case["kernels"], case["dests"]
        s["origin"], s["dests"] = _devices(D)
        if kind == "wave":
            s["kernels"] = _kernels(g, K)
            if case["variant"] == "metrics":
                s["metrics"] = _metrics(g, K)
                # the register table knows about half of the kernels on a destination
                regs = _randint(g, 16, 256, D * K).view(D, K)
                s["regs"] = torch.where(_randint(g, 0, 2, D * K).view(D, K) == 0, -1, regs).to(torch.int16)
            elif case["variant"] == "totals":
                s["partials"] = batched.WavePartials(K, D)
        elif kind == "host":
            s["arrays"] = _host_arrays(_kernels(g, K))
        else:
            s["pipe"] = hostio.WaveScaleHost(s["origin"], s["dests"], K)
            s["blocks"] = [hostio.pack_kernels(_host_arrays(_kernels(g, K))) for _ in range(s["pipe"].depth)]
    elif kind == "trace":
        s["origin"], dests = _devices(6)
        s["dests"] = dests[1:]
        s["predictor"] = Predictor()
        for op in MLP_SHARE:
            pred = _predictor(g, op, "bf16")
            pred.device_row(s["origin"].name)
            setattr(s["predictor"], op + "_pred", pred)
        s["operations"] = _operations(g, case["iterations"], s["origin"])
        if case["again"]:
            s["trace"] = Trace(s["origin"], s["operations"])
            s["trace"].to_devices(s["dests"], s["predictor"])
    else:
        I = case["iterations"]
        s["origin"], s["dests"] = _devices(6)
        s["kernels"] = _kernels(g, I * workloads.ITER_KERNELS, launchable=True)
        s["overhead"] = _uniform(g, 0, 10_000, I * workloads.ITER_KERNELS).float()
        s["offsets"] = torch.arange(I + 1, device="cuda") * workloads.ITER_KERNELS
        s["special"] = {}
        for op in MLP_SHARE:
            n = I * workloads.ITER_SPECIAL[op]
            handle = _handle(_predictor(g, op, "bf16"))
            feats, _ = _queries(g, op, n)
            ms = torch.exp(_uniform(g, math.log(0.02), math.log(50.0), n)).float()
            s["special"][op] = iteration.SpecialOps(handle, feats, ms, torch.arange(I + 1, device="cuda")
                                                    * workloads.ITER_SPECIAL[op])
    return s


# ---------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------
def _wave_planes(res):
    """The planes of a WaveResult; unsigned 32-bit ones as int32 (same bits)."""
    out = [res.scaled_ns, res.dest_occupancy, res.dest_waves.view(torch.int32), res.origin_occupancy,
           res.origin_waves.view(torch.int32)]
    return out if res.status is None else out + [res.status]


def run(s):
    case, kind = s["case"], s["kind"]
    if kind == "predict":
        pred = s["pred"]
        return [pred.predict(f, name) for f, name in s["queries"]]
    if kind == "mlp":
        if case["host"]:
            return s["handle"].predict_host(s["feats"], s["rows"])
        out = s["handle"].predict(s["feats"], s["rows"])
        if case["totals"]:
            return out, batched.group_sum(out, s["rows"], len(workloads.BENCH_DEVICES))
        return out
    if kind == "wave":
        variant = case["variant"]
        if variant == "metrics":
            return _wave_planes(batched.wave_scale(s["kernels"], s["origin"], s["dests"], dest_regs=s["regs"],
                                                   metrics=s["metrics"]))
        if variant == "totals":
            res = batched.wave_scale(s["kernels"], s["origin"], s["dests"], partials=s["partials"])
            return _wave_planes(res) + [s["partials"].totals()]
        return _wave_planes(batched.wave_scale(s["kernels"], s["origin"], s["dests"],
                                               want_status=variant == "status"))
    if kind == "host":
        res = batched.wave_scale_host(s["arrays"], s["origin"], s["dests"])
        return [res[k] for k in ("scaled_ns", "dest_occupancy", "dest_waves", "origin_occupancy", "origin_waves")]
    if kind == "pipeline":
        pipe = s["pipe"]
        for slot, block in enumerate(s["blocks"]):
            pipe.submit(block, slot)
        for slot in range(pipe.depth):
            pipe.wait(slot)
        return [out["scaled_ns"] for out in pipe.host_out]
    if kind == "trace":
        trace = s["trace"] if case["again"] else Trace(s["origin"], s["operations"])
        out = []
        for predicted in trace.to_devices(s["dests"], s["predictor"]):
            out += [predicted.run_time_ms, predicted.operations.run_times_ms]
        return out
    totals, res = iteration.predict_iteration_totals(
        s["kernels"], s["overhead"], s["offsets"], s["special"], s["origin"], s["dests"], 0, range(6))
    return [totals] + _wave_planes(res)


# ---------------------------------------------------------------------------
# What one pass cannot do without
# ---------------------------------------------------------------------------
def _mlp_work(op, queries, precision):
    F = len(workloads.OP_FEATURES[op])
    params = (F + 4) * WIDTH + LAYERS * WIDTH * WIDTH + WIDTH
    return params * (2 if precision == "bf16" else 4) + queries * (4 * F + 1 + 4), 2 * params * queries


def _wave_bytes(K, D, variant):
    per_kernel, per_pair = 20 + 5, 9
    if variant == "metrics":
        per_kernel, per_pair = 16 + 25 + 5, 9 + 2
    elif variant == "status":
        per_pair += 1
    return K * per_kernel + K * D * per_pair


def work(case):
    kind = case["kind"]
    if kind == "predict":
        b, f = _mlp_work(case["op"], case["calls"], case["precision"])
    elif kind == "mlp":
        b, f = _mlp_work(case["op"], case["queries"], case["precision"])
    elif kind in ("wave", "host"):
        b, f = _wave_bytes(case["kernels"], case["dests"], case.get("variant", "plain")), 0
    elif kind == "pipeline":
        b, f = 3 * case["kernels"] * (20 + 4 * case["dests"]), 0
    else:
        passes = 1 if kind == "iterations" else 2        # kernels per ordinary operation
        targets = 6                                      # the origin and five destinations
        b, f = _wave_bytes(case["iterations"] * workloads.ITER_KERNELS * passes, targets, "plain"), 0
        for op in MLP_SHARE:
            mb, mf = _mlp_work(op, case["iterations"] * workloads.ITER_SPECIAL[op] * targets, "bf16")
            b, f = b + mb, f + mf
    return {"bytes": b, "flops": f}


def tolerance(case):
    """Integers exactly; scaled times 1e-6 (a 32-bit exponential); predictions what bfloat16 (1e-2)
    or split (1e-5: 32-bit sums of 16-bit hi + lo parts) operands give."""
    if case["kind"] in ("wave", "host", "pipeline"):
        return {"rel": 1e-6, "max": 2e-6}
    if case.get("precision") == "bf16x3":
        return {"rel": 1e-5}
    return {"rel": 1e-2}
