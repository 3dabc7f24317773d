"""Mixed iteration traces: per-iteration totals on the device against the oracle.

The shape of one iteration follows the benchmark's mixed trace: 53 conv2d, 1 linear
and 32 bmm operations predicted by their MLPs plus 74 ordinary operations of one
wave-scaled kernel each; totals within 2e-2 relative of the float64 reference.
"""
import numpy as np
import pytest
import torch

from habitat_b200 import batched, iteration, workloads
from oracle import mlp as omlp
from oracle import wave as owave

pytestmark = pytest.mark.gpu

PER_ITER = {"conv2d": 53, "linear": 1, "bmm": 32}
KERNELS_PER_ITER = 74


def _make(I, seed, origin_spec):
    def occ(block, smem, regs):
        return np.array([owave.occupancy(origin_spec, b, s, r)[0] for b, s, r in zip(block, smem, regs)])
    kernels = workloads.make_kernels(I * KERNELS_PER_ITER, seed, valid_only=True, origin=occ)
    g = workloads.rng(seed + 1)
    overhead = g.uniform(0, 10_000, size=I * KERNELS_PER_ITER).astype(np.float32)      # ns
    ops = {}
    for op, n in PER_ITER.items():
        feats, _ = workloads.make_queries(op, I * n, seed + 7 + len(op))
        rt = np.exp(g.uniform(np.log(0.02), np.log(50.0), size=I * n)).astype(np.float32)
        ops[op] = (feats, rt)
    return kernels, overhead, ops


@pytest.mark.parametrize("I", [3, 64, 512])
def test_iteration_totals(bench_devices, I):
    origin, dests = bench_devices[0], bench_devices
    kernels, overhead, ops = _make(I, 4004, origin.spec_tuple())
    koff = np.arange(I + 1, dtype=np.int64) * KERNELS_PER_ITER
    devf = workloads.BENCH_DEVICE_FEATURES

    special, weights, stats = {}, {}, {}
    for op, (feats, rt) in ops.items():
        w = workloads.torch_init_mlp_weights(op)
        dev_all = np.tile(np.arange(6, dtype=np.uint8), len(feats))[:len(feats)]
        mu, sigma = workloads.batch_mu_sigma(feats, dev_all)
        weights[op], stats[op] = w, (mu, sigma)
        h = batched.MLPHandle(feats.shape[1], mu=mu, sigma=sigma, device_features=devf, **w)
        off = torch.from_numpy(np.arange(I + 1, dtype=np.int64) * PER_ITER[op]).cuda()
        special[op] = iteration.SpecialOps(h, torch.from_numpy(feats).cuda(), torch.from_numpy(rt).cuda(), off)

    totals, wave = iteration.predict_iteration_totals(
        batched.KernelBatch.from_numpy(kernels), torch.from_numpy(overhead).cuda(),
        torch.from_numpy(koff).cuda(), special, origin, dests, 0, list(range(6)))
    torch.cuda.synchronize()
    for s in special.values():
        s.handle.check_status()
    got = totals.cpu().numpy()
    assert not torch.isnan(wave.scaled_ns).any()       # valid-only kernels never raise
    assert batched.wave_scale_path() == "wave_scale_lut_kernel"

    # reference: the oracle, float64, operation by operation
    specs = [d.spec_tuple() for d in dests]
    ref = owave.wave_scale_batch(specs, 0, list(range(6)), kernels, want_limits=False)
    want = np.zeros((I, 6))
    for d in range(6):
        ns = kernels["run_time_ns"] if d == 0 else ref["scaled_ns"][d]     # row 0 is the origin itself
        want[:, d] = (overhead.astype(np.float64) + ns).reshape(I, -1).sum(axis=1) / 1e6
    for op, (feats, rt) in ops.items():
        mu, sigma = stats[op]
        n = len(feats)
        p_orig = omlp.predict(weights[op], feats, np.zeros(n, np.uint8), devf, mu, sigma, np.float64)
        for d in range(6):
            if d == 0:
                ms = rt.astype(np.float64)
            else:
                p_dest = omlp.predict(weights[op], feats, np.full(n, d, np.uint8), devf, mu, sigma, np.float64)
                ms = np.maximum(rt.astype(np.float64) * p_dest / p_orig, 0)
            want[:, d] += ms.reshape(I, -1).sum(axis=1)
    assert np.abs(got - want).max() <= 2e-2 * np.abs(want).min()
    assert np.abs(got[:, 0] - want[:, 0]).max() <= 1e-6 * want[:, 0].max()   # identity column
    print("config-4 style totals, max rel err %.3g" % (np.abs(got - want) / want).max())


def test_strided_features_and_longer_overheads(bench_devices):
    """Features of any layout and overheads beyond the kernels are taken; the totals are those of plain arrays."""
    I, origin, dests = 3, bench_devices[0], bench_devices
    kernels, overhead, ops = _make(I, 77, origin.spec_tuple())
    feats, rt = ops["bmm"]
    mu, sigma = workloads.batch_mu_sigma(feats, np.tile(np.arange(6, dtype=np.uint8), len(feats))[:len(feats)])
    h = batched.MLPHandle(4, mu=mu, sigma=sigma, device_features=workloads.BENCH_DEVICE_FEATURES,
                          **workloads.torch_init_mlp_weights("bmm"))
    off = torch.arange(I + 1, device="cuda") * PER_ITER["bmm"]
    koff = torch.arange(I + 1, device="cuda") * KERNELS_PER_ITER
    f = torch.from_numpy(feats).cuda()
    over = torch.from_numpy(overhead).cuda()

    def totals(features, overheads):
        special = {"bmm": iteration.SpecialOps(h, features, torch.from_numpy(rt).cuda(), off)}
        return iteration.predict_iteration_totals(batched.KernelBatch.from_numpy(kernels), overheads, koff, special,
                                                  origin, dests, 0, list(range(6)))[0]
    want = totals(f, over)
    strided = f.t().contiguous().t()
    assert not strided.is_contiguous()
    assert torch.equal(totals(strided, over), want)
    assert torch.equal(totals(f, torch.cat([over, torch.full((5,), float("nan"), device="cuda")])), want)
    h.close()


def test_predictors_with_a_predict_of_their_own(bench_devices):
    """Handles and runtime predictors that predict otherwise are asked, side by side with ordinary ones: totals and
    traces follow their predictions."""
    from habitat_b200.analysis.arguments import Arguments
    from habitat_b200.analysis.mlp.mlp import RuntimePredictor
    from habitat_b200.analysis.operation import MeasuredOperation
    from habitat_b200.analysis.predictor import Predictor
    from habitat_b200.analysis.run_time import RunTimeMeasurement
    from habitat_b200.analysis.trace import Trace
    I, origin, dests = 3, bench_devices[0], bench_devices
    kernels, overhead, ops = _make(I, 78, origin.spec_tuple())
    koff = torch.arange(I + 1, device="cuda") * KERNELS_PER_ITER

    class Slower(batched.MLPHandle):
        def predict(self, op_features, device_row, out=None):
            return op_features[:, 0] * (1.0 + device_row.float())       # of device r: 1 + r times device 0's

    special = {}
    for op, cls in (("linear", batched.MLPHandle), ("bmm", Slower)):
        feats, rt = ops[op]
        mu, sigma = workloads.batch_mu_sigma(feats, np.tile(np.arange(6, dtype=np.uint8), len(feats))[:len(feats)])
        h = cls(4, mu=mu, sigma=sigma, device_features=workloads.BENCH_DEVICE_FEATURES,
                **workloads.torch_init_mlp_weights(op))
        special[op] = iteration.SpecialOps(h, torch.from_numpy(feats).cuda(), torch.from_numpy(rt).cuda(),
                                           torch.arange(I + 1, device="cuda") * PER_ITER[op])

    def totals(which):
        return iteration.predict_iteration_totals(batched.KernelBatch.from_numpy(kernels), torch.from_numpy(overhead).cuda(),
                                                  koff, which, origin, dests, 0, list(range(6)))[0].cpu().numpy()
    added = totals(special) - totals({"linear": special["linear"]})
    measured = ops["bmm"][1].astype(np.float64).reshape(I, -1).sum(axis=1)
    np.testing.assert_allclose(added, measured[:, None] * np.arange(1, 7), rtol=1e-6)

    class Slow(RuntimePredictor):
        def predict_batch(self, op_features, device_rows):
            return op_features[:, 1] * torch.where(device_rows == self.device_row(origin.name), 1.0, 5.0)

    predictor = Predictor()
    for cls, op in ((Slow, "linear"), (RuntimePredictor, "bmm")):
        pred = cls(op, 2, 1024)
        with torch.no_grad():
            pred.model.fc2.bias.fill_(1.0)
        pred.mu, pred.sigma = np.zeros(8), np.full(8, 1e4)
        setattr(predictor, op + "_pred", pred)
    run = RunTimeMeasurement(0.5, [], origin)
    trace = Trace(origin, [MeasuredOperation("linear", Arguments(((8, 16), (32, 16), None), {}), run, None, origin),
                           MeasuredOperation("bmm", Arguments(((4, 8, 16), (4, 16, 8)), {}), run, run, origin)])
    for got in trace.to_devices(dests[1:], predictor):
        times = got.operations.run_times_ms
        assert times[0] == pytest.approx(2.5, rel=1e-6) and 0 < times[1] < 10
        assert got.run_time_ms == pytest.approx(times.sum(), rel=1e-12)


def _recorded(origin, n, seed, odd=None):
    """A trace of n conv2d, linear and bmm operations each among 2 n others of one or two kernels; `odd` replaces the
    arguments of one linear operation."""
    from habitat_b200.analysis.arguments import Arguments
    from habitat_b200.analysis.kernels import MeasuredKernel
    from habitat_b200.analysis.operation import MeasuredOperation
    from habitat_b200.analysis.run_time import RunTimeMeasurement
    from habitat_b200.analysis.trace import Trace
    from habitat_b200.habitat_cuda import KernelInstance
    g = workloads.rng(seed)

    def run(with_kernels):
        kernels = []
        for _ in range(int(g.integers(1, 3)) if with_kernels else 0):
            c = KernelInstance("k%d" % g.integers(0, 9), int(g.integers(1, 5000)), 128, 0, 1024, 32,
                               int(g.integers(2000, 10 ** 6)), [])
            kernels.append(MeasuredKernel(c, [], origin))
        return RunTimeMeasurement(float(g.uniform(0.5, 40.0)), kernels, origin)

    ops = []
    for i in range(n):
        b, f = int(g.integers(1, 64)), int(g.integers(16, 512))
        linear = Arguments(((b, f), (f, f), None), {}) if odd is None or i else odd
        for name, args in (("conv2d", Arguments(((b, 3, 32, 32), (f, 3, 3, 3), (f,), (1, 1), (1, 1), (1, 1), 1), {})),
                           ("linear", linear), ("bmm", Arguments(((b, f, 16), (b, 16, f)), {}))):
            ops.append(MeasuredOperation(name, args, run(False), run(False) if i % 2 else None, origin))
            ops.append(MeasuredOperation("relu", Arguments((), {}), run(True), run(True) if i % 3 else None, origin))
    return Trace(origin, ops)


@pytest.mark.parametrize("n", [1, 7, 200])
def test_predictors_started_during_the_walk(bench_devices, monkeypatch, n):
    """The first prediction of a trace starts its predictors before the kernels are walked; a later one, or one whose
    predictors cannot be started then (an operation recorded by keyword), runs them afterwards.  All of them give the
    same bits, for other destinations than the first ones as well, and with predictors changed in between."""
    from habitat_b200 import _native
    from habitat_b200.analysis.arguments import Arguments
    from habitat_b200.analysis.mlp.mlp import RuntimePredictor
    from habitat_b200.analysis.predictor import Predictor
    origin, dests = bench_devices[0], bench_devices[1:]

    def predictor(seed):
        p = Predictor()
        for k, op in enumerate(("conv2d", "linear", "bmm")):
            torch.manual_seed(seed + k)
            pred = RuntimePredictor(op, 2, 1024)
            F = len(pred.model.features)
            pred.mu, pred.sigma = np.full(F + 4, 10.0), np.full(F + 4, 50.0)
            pred.model.fc2.bias.data.fill_(1.0)
            setattr(p, op + "_pred", pred)
        return p

    def result(trace, targets, p):
        return [(t.run_time_ms, t.operations.run_times_ms.tobytes()) for t in trace.to_devices(targets, p)]

    started = []
    real = Predictor._start_kinds
    monkeypatch.setattr(Predictor, "_start_kinds", lambda self, *a: started.append(real(self, *a)) or started[-1])
    p, q = predictor(1), predictor(5)
    trace = _recorded(origin, n, 3)
    first = result(trace, dests, p)
    assert started.pop() is not None
    assert result(trace, dests, p) == first and result(trace, dests[:2], p) == first[:2] and not started
    other = result(trace, dests, q)
    assert other != first and result(_recorded(origin, n, 3), dests, q) == other and started.pop() is not None
    # not started: the same results
    monkeypatch.setattr(Predictor, "_start_kinds", lambda self, *a: None)
    assert result(_recorded(origin, n, 3), dests, p) == first
    monkeypatch.setattr(Predictor, "_start_kinds", lambda self, *a: started.append(real(self, *a)) or started[-1])
    by_keyword = Arguments(((4, 32), (64, 32)), {"bias": None})
    result(_recorded(origin, n, 3, by_keyword), dests, p)
    assert started.pop() is None
    # started, and the walk then finds something that is not ordinary: the general path has the same results
    class Named(type(trace.operations[1].forward.kernels[0])):
        pass
    strange = _recorded(origin, n, 3)
    kernel = strange.operations[-1].forward.kernels[0]
    kernel.__class__ = Named
    got = result(strange, dests, p)
    assert started.pop() is not None
    for (a, b), (c, d) in zip(got, first):
        assert np.allclose(np.frombuffer(b), np.frombuffer(d), rtol=1e-12) and np.isclose(a, c, rtol=1e-12)
    # results of other kinds than were started are refused, and of other devices
    capsule, kinds = real(p, *_special_of(trace), origin, dests, len(trace.operations))
    turned = [(h, f, ms, rows[:1] + rows[:0:-1], idx) for h, f, ms, rows, idx in kinds]
    for wrong in ([], turned):
        with pytest.raises(TypeError, match="other kinds"):
            _native.binding().run_group(None, None, origin, dests, None, None, wrong, (b"", b"", b"", b""),
                                        np.empty((5, 0), np.float32), np.empty((5, 0)),
                                        np.empty((5, len(trace.operations))), capsule)


def test_started_predictors_are_of_one_prediction(bench_devices):
    """Predictions of one trace that come between the first one's start of its predictors and its end, in the same thread
    after an interruption, from another stream as soon as the plan can be found, and from other threads: each has the
    results of its own destinations."""
    import threading
    from habitat_b200.analysis.arguments import Arguments
    from habitat_b200.analysis.mlp.mlp import RuntimePredictor
    from habitat_b200.analysis.operation import MeasuredOperation
    from habitat_b200.analysis.predictor import Predictor
    from habitat_b200.analysis.run_time import RunTimeMeasurement
    origin, dests = bench_devices[0], bench_devices[1:]
    p = Predictor()
    for k, op in enumerate(("conv2d", "linear", "bmm")):
        torch.manual_seed(k)
        pred = RuntimePredictor(op, 2, 1024)
        F = len(pred.model.features)
        pred.mu, pred.sigma = np.full(F + 4, 10.0), np.full(F + 4, 50.0)
        pred.model.fc2.bias.data.fill_(1.0)
        setattr(p, op + "_pred", pred)

    def result(trace, targets):
        return [t.operations.run_times_ms.tobytes() for t in trace.to_devices(targets, p)]

    class Meanwhile(dict):
        """Calls a function as soon as a plan can be found."""
        def __setitem__(self, key, plan):
            super().__setitem__(key, plan)
            if key[0] == "whole" and self.then is not None:
                then, self.then = self.then, None
                then()

    class Interrupted(RunTimeMeasurement):
        @property
        def run_time_ms(self):
            if raising:
                raise raising.pop()
            return 2.0

    raising = []

    def recorded():
        trace = _recorded(origin, 60, 11)
        trace.operations.append(MeasuredOperation("gru", Arguments((), {}), Interrupted(2.0, [], origin), None, origin))
        return trace

    want, turned = result(recorded(), dests), result(recorded(), dests[::-1])
    assert want == turned[::-1] and want != turned
    trace = recorded()
    raising.append(KeyboardInterrupt())
    with pytest.raises(KeyboardInterrupt):
        trace.to_devices(dests, p)
    assert result(trace, dests[::-1]) == turned

    trace, seen, other = recorded(), [], torch.cuda.Stream()
    trace._prediction_cache = Meanwhile()

    def on_another_stream():
        with torch.cuda.stream(other):
            seen.append(result(trace, dests[::-1]))
    trace._prediction_cache.then = on_another_stream
    assert result(trace, dests) == want and seen == [turned]

    for _ in range(10):
        trace, results = recorded(), {}
        start = threading.Barrier(4)

        def predict(i):
            with torch.cuda.stream(torch.cuda.Stream()):
                start.wait()
                results[i] = result(trace, dests if i % 2 else dests[::-1])
        threads = [threading.Thread(target=predict, args=(i,)) for i in range(4)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        assert results == {i: want if i % 2 else turned for i in range(4)}


def _special_of(trace):
    """What the walk hands over before it looks at the kernels."""
    plan = next(v for k, v in trace._prediction_cache.items() if k[0] == "whole")
    return ([plan.mlp_inputs[k][:2] for k in ("conv2d", "linear", "bmm")],
            [plan.mlp_idx[k].tobytes() for k in ("conv2d", "linear", "bmm")])


def test_operations_removed_during_the_walk(bench_devices):
    """A list of operations that is emptied while the predictors are started (another thread can): the walk over their
    kernels still has them, and records what it would have."""
    import gc
    import weakref
    from habitat_b200.analysis.predictor import _GroupPlan
    want = _GroupPlan.of_whole_trace(_recorded(bench_devices[0], 20, 5).operations, "unified", False)
    operations = _recorded(bench_devices[0], 20, 5).operations
    alive = [weakref.ref(op) for op in operations]

    def early(inputs, indices):
        operations.clear()
        gc.collect()
        assert all(ref() is not None for ref in alive)     # (before the walk goes on to them)
    got = _GroupPlan.of_whole_trace(operations, "unified", False, early)
    assert not operations and got.n_kernels == want.n_kernels > 0
    for name, plane in vars(want.flat.batch).items():
        assert torch.equal(plane, getattr(got.flat.batch, name)), name
    assert np.array_equal(got.overheads, want.overheads) and np.array_equal(got.wave_idx, want.wave_idx)


def test_traces_whose_predictors_cannot_start_go_up_in_one_piece(bench_devices):
    """An lstm operation, or one recorded by keyword, keeps the predictors from starting during the walk: features and
    records then are one upload, and nothing has to be kept for it."""
    from habitat_b200.analysis.arguments import Arguments
    from habitat_b200.analysis.operation import MeasuredOperation
    from habitat_b200.analysis.predictor import _GroupPlan
    from habitat_b200.analysis.run_time import RunTimeMeasurement
    origin = bench_devices[0]
    lstm = MeasuredOperation("lstm", Arguments(((12, 4, 64), ((2, 4, 128),), (), True, 2, 0.0, False, False, False), {}),
                             RunTimeMeasurement(1.5, [], origin), None, origin)
    plain, keyword = _recorded(origin, 5, 9), _recorded(origin, 5, 9, Arguments(((4, 32), (64, 32)), {"bias": None}))
    for operations, together in ((plain.operations, False), (plain.operations + [lstm], True), (keyword.operations, True)):
        asked, first = [], []
        plan = _GroupPlan.of_whole_trace(operations, "unified", False, lambda *a: asked.append(a) or "started", first)
        one = plan.mlp_inputs["conv2d"][0].untyped_storage().data_ptr() == \
            plan.flat.batch.num_blocks.untyped_storage().data_ptr()
        assert one == together and [a[0] is None for a in asked] == [together]
        assert first[0] == (None if together else "started") and (first[1] is None) == together
