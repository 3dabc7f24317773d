"""Fused MLP predictor kernel (through the C ABI) against the numpy oracle."""
import numpy as np
import pytest
import torch

from habitat_b200 import batched, workloads
from oracle import mlp as omlp

pytestmark = pytest.mark.gpu

DEVF = workloads.BENCH_DEVICE_FEATURES


def _run(op, Q, weights, precision, seed, mu_sigma=None):
    feats, dev = workloads.make_queries(op, Q, seed)
    mu, sigma = mu_sigma if mu_sigma is not None else workloads.batch_mu_sigma(feats, dev)
    h = batched.MLPHandle(feats.shape[1], mu=mu, sigma=sigma, device_features=DEVF,
                          precision=precision, **weights)
    out = h.predict(torch.from_numpy(feats).cuda(), torch.from_numpy(dev).cuda())
    torch.cuda.synchronize()
    h.check_status()
    got = out.cpu().numpy()
    ref32 = omlp.predict(weights, feats, dev, DEVF, mu, sigma, np.float32)
    ref64 = omlp.predict(weights, feats, dev, DEVF, mu, sigma, np.float64)
    h.close()
    return got, ref32, ref64


def _rel(got, ref):
    return np.abs(got.astype(np.float64) - ref) / np.abs(ref)


@pytest.mark.parametrize("op", ["linear", "conv2d", "bmm", "lstm"])
def test_bf16_reference_init(op):
    """Weights as the reference initialises a fresh predictor; tolerance 2e-2
    relative for the bf16 tensor-core path (float32 reference)."""
    w = workloads.torch_init_mlp_weights(op)
    got, ref32, ref64 = _run(op, 4096, w, "bf16", seed=1003)
    assert np.isfinite(got).all()
    assert _rel(got, ref32).max() <= 2e-2
    print(op, "bf16 max rel", _rel(got, ref64).max())


@pytest.mark.parametrize("Q", [1, 63, 64, 65, 127, 129, 4096 + 17, 4224 + 1, 4224 + 17, 4224 + 127])
def test_tile_tails(Q):
    """Odd sizes; from 4,225 on on the two-SM kernel, with a last tile of 1, 17 and 127 queries."""
    w = workloads.torch_init_mlp_weights("conv2d")
    feats, dev = workloads.make_queries("conv2d", 8192, 77)
    mu_sigma = workloads.batch_mu_sigma(feats, dev)
    got, ref32, _ = _run("conv2d", Q, w, "bf16", seed=77, mu_sigma=mu_sigma)
    assert got.shape == (Q,)
    assert _rel(got, ref32).max() <= 2e-2


@pytest.mark.parametrize("op", ["linear", "conv2d"])
def test_bf16_input_sensitive(op):
    """Random-init predictors are nearly constant functions, so a kernel that
    ignored its inputs would pass the case above.  Scaling fc1 and hidden
    weights by sqrt(6) keeps the activation variance through the stack and makes
    the output move with the input; errors are then judged against the spread
    of the outputs (single-pass bf16: a few percent worst case)."""
    w = workloads.init_mlp_weights(op, seed=11, gain=np.sqrt(6.0))
    got, ref32, ref64 = _run(op, 4096, w, "bf16", seed=1004)
    spread = ref64.std()
    assert spread > 0.05 * np.abs(ref64).mean()          # the outputs do vary
    err = np.abs(got - ref64)
    assert err.max() <= 8e-2 * spread + 2e-2 * np.abs(ref64).max()
    assert err.mean() <= 1e-2 * spread + 4e-3 * np.abs(ref64).mean()
    assert np.corrcoef(got, ref64)[0, 1] > 0.999


@pytest.mark.parametrize("op", ["linear", "lstm"])
def test_split_precision_config1(op):
    """hi/lo split path: 1e-4 relative against the float32 reference."""
    w = workloads.torch_init_mlp_weights(op)
    got, ref32, ref64 = _run(op, 2048 + 5, w, "bf16x3", seed=1001)
    assert _rel(got, ref32).max() <= 1e-4
    print(op, "bf16x3 max rel vs fp64", _rel(got, ref64).max())


def test_split_precision_input_sensitive():
    w = workloads.init_mlp_weights("linear", seed=12, gain=np.sqrt(6.0))
    got, ref32, ref64 = _run("linear", 2048, w, "bf16x3", seed=1005)
    err = np.abs(got - ref64)
    assert err.max() <= 2e-4 * (ref64.std() + np.abs(ref64).max())


def test_wide_sigma_and_negative_outputs():
    """sigma spanning 1 .. 1e4 and a weight set whose outputs go negative."""
    op = "conv2d"
    w = workloads.init_mlp_weights(op, seed=13, gain=np.sqrt(6.0))
    w["fc2_b"] = w["fc2_b"] - 0.5
    feats, dev = workloads.make_queries(op, 4096, 1006)
    mu, sigma = workloads.batch_mu_sigma(feats, dev)
    sigma = sigma * np.logspace(0, 4, sigma.shape[0]) / sigma.max()
    got, ref32, ref64 = _run(op, 4096, w, "bf16", seed=1006, mu_sigma=(mu, sigma))
    assert (ref64 < 0).any()
    err = np.abs(got - ref64)
    assert err.max() <= 8e-2 * ref64.std() + 2e-2 * np.abs(ref64).max()


def test_host_buffer_entry_point():
    op = "bmm"
    w = workloads.torch_init_mlp_weights(op)
    feats, dev = workloads.make_queries(op, 1000, 5)
    mu, sigma = workloads.batch_mu_sigma(feats, dev)
    h = batched.MLPHandle(4, mu=mu, sigma=sigma, device_features=DEVF, **w)
    got = h.predict_host(feats, dev)
    ref = omlp.predict(w, feats, dev, DEVF, mu, sigma)
    assert _rel(got, ref).max() <= 2e-2
    h.close()


@pytest.mark.parametrize("precision,Q", [("bf16", 74 * 128 * 3 + 77), ("bf16x3", 148 * 32 * 2 + 5)])
def test_repeatable(precision, Q):
    """The kernel's roles hand tiles, accumulators and activations to one another through
    barriers; a missing hand-over shows as results that change from launch to launch long
    before it breaks a tolerance.  Same inputs, several launches (each cluster walks more than
    one tile): bit-identical outputs."""
    w = workloads.init_mlp_weights("conv2d", seed=5, gain=np.sqrt(6.0))
    feats, dev = workloads.make_queries("conv2d", Q, 31)
    mu, sigma = workloads.batch_mu_sigma(feats, dev)
    h = batched.MLPHandle(feats.shape[1], mu=mu, sigma=sigma, device_features=DEVF,
                          precision=precision, **w)
    f, r = torch.from_numpy(feats).cuda(), torch.from_numpy(dev).cuda()
    first = h.predict(f, r).clone()
    for _ in range(8):
        again = h.predict(f, r)
        assert torch.equal(first, again)
    torch.cuda.synchronize()
    h.check_status()
    h.close()


@pytest.mark.parametrize("precision", ["bf16", "bf16x3"])
@pytest.mark.parametrize("layers", [1, 2, 3, 5])
def test_layer_by_layer(layers, precision):
    """The fused chain does not expose its activations, so each depth is checked instead: the same
    stack cut after 1, 2, 3, 5 hidden layers (own fc2 each) at 129 queries - one full tile plus one
    query - with weights that keep the activations input-dependent.  A layer that went wrong shows
    at its depth and not only in the full eight-layer result."""
    w = workloads.init_mlp_weights("bmm", seed=40 + layers, layers=layers, gain=np.sqrt(6.0))
    got, ref32, ref64 = _run("bmm", 129, w, precision, seed=1005)
    spread = ref64.std()
    err = np.abs(got - ref64)
    if precision == "bf16":
        assert err.max() <= 8e-2 * spread + 2e-2 * np.abs(ref64).max()
    else:
        assert err.max() <= 2e-4 * (spread + np.abs(ref64).max())


def test_empty_and_single_query():
    w = workloads.torch_init_mlp_weights("linear")
    feats, dev = workloads.make_queries("linear", 16, 3)
    mu, sigma = workloads.batch_mu_sigma(feats, dev)
    for precision in ("bf16", "bf16x3"):
        h = batched.MLPHandle(4, mu=mu, sigma=sigma, device_features=DEVF, precision=precision, **w)
        none = h.predict(torch.from_numpy(feats[:0]).cuda(), torch.from_numpy(dev[:0]).cuda())
        one = h.predict(torch.from_numpy(feats[:1]).cuda(), torch.from_numpy(dev[:1]).cuda())
        torch.cuda.synchronize()
        h.check_status()
        assert none.shape == (0,) and one.shape == (1,)
        ref = omlp.predict(w, feats[:1], dev[:1], DEVF, mu, sigma, np.float32)
        assert abs(float(one[0]) - ref[0]) <= 2e-2 * abs(ref[0])
        h.close()


def test_timeout_status_is_reported_once():
    """The error path of a bounded device-side wait, driven from the host: the status word a kernel
    would leave is written by hand, the next status check reports HB_ERR_DEVICE_TIMEOUT with the
    site, and the word is cleared so that later launches are judged on their own."""
    from habitat_b200 import _native
    w = workloads.torch_init_mlp_weights("bmm")
    feats, dev = workloads.make_queries("bmm", 300, seed=5)
    mu, sigma = workloads.batch_mu_sigma(feats, dev)
    h = batched.MLPHandle(feats.shape[1], mu=mu, sigma=sigma,
                          device_features=workloads.BENCH_DEVICE_FEATURES, **w)
    d_f, d_r = torch.from_numpy(feats).cuda(), torch.from_numpy(dev).cuda()
    first = h.predict(d_f, d_r).cpu().numpy()
    h.check_status()
    h.inject_status(0x212)                       # "MMA issuer gave up waiting for weights"
    with pytest.raises(_native.HabitatNativeError) as err:
        h.check_status()
    assert err.value.status == _native.HB_ERR_DEVICE_TIMEOUT and "0x212" in str(err.value)
    h.check_status()                             # reported once
    h.inject_status(0x311)
    with pytest.raises(_native.HabitatNativeError) as err:
        h.predict_host(feats, dev)               # the host-buffer entry point checks the word itself
    assert err.value.status == _native.HB_ERR_DEVICE_TIMEOUT
    again = h.predict(d_f, d_r).cpu().numpy()
    h.check_status()
    assert np.array_equal(first, again)
    h.close()


@pytest.mark.parametrize("precision,sizes", [("bf16", (1, 30, 100, 200, 300, 500, 600, 900, 1000, 1400, 1700, 2000, 4200)),
                                             ("bf16x3", (1, 14, 15, 50, 100, 200, 250, 300, 400, 500, 700, 900, 1000, 2100))])
def test_launches_that_find_the_mark_of_one_that_gave_up(precision, sizes):
    """Every shape of the small-batch kernels: a launch that finds the mark in its scratch (left by the host here) stores no
    result, reports 0x5ff and ends soon; after the report the scratch starts over and the results are what they were.
    Soon: the roles leave one after the other, up to three of them, when 64 try_waits of at most some 7,800 cycles each
    have brought nothing: 1.5 M cycles, 1.5 ms at 1 GHz."""
    from habitat_b200 import _native
    w = workloads.init_mlp_weights("linear", seed=31, gain=2.0, layers=8)
    feats, dev = workloads.make_queries("linear", max(sizes), 53)
    mu, sigma = workloads.batch_mu_sigma(feats, dev)
    h = batched.MLPHandle(4, mu=mu, sigma=sigma, device_features=DEVF, precision=precision, **w)
    d_f, d_r = torch.from_numpy(feats).cuda(), torch.from_numpy(dev).cuda()
    begin, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    for Q in sizes:
        f, r, out = d_f[:Q].contiguous(), d_r[:Q].contiguous(), torch.empty((Q,), device="cuda")
        want = h.predict(f, r).clone()
        h.check_status()
        h.inject_mark()
        out.fill_(-7.0)
        begin.record()
        h.predict(f, r, out=out)
        end.record()
        torch.cuda.synchronize()
        assert (out == -7.0).all(), Q
        took = begin.elapsed_time(end)
        print("%s, %d queries: %.2f ms" % (precision, Q, took))
        assert took < 2.5, (Q, took)
        with pytest.raises(_native.HabitatNativeError, match="0x5ff"):
            h.check_status()
        assert torch.equal(h.predict(f, r), want), Q
        h.check_status()
    h.predict_host(feats[:1], dev[:1])
    h.inject_mark()
    with pytest.raises(_native.HabitatNativeError, match="0x5ff"):
        h.predict_host(feats[:1], dev[:1])
    assert np.array_equal(h.predict_host(feats[:1], dev[:1]), h.predict(d_f, d_r).cpu().numpy()[:1])
    h.check_status()
    h.close()


@pytest.mark.parametrize("precision,sizes", [("bf16", (100, 300, 500, 600, 900, 1200, 1700, 2000)),
                                             ("bf16x3", (50, 200, 250, 300, 400, 600, 900, 1000))])
def test_no_result_when_one_block_has_given_up(precision, sizes):
    """Each shape of the kernel for clusters of SM pairs: one block gives up, the second one
    of a pair without queries of the last sums, so that everybody else goes on to the end.  No block stores a result, and
    the launch ends as a whole."""
    from habitat_b200 import _native
    w = workloads.init_mlp_weights("linear", seed=31, gain=2.0, layers=2)
    feats, dev = workloads.make_queries("linear", max(sizes), 53)
    mu, sigma = workloads.batch_mu_sigma(feats, dev)
    h = batched.MLPHandle(4, mu=mu, sigma=sigma, device_features=DEVF, precision=precision, **w)
    d_f, d_r = torch.from_numpy(feats).cuda(), torch.from_numpy(dev).cuda()
    for Q in sizes:
        f, r, out = d_f[:Q].contiguous(), d_r[:Q].contiguous(), torch.empty((Q,), device="cuda")
        want = h.predict(f, r).clone()
        h.check_status()
        h.inject_mark(block=3)
        out.fill_(-7.0)
        h.predict(f, r, out=out)
        torch.cuda.synchronize()
        assert (out == -7.0).all(), Q
        with pytest.raises(_native.HabitatNativeError):
            h.check_status()
        assert torch.equal(h.predict(f, r), want), Q
        h.check_status()
    h.close()


@pytest.mark.parametrize("width,layers", [(256, 3), (1000, 2), (64, 1)])
def test_other_layer_sizes(width, layers):
    """RuntimePredictor(model_name, layers, layer_size) takes any size in the reference
    (analysis/mlp/mlp.py:113-131); widths up to 1024 run zero-padded on the 1024-wide kernel."""
    op = "lstm"
    w = workloads.init_mlp_weights(op, seed=width + layers, layers=layers, width=width, gain=np.sqrt(6.0))
    for precision, tol in (("bf16", 4e-2), ("bf16x3", 1e-4)):
        got, ref32, ref64 = _run(op, 700, w, precision, seed=width)
        spread = np.abs(ref64).max()
        assert np.abs(got - ref64).max() <= tol * spread, (precision, np.abs(got - ref64).max() / spread)
    with pytest.raises(_native_error()):
        wide = workloads.init_mlp_weights(op, seed=1, layers=1, width=1088)
        _run(op, 10, wide, "bf16", seed=1)


def _native_error():
    from habitat_b200 import _native
    return _native.HabitatNativeError


@pytest.mark.parametrize("op,gain,layers,bound", [
    # bounds: about three times the differences measured on a B200 (4.8e-4, 1.6e-3, 1.2e-4, 4.6e-4, 2.3e-3);
    # the replay itself is 7.7e-4 ... 8.4e-3 away from float64 on the same cases
    ("conv2d", 1.0, 8, 1.5e-3), ("linear", 1.0, 8, 5e-3), ("lstm", np.sqrt(6.0), 1, 4e-4),
    ("bmm", np.sqrt(6.0), 2, 1.5e-3), ("lstm", np.sqrt(6.0), 4, 7e-3)])
def test_bf16_mode_against_its_own_arithmetic(op, gain, layers, bound):
    """The bf16 kernel against a numpy replay of exactly its arithmetic (bfloat16 rounding of hidden
    weights and activations, float32 accumulation, split fc1).  What is left is the order of the
    float32 additions, which now and then tips an activation over a bfloat16 rounding boundary (one
    part in 256 of that activation).  With the reference's initialisation such flips die out from
    layer to layer; with variance-preserving weights (outputs that move with the inputs) they
    persist, so those are checked on shallow networks, where a layer's arithmetic shows directly."""
    w = workloads.init_mlp_weights(op, seed=17, gain=gain, layers=layers)
    feats, dev = workloads.make_queries(op, 3000, seed=23)
    mu, sigma = workloads.batch_mu_sigma(feats, dev)
    h = batched.MLPHandle(feats.shape[1], mu=mu, sigma=sigma, device_features=DEVF, **w)
    got = h.predict(torch.from_numpy(feats).cuda(), torch.from_numpy(dev).cuda()).cpu().numpy()
    h.check_status()
    h.close()
    replay = omlp.forward_bf16(w, omlp.normalise(feats, dev, DEVF, mu, sigma))
    ref64 = omlp.predict(w, feats, dev, DEVF, mu, sigma, np.float64)
    scale = np.abs(ref64).max()
    diff = np.abs(got - replay).max() / scale
    print("%s gain %.2f, %d layers: device vs bf16 replay %.3g of the output scale; replay vs float64 %.3g"
          % (op, gain, layers, diff, np.abs(replay - ref64).max() / scale))
    assert diff <= bound


@pytest.mark.parametrize("precision", ["bf16", "bf16x3"])
def test_small_batches(precision):
    """Batches of up to 4,224 (split: 2,112) queries run on clusters of blocks that exchange their activations; the
    shapes change at 42, 224, 448, 560, 672, 960, 1,440 and 1,920 (split: 14 and half of the others).  Sizes on both
    sides of every change: each prediction equals, to the last bit, the one the same query gets in a full round
    of the two-SM kernel, and that round is within the mode's tolerance of the oracle
    (bf16 on variance-preserving weights: 2e-2 of the output scale, as in the input-sensitive test)."""
    n = 9472 if precision == "bf16" else 4736
    w = workloads.init_mlp_weights("conv2d", seed=9, gain=2.0)
    feats, dev = workloads.make_queries("conv2d", n, 41)
    mu, sigma = workloads.batch_mu_sigma(feats, dev)
    h = batched.MLPHandle(feats.shape[1], mu=mu, sigma=sigma, device_features=DEVF, precision=precision, **w)
    f, r = torch.from_numpy(feats).cuda(), torch.from_numpy(dev).cuda()
    full = h.predict(f, r)
    ref = omlp.predict(w, feats, dev, DEVF, mu, sigma, np.float64)
    err = np.abs(full.cpu().numpy() - ref).max() / np.abs(ref).max()
    assert err <= (2e-2 if precision == "bf16" else 1e-4), err
    edges = [42, 224, 448, 560, 672, 960, 1440, 1920, 4224]
    if precision == "bf16x3":
        edges = [14] + [e // 2 for e in edges[1:]]
    for Q in [1, 2, 15, 16, 17, 33] + [e + d for e in edges for d in (0, 1)]:
        lo = n - Q if Q % 2 else 7
        for _ in range(2):
            got = h.predict(f[lo:lo + Q].contiguous(), r[lo:lo + Q].contiguous())
            assert torch.equal(got, full[lo:lo + Q]), Q
    h.check_status()
    h.close()


@pytest.mark.parametrize("precision", ["bf16", "bf16x3"])
@pytest.mark.parametrize("layers", [1, 2, 3, 8])
def test_few_queries(precision, layers):
    """Up to 42 queries (split: 14) run on at most seven groups of up to six (two), which exchange their activations
    through distributed shared memory, two buffers in turn: odd and even numbers of layers, every size up to the first
    ones that run otherwise, each prediction with the bits it has in a full round of the two-SM kernel."""
    w = workloads.init_mlp_weights("lstm", seed=29, gain=2.0, layers=layers)
    feats, dev = workloads.make_queries("lstm", 9472 if precision == "bf16" else 4736, 47)
    mu, sigma = workloads.batch_mu_sigma(feats, dev)
    h = batched.MLPHandle(feats.shape[1], mu=mu, sigma=sigma, device_features=DEVF, precision=precision, **w)
    f, r = torch.from_numpy(feats).cuda(), torch.from_numpy(dev).cuda()
    full = h.predict(f, r)
    for Q in range(1, 45):
        lo = 61 * Q
        got = h.predict(f[lo:lo + Q].contiguous(), r[lo:lo + Q].contiguous())
        assert torch.equal(got, full[lo:lo + Q]), Q
    h.check_status()
    h.close()


def test_small_batches_on_streams_and_in_a_graph():
    """Small batches keep scratch per stream: interleaved launches of two predictors on more streams than
    there is scratch for, a captured launch, and a launch after an error status all give the same bits."""
    from habitat_b200 import _native
    feats, dev = workloads.make_queries("linear", 500, 43)
    mu, sigma = workloads.batch_mu_sigma(feats, dev)
    f, r = torch.from_numpy(feats).cuda(), torch.from_numpy(dev).cuda()
    hs = [batched.MLPHandle(4, mu=mu, sigma=sigma, device_features=DEVF, **workloads.init_mlp_weights(
        "linear", seed=s, layers=layers, gain=2.0)) for s, layers in ((1, 8), (2, 3))]
    want = [h.predict(f, r).clone() for h in hs]
    torch.cuda.synchronize()
    outs = []
    streams = [torch.cuda.Stream() for _ in range(20)]
    for i in range(60):
        with torch.cuda.stream(streams[i % 20]):
            outs.append((i % 2, hs[i % 2].predict(f, r)))
    torch.cuda.synchronize()
    for k, out in outs:
        assert torch.equal(out, want[k])
    g = torch.cuda.CUDAGraph()
    out = torch.empty_like(want[0])
    with torch.cuda.graph(g):
        hs[0].predict(f, r, out=out)
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, want[0])
    hs[0].inject_status(0x532)
    with pytest.raises(_native.HabitatNativeError):
        hs[0].check_status()
    for k in (0, 1):
        assert torch.equal(hs[k].predict(f, r), want[k])
    for h in hs:
        h.check_status()
        h.close()


@pytest.mark.parametrize("sizes", [[(1, 1), (1, 1), (1, 1), (1, 1)], [(40, 6), (16, 1)], [(264, 4), (250, 4)],
                                   [(1056, 1), (4, 4)], [(352, 6), (1, 1)], [(53, 6), (1, 6), (0, 6), (32, 6)],
                                   [(2112, 1), (2112, 1)], [(2113, 1), (300, 6), (7, 2)], [(9472, 1), (2500, 4), (9, 3)],
                                   [(4224, 1), (2112, 1)], [(4225, 1), (2113, 1), (7, 2)], [(1408, 3), (37, 6), (64, 1), (3, 2)]])
def test_batches_side_by_side(sizes):
    """Batches of several predictors in one call take other shapes than alone where they then fit on the GPU
    together, or one list of tiles; each prediction has the bits it has alone.  Sizes around full shapes, an
    empty batch, small ones beside one that fills the GPU."""
    import ctypes
    from habitat_b200 import _native
    items, keep, outs, want = (_native.MlpGrid * len(sizes))(), [], [], []
    for i, (n, devices) in enumerate(sizes):
        precision = "bf16x3" if i == 1 else "bf16"
        feats, dev = workloads.make_queries("linear", max(n, 2), 50 + i)
        mu, sigma = workloads.batch_mu_sigma(feats, dev)
        h = batched.MLPHandle(4, mu=mu, sigma=sigma, device_features=DEVF, precision=precision,
                              **workloads.init_mlp_weights("linear", seed=i, layers=3 + i, gain=2.0))
        f = torch.from_numpy(feats[:n]).cuda()
        rows = bytes((5 * i + k) % len(DEVF) for k in range(devices))
        out = torch.full((devices * n,), float("nan"), device="cuda")
        each = torch.tensor(list(rows), dtype=torch.uint8, device="cuda").repeat_interleave(n)
        want.append(h.predict(f.repeat(devices, 1).contiguous(), each) if n else out.clone())
        items[i] = _native.MlpGrid(h._handle.value, f.data_ptr(), n, ctypes.cast(ctypes.c_char_p(rows), ctypes.c_void_p),
                                   devices, out.data_ptr())
        keep.append((h, f, rows))
        outs.append(out)
    for _ in range(3):
        _native.check(_native.load().hb_mlp_predict_grid(items, len(sizes), torch.cuda.current_stream().cuda_stream))
        for k, (got, ref) in enumerate(zip(outs, want)):
            assert torch.equal(got, ref), k
            got.fill_(float("nan"))
    for h, _, _ in keep:
        h.check_status()
        h.close()


@pytest.mark.parametrize("precision,sizes,listed", [("bf16", (662, 326, 97), True), ("bf16", (53, 32), False), ("bf16", (485, 527), True),
                                                    ("bf16x3", (83, 114, 275, 82), True), ("bf16x3", (9, 38, 33), False)])
def test_batches_that_would_follow_one_another(precision, sizes, listed):
    """Batches for six devices that each take most of the GPU on the small-batch kernels go to the two-SM kernel as one list of
    tiles, which leaves its cycle counters with the first predictor; others run side by side.  The predictions are the same."""
    import ctypes
    from habitat_b200 import _native
    items, keep, want = (_native.MlpGrid * len(sizes))(), [], []
    rows = bytes(range(6))
    for i, n in enumerate(sizes):
        feats, dev = workloads.make_queries("bmm", n, 80 + i)
        mu, sigma = workloads.batch_mu_sigma(feats, dev)
        h = batched.MLPHandle(4, mu=mu, sigma=sigma, device_features=DEVF, precision=precision,
                              **workloads.init_mlp_weights("bmm", seed=i, layers=3, gain=2.0))
        f, out = torch.from_numpy(feats).cuda(), torch.full((6 * n,), float("nan"), device="cuda")
        each = torch.tensor(list(rows), dtype=torch.uint8, device="cuda").repeat_interleave(n)
        want.append(h.predict(f.repeat(6, 1).contiguous(), each))
        items[i] = _native.MlpGrid(h._handle.value, f.data_ptr(), n, ctypes.cast(ctypes.c_char_p(rows), ctypes.c_void_p), 6,
                                   out.data_ptr())
        keep.append((h, f, out))
    _native.check(_native.load().hb_mlp_predict_grid(items, len(sizes), torch.cuda.current_stream().cuda_stream))
    first = keep[max(range(len(sizes)), key=sizes.__getitem__)][0]
    assert (first.phase_cycles()["slots"] > 0) == listed
    for (h, _, out), ref in zip(keep, want):
        assert torch.equal(out, ref)
        h.check_status()
        h.close()


@pytest.mark.parametrize("precision,round_q,most", [("bf16", 9472, 4224), ("bf16x3", 4736, 2112)])
def test_last_round_of_few_tiles(precision, round_q, most):
    """Queries beyond full rounds of the two-SM kernel (74 tiles) go to the kernel for small batches while they fit
    there: on both sides of that and of where the shapes change, one or two rounds, alone and as a grid with a second batch
    in the list, each prediction has the bits it has in full rounds."""
    import ctypes
    from habitat_b200 import _native
    n = 2 * round_q + 301
    feats, dev = workloads.make_queries("bmm", n, 61)
    mu, sigma = workloads.batch_mu_sigma(feats, dev)
    h = batched.MLPHandle(4, mu=mu, sigma=sigma, device_features=DEVF, precision=precision,
                          **workloads.init_mlp_weights("bmm", seed=7, layers=3, gain=2.0))
    f, r = torch.from_numpy(feats).cuda(), torch.from_numpy(dev).cuda()
    want = h.predict(f[:2 * round_q], r[:2 * round_q])
    want = torch.cat([want, h.predict(f[n - round_q:].contiguous(), r[n - round_q:].contiguous())[round_q - 301:]])
    shapes = [parts * columns * clusters for parts in (2 if precision == "bf16" else 1,) for columns, clusters in PAIR_SHAPES]
    assert shapes[-1] == most
    for q in [round_q, round_q + 1, 2 * round_q, n] + [round_q + e + d for e in shapes for d in (0, 1)]:
        for _ in range(2):
            assert torch.equal(h.predict(f[:q].contiguous(), r[:q].contiguous()), want[:q]), q
    # seven devices x m rows: the cut falls inside a device's rows; the second batch keeps its place in the list
    m, small = (round_q + 900) // 7, (round_q // 4) // 3
    rows = [bytes(range(6)) + b"\x02", b"\x01\x04\x03"]
    items, outs = (_native.MlpGrid * 2)(), []
    for i, k in enumerate((m, small)):
        outs.append(torch.full((len(rows[i]) * k,), float("nan"), device="cuda"))
        items[i] = _native.MlpGrid(h._handle.value, f.data_ptr(), k, ctypes.cast(ctypes.c_char_p(rows[i]), ctypes.c_void_p),
                                   len(rows[i]), outs[i].data_ptr())
    _native.check(_native.load().hb_mlp_predict_grid(items, 2, torch.cuda.current_stream().cuda_stream))
    for k, out, devices in zip((m, small), outs, rows):
        for b, d in enumerate(devices):
            one = torch.full((k,), d, dtype=torch.uint8, device="cuda")
            assert torch.equal(out[b * k:(b + 1) * k], h.predict(f[:k].contiguous(), one)), (k, b)
    h.check_status()
    h.close()


@pytest.mark.parametrize("precision", ["bf16", "bf16x3"])
@pytest.mark.parametrize("op", ["conv2d", "bmm"])
def test_few_host_queries(op, precision):
    """Up to 16 queries from host memory travel as kernel parameters, to as many groups as there are (up to seven): every
    count on both sides of that, each query different, has the bits of the device entry point."""
    feats, dev = workloads.make_queries(op, 64, 71)
    mu, sigma = workloads.batch_mu_sigma(feats, dev)
    h = batched.MLPHandle(feats.shape[1], mu=mu, sigma=sigma, device_features=DEVF, precision=precision,
                          **workloads.init_mlp_weights(op, seed=3, layers=3, gain=2.0))
    want = h.predict(torch.from_numpy(feats).cuda(), torch.from_numpy(dev).cuda()).cpu().numpy()
    assert len(set(want.tolist())) > 48
    for Q in range(1, 18):
        lo = 3 * Q
        if lo + Q > 64:
            lo = 64 - Q
        assert np.array_equal(h.predict_host(feats[lo:lo + Q], dev[lo:lo + Q]), want[lo:lo + Q]), Q
    for q in (0, 9, 63):
        assert h.predict_one(feats[q].tolist(), int(dev[q])) == want[q]
    h.close()


def test_two_threads_with_batches_side_by_side_on_one_stream():
    """Calls of two threads on one stream, each with launches that run side by side or with a last round of its own:
    the launches of a call stay together, so that every call has the bits it has alone."""
    import ctypes
    import threading
    from habitat_b200 import _native
    lib, stream = _native.load(), torch.cuda.current_stream().cuda_stream
    n, devices = (53, 32, 9), 6
    feats, dev = workloads.make_queries("bmm", 9900, 81)
    mu, sigma = workloads.batch_mu_sigma(feats, dev)
    hs = [batched.MLPHandle(4, mu=mu, sigma=sigma, device_features=DEVF, **workloads.init_mlp_weights(
        "bmm", seed=s, layers=4, gain=2.0)) for s in range(3)]
    f, r = torch.from_numpy(feats).cuda(), torch.from_numpy(dev).cuda()
    rows = bytes(range(devices))
    calls = 60
    outs = [[[torch.full((devices * k,), float("nan"), device="cuda") for k in n] for _ in range(calls)] for _ in range(2)]
    tails = [[torch.full((9900,), float("nan"), device="cuda") for _ in range(calls // 10)] for _ in range(2)]
    errors = []

    def grid(mine):
        items = (_native.MlpGrid * 3)()
        for i in range(3):
            items[i] = _native.MlpGrid(hs[i]._handle.value, f.data_ptr(), n[i],
                                       ctypes.cast(ctypes.c_char_p(rows), ctypes.c_void_p), devices, mine[i].data_ptr())
        return lib.hb_mlp_predict_grid(items, 3, stream)

    def work(t):
        for c in range(calls):
            errors.append(grid(outs[t][c]))
            if c % 10 == t:
                errors.append(lib.hb_mlp_predict(hs[t]._handle, ctypes.c_void_p(f.data_ptr()), ctypes.c_void_p(r.data_ptr()),
                                                 9900, ctypes.c_void_p(tails[t][c // 10].data_ptr()), stream))
    torch.cuda.synchronize()
    threads = [threading.Thread(target=work, args=(t,)) for t in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not any(errors)
    for i in range(3):
        each = torch.arange(devices, device="cuda").to(torch.uint8).repeat_interleave(n[i])
        want = hs[i].predict(f[:n[i]].repeat(devices, 1).contiguous(), each)
        for t in range(2):
            for c in range(calls):
                assert torch.equal(outs[t][c][i], want), (t, c, i)
    for t in range(2):
        want = hs[t].predict(f, r)
        for out in tails[t]:
            assert torch.equal(out, want), t
    for h in hs:
        h.check_status()
        h.close()


def test_given_result_has_to_cover_the_queries():
    feats, dev = workloads.make_queries("bmm", 100, 91)
    mu, sigma = workloads.batch_mu_sigma(feats, dev)
    h = batched.MLPHandle(4, mu=mu, sigma=sigma, device_features=DEVF, **workloads.torch_init_mlp_weights("bmm", layers=2))
    f, r = torch.from_numpy(feats).cuda(), torch.from_numpy(dev).cuda()
    want = h.predict(f, r)
    for out in (torch.empty(99, device="cuda"), torch.empty(100), torch.empty(100, dtype=torch.float64, device="cuda"),
                torch.empty(200, device="cuda")[::2]):
        with pytest.raises((ValueError, TypeError)):
            h.predict(f, r, out=out)
    for out in (torch.empty(120, device="cuda"), torch.empty(100).pin_memory()):
        h.predict(f, r, out=out)
        torch.cuda.synchronize()
        assert torch.equal(out[:100].cpu(), want.cpu())
    h.close()


def test_small_batches_on_ever_new_streams():
    """A program with a stream per request keeps the kernel for small batches (the two-SM kernel would leave its cycle
    counters) and its bits: 64 streams one after the other, some with three predictors side by side, then all of
    them at once."""
    import ctypes
    from habitat_b200 import _native
    feats, dev = workloads.make_queries("linear", 300, 95)
    mu, sigma = workloads.batch_mu_sigma(feats, dev)
    f, r = torch.from_numpy(feats).cuda(), torch.from_numpy(dev).cuda()
    hs = [batched.MLPHandle(4, mu=mu, sigma=sigma, device_features=DEVF, **workloads.init_mlp_weights(
        "linear", seed=s, layers=3, gain=2.0)) for s in range(3)]
    want = [h.predict(f, r) for h in hs]
    n, rows = 40, bytes([1, 4, 2])
    each = torch.tensor(list(rows), dtype=torch.uint8, device="cuda").repeat_interleave(n)
    want_grid = [h.predict(f[:n].repeat(3, 1).contiguous(), each) for h in hs]
    outs = [torch.empty((3 * n,), device="cuda") for _ in hs]
    items = (_native.MlpGrid * 3)(*[
        _native.MlpGrid(h._handle.value, f.data_ptr(), n, ctypes.cast(ctypes.c_char_p(rows), ctypes.c_void_p), 3,
                        out.data_ptr()) for h, out in zip(hs, outs)])
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream(priority=-(i % 2)) for i in range(64)]
    assert len({s.cuda_stream for s in streams}) > 40
    for turn in range(2):
        for i, s in enumerate(streams):
            with torch.cuda.stream(s):
                if i % 3 == turn:
                    for out in outs:
                        out.fill_(float("nan"))
                    _native.check(_native.load().hb_mlp_predict_grid(items, 3, s.cuda_stream))
                got = hs[i % 2].predict(f, r)
            s.synchronize()
            assert torch.equal(got, want[i % 2])
            if i % 3 == turn:
                for out, ref in zip(outs, want_grid):
                    assert torch.equal(out, ref)
    assert [h.phase_cycles()["slots"] for h in hs] == [0, 0, 0]
    results = []
    for i in range(256):
        with torch.cuda.stream(streams[i % 64]):
            results.append(hs[i % 3].predict(f, r))
    torch.cuda.synchronize()
    for i, got in enumerate(results):
        assert torch.equal(got, want[i % 3]), i
    for h in hs:
        h.check_status()
        h.close()


def test_cycle_counters():
    """The counters of the two-SM kernel's first cluster: slots and copies of whole tiles, a first copy of plausible
    length, and the issuer's waits within its whole loop."""
    w = workloads.init_mlp_weights("bmm", seed=2, layers=3, gain=2.0)
    feats, dev = workloads.make_queries("bmm", 74 * 128 * 2, 9)
    mu, sigma = workloads.batch_mu_sigma(feats, dev)
    for precision, parts in (("bf16", 1), ("bf16x3", 2)):
        h = batched.MLPHandle(4, mu=mu, sigma=sigma, device_features=DEVF, precision=precision, **w)
        Q = len(feats) // parts                                  # two rounds of tiles
        h.predict(torch.from_numpy(feats[:Q]).cuda(), torch.from_numpy(dev[:Q]).cuda())
        h.check_status()
        c = h.phase_cycles()
        slots = 2 * 3 * 64 * parts                               # (fc1's four are not counted)
        assert c["slots"] == slots
        assert 0 <= c["copies"] - (slots + 2 * 4) / 3 < 1        # one producer of three
        assert 300 < c["producer_copy"] < c["mma_total_cycles"] / 4
        assert 0 < c["mma_wait_act"] + c["mma_wait_weights"] + c["mma_wait_tmem"] < c["mma_total_cycles"]
        h.close()


def test_small_batches_switched_off():
    """HB_MLP_WIDE=0 keeps every batch on the two-SM kernel, which leaves its cycle counters; without it small batches
    from host memory leave none.  The predictions are the same."""
    import os
    import subprocess
    import sys
    code = """
import os
import numpy as np, torch
from habitat_b200 import batched, workloads
feats, dev = workloads.make_queries("bmm", 300, 97)
mu, sigma = workloads.batch_mu_sigma(feats, dev)
w = workloads.init_mlp_weights("bmm", seed=2, layers=2, gain=2.0)
want = None
for Q in (300, 17, 16, 1):
    h = batched.MLPHandle(4, mu=mu, sigma=sigma, device_features=workloads.BENCH_DEVICE_FEATURES, **w)
    got = h.predict_host(feats[:Q], dev[:Q])
    want = got if want is None else want
    assert np.array_equal(got, want[:Q]), Q
    assert (h.phase_cycles()["slots"] > 0) == ("HB_MLP_WIDE" in os.environ), Q
    h.close()
print(want.tobytes().hex()[:200])
"""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    outs = []
    for env in (dict(os.environ), dict(os.environ, HB_MLP_WIDE="0")):
        r = subprocess.run([sys.executable, "-c", code], env=env, capture_output=True, text=True, timeout=300, cwd=root)
        assert r.returncode == 0, r.stderr
        outs.append(r.stdout)
    assert outs[0] == outs[1]


def test_scratch_of_a_stream_grows_with_the_shapes_it_uses():
    """What a stream's small batches keep of the GPU's memory: 2.2 MB of sums from the first one on, and each shape's activations
    (0.9 to 17 MB) from its first batch on; both are given back with the last predictor.  Bounds: those sizes, and the 2 MB
    that memory is handed out in.  A stream that has had all shapes before leaves what loading the kernels takes out of
    the count."""
    import os
    import subprocess
    import sys
    code = """
import torch
from habitat_b200 import batched, workloads
feats, dev = workloads.make_queries("bmm", 4224, 97)
mu, sigma = workloads.batch_mu_sigma(feats, dev)
w = workloads.init_mlp_weights("bmm", seed=2, layers=2, gain=2.0)
def handle():
    return batched.MLPHandle(4, mu=mu, sigma=sigma, device_features=workloads.BENCH_DEVICE_FEATURES, **w)
h = handle()
f, r, out = torch.from_numpy(feats).cuda(), torch.from_numpy(dev).cuda(), torch.empty(4224, device="cuda")
sizes = (1, 224, 448, 560, 672, 960, 1440, 1920, 4224)
streams = [torch.cuda.Stream() for _ in range(2)]
def run(Q, s):
    with torch.cuda.stream(s):
        h.predict(f[:Q], r[:Q], out=out[:Q])
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]
for Q in sizes:
    free = run(Q, streams[0])
mb = 1 << 20
took = []
for Q in sizes:
    now = run(Q, streams[1])
    took.append((free - now) / mb)
    free = now
    assert run(Q, streams[1]) == now, Q
print(took)
need = [2.2] + [clusters * 8192 * columns / mb for clusters, columns in
                ((7, 16), (7, 32), (7, 40), (7, 48), (15, 32), (15, 48), (15, 64), (33, 64))]
assert all(t <= n + 2 for t, n in zip(took, need)), (took, need)
h.check_status()
h.close()
h = handle()
assert torch.cuda.mem_get_info()[0] - free > 2 * 40 * mb
h.close()
"""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300, cwd=root)
    print(r.stdout)
    assert r.returncode == 0, r.stderr


# Shapes of the kernel for clusters of SM pairs: columns per CTA, clusters at a time.
PAIR_SHAPES = ((16, 7), (32, 7), (40, 7), (48, 7), (32, 15), (48, 15), (64, 15), (64, 33))


def _clusters(Q, precision):
    """Clusters of SM pairs that a batch alone runs on (0: it runs on another kernel)."""
    parts = 2 if precision == "bf16" else 1
    if Q <= (42 if precision == "bf16" else 14):
        return 0
    for columns, clusters in PAIR_SHAPES:
        if Q <= parts * columns * clusters:
            groups = -(-Q // (parts * columns))
            return -(-Q // -(-Q // groups))
    return 0


@pytest.mark.parametrize("precision,edges", [("bf16", (28, 224, 448, 560, 672, 960, 1440, 1920, 4224)),
                                             ("bf16x3", (14, 112, 224, 280, 336, 480, 720, 960, 2112))])
@pytest.mark.parametrize("layers", [1, 2, 3, 8])
def test_clusters_of_pairs(precision, edges, layers):
    """Each shape of the kernel for clusters of SM pairs at both ends of its range, with groups that are not
    full and halves of different lengths, and the size past the last shape: each prediction has the bits it has in a full
    round of the two-SM kernel's tiles (two buffers alternate by layer, so odd and even numbers of layers).  Once with
    what the blocks exchange taken for stale, so that the network runs a second time, and as usual after that."""
    n = 9472 if precision == "bf16" else 4736
    w = workloads.init_mlp_weights("conv2d", seed=37, gain=2.0, layers=layers)
    feats, dev = workloads.make_queries("conv2d", n, 59)
    mu, sigma = workloads.batch_mu_sigma(feats, dev)
    h = batched.MLPHandle(feats.shape[1], mu=mu, sigma=sigma, device_features=DEVF, precision=precision, **w)
    f, r = torch.from_numpy(feats).cuda(), torch.from_numpy(dev).cuda()
    full = h.predict(f, r)
    for e in edges:
        for Q in (e, e + 1, e - 1, e - 13):
            lo = (17 * Q) % (n - Q)
            for turn in range(4):
                runs = h.second_runs()
                if turn == 1 and _clusters(Q, precision):
                    h.inject_stale()
                got = h.predict(f[lo:lo + Q].contiguous(), r[lo:lo + Q].contiguous())
                assert torch.equal(got, full[lo:lo + Q]), (Q, turn)
                assert turn != 1 or h.second_runs() - runs == _clusters(Q, precision), Q
    h.check_status()
    h.close()


def test_every_word_of_an_exchange_is_looked_at():
    """In the library built with -DHB_BOUNDS_CHECK (a process of its own): one word with the wrong signs in the output of one
    layer, in each cluster.  Whichever K quarter, row block, half of the queries or layer it is in, every cluster runs the
    network once more and the predictions are the usual ones."""
    import os
    import subprocess
    import sys
    from habitat_b200 import build as hb_build
    if not os.path.exists(hb_build.CHECKED_LIB_PATH):
        pytest.fail("libhabitat_b200_checked.so is not built (python -m habitat_b200.build --checked)")
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", "from tests.test_mlp_gpu import _plant_words as t\nt('bf16')\nt('bf16x3')"],
                       env=dict(os.environ, HABITAT_B200_LIB=hb_build.CHECKED_LIB_PATH), capture_output=True, text=True,
                       timeout=300, cwd=root)
    assert r.returncode == 0, r.stderr
    h = batched.MLPHandle(4, mu=np.zeros(8), sigma=np.ones(8), device_features=DEVF,
                          **workloads.init_mlp_weights("bmm", seed=41, layers=1))
    with pytest.raises(_native_error(), match="HB_BOUNDS_CHECK"):
        h.inject_stale(0, 0, 0)
    h.close()


def _plant_words(precision):
    """All words of a row, every group of eight rows, the rows at the edges of what the warps share out, and random ones, in full
    batches of each shape."""
    layers = 3
    w = workloads.init_mlp_weights("bmm", seed=41, gain=2.0, layers=layers)
    feats, dev = workloads.make_queries("bmm", 4224, 67)
    mu, sigma = workloads.batch_mu_sigma(feats, dev)
    h = batched.MLPHandle(4, mu=mu, sigma=sigma, device_features=DEVF, precision=precision, **w)
    for columns, clusters in PAIR_SHAPES:
        Q = clusters * columns * (2 if precision == "bf16" else 1)
        f, r, out = torch.from_numpy(feats[:Q]).cuda(), torch.from_numpy(dev[:Q]).cuda(), torch.empty(Q, device="cuda")
        want = h.predict(f, r).clone()
        assert _clusters(Q, precision) == clusters
        g = np.random.default_rng(columns + clusters)
        places = [(k % layers, 331 * k % 1024, k) for k in range(columns)]
        places += [(k % layers, 8 * k + k % 8, int(g.integers(columns))) for k in range(128)]
        places += [(L, k, word) for L in range(layers) for k in (0, 127, 128, 255, 256, 511, 512, 639, 640, 767, 768, 1023)
                   for word in (0, columns - 1)]
        places += [(int(g.integers(layers)), int(g.integers(1024)), int(g.integers(columns))) for _ in range(100)]
        runs = h.second_runs()
        for place in places:
            h.inject_stale(*place)
            out.fill_(float("nan"))
            h.predict(f, r, out=out)
            now = h.second_runs()
            # (a word that really was stale: one launch in 40,000, and only while other streams are at work)
            assert now - runs == clusters, (columns, clusters, place)
            assert torch.equal(out, want), (columns, clusters, place)
            runs = now
    h.check_status()
    h.close()
