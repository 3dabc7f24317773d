"""Which arrays wave_scale_host takes: what reaches the library, for which a function of the test stands in."""
import ctypes

import numpy as np
import pytest

from habitat_b200 import _native, batched, device_table, habitat_cuda, workloads

FIELDS = {"num_blocks": np.int32, "block_size": np.uint16, "regs_per_thread": np.uint16, "smem_bytes": np.uint32,
          "run_time_ns": np.float32, "gamma": np.float32}


@pytest.fixture
def library():
    """The records that the stand-in for hb_wave_scale_host has been called with."""
    calls = []

    @ctypes.CFUNCTYPE(ctypes.c_int32, ctypes.POINTER(ctypes.c_void_p), ctypes.c_int64, ctypes.c_int32, ctypes.c_void_p,
                      ctypes.c_int32, ctypes.c_void_p, ctypes.c_void_p)
    def stand_in(kernels, K, origin, dests, D, regs, out):
        calls.append([np.frombuffer(ctypes.string_at(kernels[i], K * np.dtype(t).itemsize), t)
                      for i, t in enumerate(FIELDS.values())])
        return 0

    binding, lib = _native.binding(), _native.load()
    real = {name: ctypes.cast(getattr(lib, name), ctypes.c_void_p).value for name in _native.EXPORTS}
    rest = (device_table.row_of, _native.check, batched.WaveResult, habitat_cuda.DeviceProperties)
    binding.setup(dict(real, hb_wave_scale_host=ctypes.cast(stand_in, ctypes.c_void_p).value), *rest)
    yield calls
    binding.setup(real, *rest)


def test_arrays_that_go_on_behind_the_kernels(bench_devices, library):
    """num_blocks says how many kernels there are; the other arrays have to cover them."""
    made = workloads.make_kernels(100, seed=3)
    kernels = {f: made[f].astype(t) for f, t in FIELDS.items()}
    longer = {f: np.concatenate([a, a[:9]]) if f != "num_blocks" else a for f, a in kernels.items()}
    for arrays in (kernels, longer):
        res = batched.wave_scale_host(arrays, bench_devices[0], bench_devices)
        assert res["scaled_ns"].shape == (6, 100) and res["origin_waves"].shape == (100,)
        for got, f in zip(library.pop(), FIELDS):
            assert np.array_equal(got, kernels[f]), f
    for f in list(FIELDS)[1:]:
        with pytest.raises(ValueError):
            batched.wave_scale_host(dict(kernels, **{f: kernels[f][:-1]}), bench_devices[0], bench_devices)
    assert not library
