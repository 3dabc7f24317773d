"""Arguments of predict_iteration_totals that do not fit are refused before anything is launched."""
import types

import pytest
import torch

from habitat_b200 import batched, iteration


def _call(bench_devices, width=4, rows=range(6), dims=2):
    zeros = lambda dtype: torch.zeros(10, dtype=dtype)
    kernels = batched.KernelBatch(zeros(torch.int32), zeros(torch.uint16), zeros(torch.uint16), zeros(torch.uint32),
                                  zeros(torch.float32), zeros(torch.float32))
    handle = object.__new__(batched.MLPHandle)
    handle.n_op_features, handle._handle = 4, types.SimpleNamespace(value=0)
    handle.close = lambda: None
    features = torch.zeros((4, width) if dims == 2 else (4,))
    special = {"bmm": iteration.SpecialOps(handle, features, torch.zeros(4), torch.tensor([0, 4]))}
    return iteration.predict_iteration_totals(kernels, torch.zeros(10), torch.tensor([0, 10]), special,
                                              bench_devices[0], bench_devices, 0, rows)


@pytest.mark.parametrize("bad", [dict(width=3), dict(width=8), dict(dims=1), dict(rows=range(4)), dict(rows=[])])
def test_what_does_not_fit_is_refused(bench_devices, bad):
    """Features of another width or too few device rows would have the kernels read past their arrays."""
    with pytest.raises(ValueError):
        _call(bench_devices, **bad)


def test_what_fits_gets_as_far_as_the_tensors(bench_devices):
    with pytest.raises(TypeError, match="CUDA tensor"):
        _call(bench_devices)
