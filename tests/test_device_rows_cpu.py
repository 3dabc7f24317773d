"""Rows of the device table that devices carry with them: what the native binding hands to the library."""
import copy
import os
import pickle
import subprocess
import sys

import pytest

from habitat_b200 import device_table
from habitat_b200.habitat_cuda import DeviceProperties

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# Reads pickled devices and prints the rows the library is called with, after `first` devices have been used:
# a function of this script stands in for hb_wave_scale_host.
_CHILD = """
import ctypes, pickle, sys
import numpy as np
from habitat_b200 import _native, batched, device_table, habitat_cuda, workloads
devices = pickle.load(sys.stdin.buffer)
table = device_table.load_device_file()
for name in sys.argv[1].split(","):
    device_table.row_of(table[name])
binding, lib, seen = _native.binding(), _native.load(), []

@ctypes.CFUNCTYPE(ctypes.c_int32, ctypes.c_void_p, ctypes.c_int64, ctypes.c_int32, ctypes.POINTER(ctypes.c_int32),
                  ctypes.c_int32, ctypes.c_void_p, ctypes.c_void_p)
def stand_in(kernels, K, origin, dests, D, regs, out):
    seen.extend([origin] + [dests[d] for d in range(D)])
    return 0

addresses = {name: ctypes.cast(getattr(lib, name), ctypes.c_void_p).value for name in _native.EXPORTS}
addresses["hb_wave_scale_host"] = ctypes.cast(stand_in, ctypes.c_void_p).value
binding.setup(addresses, device_table.row_of, _native.check, batched.WaveResult, habitat_cuda.DeviceProperties)
batched.wave_scale_host(workloads.make_kernels(4, seed=1), devices[0], devices[1:])
for row, device in zip(seen, devices):
    assert device_table._rows[row] == device.spec_tuple(), (device, row)
print(len(seen), "rows")
"""


def _in_fresh_interpreter(blob, first):
    out = subprocess.run([sys.executable, "-c", _CHILD, first], input=blob, capture_output=True, cwd=ROOT)
    assert out.returncode == 0, out.stderr.decode()[-2000:]
    return out.stdout.decode().split()[0]


@pytest.mark.parametrize("legacy", [False, True])
def test_used_devices_in_another_process(device_file, legacy):
    """Devices that have been used keep no row of this process when they go to another one, nor do pickles
    that hold such a row."""
    names = ["V100", "T4", "RTX2080Ti"]
    devices = [copy.copy(device_file[n]) for n in names]
    for d in devices:
        device_table.row_of(d)
    assert all(hasattr(d, "_row_token") for d in devices)
    blob = pickle.dumps(devices)
    if legacy:
        blob = pickle.dumps([_WithRow(d) for d in devices])
    assert _in_fresh_interpreter(blob, "P100,P4000,RTX2070,T4") == "3"


class _WithRow:
    """Pickles as the device did when its row was part of its state."""

    def __init__(self, device):
        self.device = device

    def __reduce__(self):
        state = {"_name": self.device.name, "_fields": dict(self.device._fields), "_row_token": 64 + 1}
        return DeviceProperties.__new__, (DeviceProperties,), state


def test_copies_and_other_classes_are_looked_up(device_file):
    """A copy starts without a row, and an object of another class is asked for its values each time."""
    device = device_file["T4"]
    device_table.row_of(device)
    for other in (copy.copy(device), copy.deepcopy(device), pickle.loads(pickle.dumps(device))):
        assert not hasattr(other, "_row_token")
        assert other.spec_tuple() == device.spec_tuple() and other.name == device.name
        assert device_table.row_of(other) == device_table.row_of(device)
    with pytest.raises(TypeError):
        device._fields["num_sms"] = 1

    class Changing(DeviceProperties):
        def spec_tuple(self):
            return self.spec

    changing = Changing("x", **device._fields)
    for name in ("T4", "V100"):
        changing.spec = device_file[name].spec_tuple()
        assert device_table.row_of(changing) == device_table.row_of(device_file[name])
        assert not hasattr(changing, "_row_token")

    class Elsewhere(DeviceProperties):
        def __init__(self, spec):
            self._name, self.spec = "y", spec

        def spec_tuple(self):
            return self.spec

    kept = copy.deepcopy(Elsewhere(device.spec_tuple()))
    assert kept.spec_tuple() == device.spec_tuple() and device_table.row_of(kept) == device_table.row_of(device)
