"""Copies of a state's bodies to host memory (nbGetBodiesCUDA): both sides of the 4 MB from which
pageable memory is reached through page-locked slots, a last slot filled to any part, every kind of
memory side by side, and a device pointer given by mistake, which is the driver's to answer at any
size."""
import subprocess
import sys

import numpy as np
import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

LINE = -(-(4 << 20) // 24)              # the fewest bodies whose positions take 4 MB
SLOT = (1 << 20) / 24.0                 # bodies a slot


def _state(n):
    from milkywayathome_client_b200 import NBodyState
    rng = np.random.default_rng(n)
    pos, vel = rng.standard_normal((n, 3)), rng.standard_normal((n, 3))
    st = NBodyState(n, 0)
    st.set_bodies(pos, vel, np.ones(n), 4.0)
    return st, pos, vel


@pytest.mark.parametrize("n", [LINE - 1, LINE, LINE + 1, int(5 * SLOT), int(8 * SLOT) + 1,
                               int(9 * SLOT), int(16.5 * SLOT), int(24 * SLOT) + 2])
def test_pageable_memory(n):
    st, pos, vel = _state(n)
    with st:
        for _ in range(2):              # the slots are made, then used again
            x, v = st.bodies()
            assert np.array_equal(x, pos) and np.array_equal(v, vel)


@pytest.mark.parametrize("n", [LINE - 1, LINE + 1])
def test_page_locked_and_managed_memory_beside_pageable(n):
    import torch
    runtime = pytest.importorskip("cuda.bindings.runtime")
    import ctypes
    st, pos, vel = _state(n)
    with st:
        pinned = torch.empty((n, 3), dtype=torch.float64, pin_memory=True).numpy()
        err, ptr = runtime.cudaMallocManaged(24 * n, 1)
        assert int(err) == 0
        managed = np.ctypeslib.as_array((ctypes.c_double * (3 * n)).from_address(int(ptr)))
        managed = managed.reshape(n, 3)
        for a, b in ((pinned, np.empty((n, 3))), (np.empty((n, 3)), pinned),
                     (managed, np.empty((n, 3))), (pinned, managed)):
            a[:] = b[:] = 0.0
            st.bodies(out=(a, b))
            assert np.array_equal(a, pos) and np.array_equal(b, vel)
        del managed, a, b
        assert int(runtime.cudaFree(ptr)[0]) == 0


DEVICE_POINTER = r'''
import sys
import torch
from milkywayathome_client_b200 import NBodyState
import numpy as np
status = []
for n in (%d, %d):
    st = NBodyState(n, 0)
    st.set_bodies(np.ones((n, 3)), np.ones((n, 3)), np.ones(n), 4.0)
    out = torch.zeros((n, 3), dtype=torch.float64, device="cuda:0")
    torch.cuda.synchronize()
    status.append(st.lib.nbGetBodiesCUDA(st._h, out.data_ptr(), None))
print("statuses", *status)
'''


def test_a_device_pointer_gets_a_status_at_any_size():
    """In a process of its own, for a host write to a device address would end it.  The buffer is
    as large as the copy, so nothing is out of range either way."""
    r = subprocess.run([sys.executable, "-c", DEVICE_POINTER % (LINE - 1, LINE + 1)], cwd=ROOT,
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    below, above = r.stdout.split("statuses")[1].split()
    assert below == above
