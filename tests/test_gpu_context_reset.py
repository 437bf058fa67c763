"""Calls before and after the device's context was reset (cuDevicePrimaryCtxReset, what
cudaDeviceReset and CUDA.jl's device_reset! do): the device blocks, status slots and
staging buffers that the library keeps between calls go with the context, and the next
call has to take new ones. In a process of its own, whose context it is."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

SCRIPT = """
import ctypes, sys
import numpy as np
import pdot
from pdot import instances

driver = ctypes.CDLL("libcuda.so.1")
params = pdot.default_parameters(1e-9, iteration_limit=200)
small = instances.uniform_sqeuclid(127, 93, seed=1)
large = instances.uniform_sqeuclid(1500, 1501, seed=2)  # 18 MB: staged copies
batch = [instances.uniform_sqeuclid(40 + k, 50, seed=k) for k in range(3)]

def calls():
    outs = [pdot.optimize(params, p) for p in (small, large)] + list(pdot.optimize_batched(params, batch)[0])
    return [np.array(x) for o in outs for x in (o.primal_solution, o.dual_source_solution, o.dual_target_solution)]

want = calls()
for _ in range(2):
    assert driver.cuDevicePrimaryCtxReset_v2(0) == 0
    for a, b in zip(want, calls(), strict=True):
        assert np.array_equal(a, b)
print("same after two resets")
"""


def test_calls_after_a_context_reset(built):
    root = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pdot.jl_b200")
    done = subprocess.run([sys.executable, "-c", SCRIPT], env=dict(os.environ, PYTHONPATH=root), capture_output=True,
                          text=True, timeout=300)
    assert done.returncode == 0, done.stderr[-2000:]
    assert "same after two resets" in done.stdout
