"""Contexts that come and go on the GPU: released in another order than they
were created, more of them than share a pinned block, and one that is created
after a device reset while an older handle was never destroyed (in a process of
its own; cudaDeviceReset ends that process's own CUDA context only)."""
import os
import subprocess
import sys

import numpy as np
import pytest

from gpudock_b200 import lib, synth

pytestmark = pytest.mark.gpu


def test_mixed_order():
    cx = synth.make_complex(synth.ComplexSpec(pnp=900, lna=20), seed=99)
    poses = synth.random_poses(np.random.default_rng(1), 40, box=3.0)
    large = synth.random_poses(np.random.default_rng(2), 8000, box=3.0)

    def run(ctx):
        d = lib.DeviceComplex(ctx, cx)
        out = d.energy_poses(poses)[0], d.energy_poses(large)[0]
        d.close()
        return out

    ctxs = [lib.Context(0) for _ in range(6)]
    want = run(ctxs[0])

    def check(ctx):
        for a, b in zip(run(ctx), want):
            assert np.array_equal(a, b)

    for c in ctxs:
        check(c)
    for k in (4, 0, 1):
        ctxs[k].close()
        check(ctxs[5])
    for k in (1, 4):
        ctxs[k] = lib.Context(0)
        check(ctxs[k])
    for k in (2, 5, 1, 3, 4):
        check(ctxs[k])
        ctxs[k].close()
    last = lib.Context(0)
    check(last)
    last.close()


AFTER_RESET = """
import os, sys
import numpy as np
from cuda.bindings import runtime as rt
from gpudock_b200 import lib, synth
cx = synth.make_complex(synth.ComplexSpec(pnp=900, lna=20), seed=99)
poses = synth.random_poses(np.random.default_rng(1), 40, box=3.0)
old = lib.Context(0)
want = lib.DeviceComplex(old, cx).energy_poses(poses)[0]
assert rt.cudaDeviceReset()[0] == rt.cudaError_t.cudaSuccess
new = [lib.Context(0) for _ in range(5)]
for c in new:
    d = lib.DeviceComplex(c, cx)
    assert np.array_equal(d.energy_poses(poses)[0], want)
    d.close()
    c.close()
print("equal", flush=True)
os._exit(0)  # the old handles are never destroyed
"""


def test_context_after_device_reset():
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    res = subprocess.run([sys.executable, "-c", AFTER_RESET], cwd=root, capture_output=True,
                         text=True, timeout=300)
    assert res.returncode == 0 and "equal" in res.stdout, res.stderr
