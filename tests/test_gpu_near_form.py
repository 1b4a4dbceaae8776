"""Runs whose points are nearly all within reach of the ligand take them all in
the full form: the same bits as the kernel that sorts them into near and far,
whichever of the two a context's runs get, and the share of far points behind
the choice."""
import numpy as np
import pytest

from gpudock_b200 import abi, lib, synth
from tests.test_gpu_split import FLAGS, _check_records

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lna,pnp", [(9, 33), (37, 400), (70, 129), (96, 700)])
@pytest.mark.parametrize("sched,split", [(abi.SCHED_WAVES, 1), (abi.SCHED_WAVES, 2),
                                         (abi.SCHED_PERSISTENT, 1)])  # (unsplit plans only)
def test_same_bits_as_the_sorting_kernel(lna, pnp, sched, split):
    """A small protein (near kernel) and the same one in a batch beside a large
    share of far points (sorting kernel: the plan's average decides)."""
    ctx = lib.Context(0)
    ctx.set_split(split)
    ctx.set_schedule(sched, 3 if sched == abi.SCHED_PERSISTENT else 0)
    cx = synth.make_complex(synth.ComplexSpec(pnp=pnp, lna=lna, n_lig=4, n_prt=2,
                                              n_psp=32 if pnp >= 100 else 0), seed=106)
    far = synth.make_complex(synth.ComplexSpec(pnp=pnp, lna=lna, n_lig=4, n_prt=2,
                                               n_psp=32 if pnp >= 100 else 0), seed=106)
    far.lig_center = (far.lig_center + np.float32([200.0, 0.0, 0.0])).astype(np.float32)
    far._struct = None
    _, mb = lib.set_temperature(8, 0.004, 0.04)
    d, d_far = lib.DeviceComplex(ctx, cx), lib.DeviceComplex(ctx, far)
    r = lib.Remc(d, 40, 10, mb, seed=12, flags=FLAGS)
    r.init()
    r.run(40)
    alone = r.read()
    _check_records(cx, alone, mb)
    mc = lambda: abi.mc_params(40, 10, mb, seed=12, flags=FLAGS)
    b = lib.Batch(ctx, [d, d_far, d_far], [mc(), mc(), mc()])
    b.init()
    b.run(40)
    beside = b.read(0)
    for name in ("energy", "movematrix", "idx_tmp", "acs_mc", "record"):
        assert np.array_equal(getattr(alone, name), getattr(beside, name)), name
    b.close()
    r.close()
    ctx.set_schedule(abi.SCHED_AUTO)
    ctx.close()
