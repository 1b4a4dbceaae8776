"""Units with few replicas (lane packing: the lanes of a warp hold the replicas
several times over and share the points) against the oracle: replica counts
at the edges of the packings, split and not, resident and streamed proteins,
with the MCC score and the trajectory record on; and the same bits under the
persistent schedule and in a run that is resumed."""
import numpy as np
import pytest

from gpudock_b200 import abi, lib, synth
from tests.test_gpu_remc import _replay_checks
from tests.test_gpu_split import FLAGS, _check_records

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = lib.Context(0)
    yield c
    c.close()


def _run(ctx, d, n_tmp, steps=(20, 20), flags=FLAGS):
    _, mb = lib.set_temperature(n_tmp, 0.004, 0.04)
    r = lib.Remc(d, sum(steps), 10, mb, seed=12, flags=flags)
    r.init()
    for n in steps:
        r.run(n)
    return r.read(), mb


# replicas of a unit: 1 .. 4 (8 lane groups), 5 .. 8, 9 .. 16, and units of
# different packings in one run (7 x 8 temperatures: 32 and 24; 9 x 4: 32 and 4)
@pytest.mark.parametrize("n_lig,n_tmp", [(1, 1), (3, 1), (1, 4), (1, 5), (1, 8), (2, 5), (2, 8),
                                         (1, 16), (9, 4), (7, 8)])
@pytest.mark.parametrize("split", [1, 8])
def test_packed_units(ctx, n_lig, n_tmp, split):
    cx = synth.make_complex(synth.ComplexSpec(pnp=1237, lna=19, n_lig=n_lig, n_prt=2), seed=91)
    ctx.set_split(split)
    d = lib.DeviceComplex(ctx, cx)
    out, mb = _run(ctx, d, n_tmp)
    _check_records(cx, out, mb)
    _replay_checks(cx, mb, out.record, 12, 10, n_tmp)
    # one launch of the whole length, and the persistent schedule (unsplit)
    again, _ = _run(ctx, d, n_tmp, steps=(40,))
    assert np.array_equal(out.energy, again.energy)
    assert np.array_equal(out.record, again.record)
    if split == 1:
        ctx.set_schedule(abi.SCHED_PERSISTENT, 3)
        again, _ = _run(ctx, d, n_tmp, steps=(40,))
        ctx.set_schedule(abi.SCHED_AUTO)
        assert np.array_equal(out.energy, again.energy)
    ctx.set_split(0)


def test_packed_streamed(ctx):
    """A protein that streams through the ring, on one CTA."""
    cx = synth.make_complex(synth.ComplexSpec(pnp=9000, lna=50, n_lig=1), seed=92)
    ctx.set_split(1)
    d = lib.DeviceComplex(ctx, cx)
    out, mb = _run(ctx, d, 8, steps=(10,))
    ctx.set_split(0)
    _check_records(cx, out, mb)


@pytest.mark.parametrize("n", [3, 21, 150])
def test_batch_splits(ctx, n):
    """A batch whose complexes get different numbers of CTAs per unit (all
    their own most; the costliest more; one each): recorded states and
    decisions of every complex."""
    raw, _, _ = synth.default_ff()
    prt = synth.make_protein(np.random.Generator(np.random.PCG64(93)),
                             synth.ComplexSpec(pnp=1900, lna=8), 8.0, raw)
    cxs = [synth.make_complex(synth.ComplexSpec(pnp=1900, lna=8 + (i * 88) // n, n_lig=1 + i % 4),
                              seed=94 + i, protein=prt) for i in range(n)]
    _, mb = lib.set_temperature(8, 0.004, 0.04)
    base = lib.DeviceComplex(ctx, cxs[0])
    dcxs = [lib.DeviceComplex(ctx, cx, share=base) for cx in cxs]
    b = lib.Batch(ctx, dcxs, [abi.mc_params(10, 10, mb, seed=12, flags=FLAGS) for _ in cxs])
    b.init()
    b.run(10)
    for i in range(0, n, max(1, n // 12)):
        _check_records(cxs[i], b.read(i), mb, steps=(0,))
    b.close()
