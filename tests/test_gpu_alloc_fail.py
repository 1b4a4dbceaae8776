"""Device allocations that fail at each place that makes one
(gd_ctx_set_alloc_fail): an upload gives back the memory it had taken; a pose
call and a similarity matrix return GD_ENOMEM for what they cannot do without,
and the same results without what they can; the hook is used up each time."""
import numpy as np
import pytest

from gpudock_b200 import abi, lib, synth
from oracle import oracle as orc
from tests import tolerance as tol
from tests.test_gpu_resilience import _pool_used

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = lib.Context(0)
    yield c
    c.close()


def _high(reset=False):
    from cuda.bindings import runtime as rt
    err, pool = rt.cudaDeviceGetDefaultMemPool(0)
    attr = rt.cudaMemPoolAttr.cudaMemPoolAttrUsedMemHigh
    if reset:
        from cuda.bindings import driver
        rt.cudaMemPoolSetAttribute(pool, attr, driver.cuuint64_t(0))
    return int(rt.cudaMemPoolGetAttribute(pool, attr)[1])


def _used_up(ctx, cx):
    lib.DeviceComplex(ctx, cx).close()


def test_upload_gives_back_what_it_took(ctx):
    cx = synth.make_complex(synth.ComplexSpec(pnp=900, lna=24), seed=101)
    used = _pool_used()
    for nth in (1, 2, 9, 15):
        _high(reset=True)
        ctx.set_alloc_fail(nth)
        with pytest.raises(lib.GdError) as exc:
            lib.DeviceComplex(ctx, cx)
        assert exc.value.status == abi.GD_ENOMEM and "injected" in str(exc.value)
        assert _pool_used() == used
        assert (_high() > used) == (nth > 1)  # it had taken memory
    _used_up(ctx, cx)


@pytest.mark.parametrize("n", [2500, 20000])  # cells in one launch, in four
def test_pose_workspace(ctx, n):
    cx = synth.make_complex(synth.ComplexSpec(pnp=2500, lna=50), seed=95)
    poses = synth.random_poses(np.random.default_rng(n), n, box=6.0)
    d = lib.DeviceComplex(ctx, cx)
    ctx.set_alloc_fail(1)  # the poses and results
    with pytest.raises(lib.GdError) as exc:
        d.energy_poses(poses)
    assert exc.value.status == abi.GD_ENOMEM
    ctx.set_alloc_fail(2)  # the cells: one launch without them
    n0 = ctx.launches
    terms, raw = d.energy_poses(poses)
    assert ctx.launches == n0 + 1
    _used_up(ctx, cx)
    terms_r, raw_r, asum = orc.energy_poses(cx, poses[:100])
    bad, rel = tol.check_raw(raw[:100], raw_r, asum)
    assert not bad.any(), np.nanmax(rel, axis=0)
    bad, rel = tol.check_terms(terms[:100], terms_r, raw_r, asum, cx.ff)
    assert not bad.any(), np.nanmax(rel, axis=0)
    n0 = ctx.launches
    d.energy_poses(poses)
    assert ctx.launches > n0 + 1
    d.close()


def test_similarity_workspace(ctx):
    cx = synth.make_complex(synth.ComplexSpec(pnp=900, lna=24, n_lig=2), seed=103)
    rng = np.random.default_rng(3)
    confs = np.zeros((70, 8), np.float32)
    confs[:, 1] = rng.integers(0, 2, 70)
    confs[:, 2:] = rng.normal(0.0, 1.0, (70, 6))
    d = lib.DeviceComplex(ctx, cx)
    want = orc.similarity_matrix(cx, confs)
    # inputs, union, bounds, counts, ranks, the lists (optional), matrix, maps
    for nth in range(1, 9):
        ctx.set_alloc_fail(nth)
        if nth == 6:
            assert np.array_equal(d.similarity_matrix(confs), want)
        else:
            with pytest.raises(lib.GdError) as exc:
                d.similarity_matrix(confs)
            assert exc.value.status == abi.GD_ENOMEM
        _used_up(ctx, cx)
    assert np.array_equal(d.similarity_matrix(confs), want)
    d.close()


def test_large_workspace_is_of_the_default_pool(ctx):
    """A matrix beyond what the work pool keeps: its memory is the default
    pool's, for uploads and runs to take next, and given back."""
    cx = synth.make_complex(synth.ComplexSpec(pnp=300, lna=8), seed=105)
    n = 4200
    confs = np.zeros((n, 8), np.float32)
    confs[:, 2:] = np.random.default_rng(4).normal(0.0, 1.0, (n, 6))
    d = lib.DeviceComplex(ctx, cx)
    used = _pool_used()
    _high(reset=True)
    got = d.similarity_matrix(confs)
    assert _high() >= used + got.nbytes and _pool_used() == used
    pick = np.arange(0, n, 97)
    assert np.array_equal(got[np.ix_(pick, pick)], d.similarity_matrix(confs[pick]))
    d.close()
