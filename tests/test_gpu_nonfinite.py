"""Values that are not finite, in calls that take the far form of the pair
terms: the same terms are NaN as where every point takes the full form (a call
of three poses), also where every point is far of the ligand."""
import numpy as np
import pytest

from gpudock_b200 import abi, lib, synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = lib.Context(0)
    yield c
    c.close()


def _complex():
    return synth.make_complex(synth.ComplexSpec(pnp=2500, lna=50), seed=95)


def _hbond_point(cx):
    """A protein point that has an H-bond term with some atom of the ligand."""
    hdb0 = abi.enepara_to_arrays(cx.ff)["hdb0"].reshape(abi.NLT, abi.NPT)
    return int(np.nonzero((hdb0[cx.lig_t][:, cx.prt_t] > 0.1).any(0))[0][0])


def _same(got, want):
    assert np.array_equal(np.isnan(got), np.isnan(want)), (got, want)
    np.testing.assert_allclose(got, want, rtol=2e-5, atol=1e-6)


@pytest.mark.parametrize("n", [2100, 4200, 17000])  # split; cells in one launch, in four
@pytest.mark.parametrize("far", [0.0, 60.0, 300.0])
@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
def test_angles(ctx, n, far, bad):
    cx = _complex()
    poses = synth.random_poses(np.random.default_rng(n), n, box=6.0)
    poses[-3:, 0] += np.float32(far)
    for k in range(3):
        poses[n - 3 + k, 3 + k] = bad
    d = lib.DeviceComplex(ctx, cx)
    terms, raw = d.energy_poses(poses)
    want, want_raw = d.energy_poses(poses[-3:])
    assert np.isnan(want_raw[:, [0, 1, 2, 4]]).all()
    _same(raw[-3:], want_raw)
    _same(terms[-3:], want)
    assert np.isfinite(terms[:-3]).all()


@pytest.mark.parametrize("what", ["atom", "point"])
@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("far", [0.0, 60.0, 300.0])
def test_coordinates(ctx, what, bad, far):
    """Poses in cells, and the start energies of units of 32 and of 8 replicas."""
    cx = _complex()
    cx.lig_center = (cx.lig_center + np.float32([far, 0.0, 0.0])).astype(np.float32)
    if what == "atom":
        cx.lig_xyz[:, 7, 1] = bad
    else:
        cx.prt_xyz[:, _hbond_point(cx), 0] = bad
    cx._struct = None
    d = lib.DeviceComplex(ctx, cx)
    poses = np.zeros((4200, 6), np.float32)
    want, want_raw = d.energy_poses(poses[:3])
    assert np.isnan(want_raw[0, [0, 2, 4]]).all()  # (1/d is 0 at an infinite distance)
    terms, raw = d.energy_poses(poses)
    _same(raw[:3], want_raw)
    _same(terms[:3], want)
    for n_tmp in (32, 8):
        _, mb = lib.set_temperature(n_tmp, 0.004, 0.04)
        r = lib.Remc(d, 10, 10, mb)
        r.init()
        _same(r.read().energy[:1], want[:1])
        r.close()
