"""Large pose calls, whose poses are dealt into cells of their translation,
and small ones, whose points are split over clusters and lane groups: every
pose against the oracle, poses without a usable translation, far outliers and
duplicates among them; and the same bits in any order of the poses."""
import numpy as np
import pytest

from gpudock_b200 import abi, lib, synth
from oracle import oracle as orc
from tests import tolerance as tol

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = lib.Context(0)
    yield c
    c.close()


def _check(cx, poses, terms, raw, pick):
    terms_r, raw_r, asum = orc.energy_poses(cx, poses[pick])
    bad, rel = tol.check_raw(raw[pick], raw_r, asum)
    assert not bad.any(), np.nanmax(rel, axis=0)
    bad, rel = tol.check_terms(terms[pick], terms_r, raw_r, asum, cx.ff)
    assert not bad.any(), np.nanmax(rel, axis=0)


# 2,500 x 50: cells from 2,048 poses on, in one launch up to 16,384; pose counts
# at the edges of blocks and of the rule; boxes of one cell and of many
@pytest.mark.parametrize("n", [2047, 2048, 4097, 16384, 16385, 20001])
@pytest.mark.parametrize("box", [0.0, 6.0, 40.0])
def test_pose_cells(ctx, n, box):
    cx = synth.make_complex(synth.ComplexSpec(pnp=2500, lna=50), seed=95)
    rng = np.random.default_rng(n)
    poses = synth.random_poses(rng, n, box=box)
    poses[7] = poses[8]                      # a duplicate
    poses[100, 0] = 900.0                    # widens the box
    poses[200, 1], poses[300, 2] = np.nan, np.inf
    poses[400, 0] = 1e5                      # no usable translation
    d = lib.DeviceComplex(ctx, cx)
    terms, raw = d.energy_poses(poses)
    perm = rng.permutation(n)
    again, _ = d.energy_poses(poses[perm])
    assert np.array_equal(again, terms[perm], equal_nan=True)
    assert np.isnan(terms[[200, 300], abi.E_TOTAL]).all()
    ok = np.setdiff1d(np.arange(n), [200, 300, 400])
    assert np.isfinite(terms[ok]).all()
    assert np.array_equal(terms[7], terms[8])
    _check(cx, poses, terms, raw, np.r_[7, 8, 100, rng.choice(ok, 150, replace=False)])


@pytest.mark.parametrize("n", [1, 7, 8, 9, 17, 33, 64, 150, 700, 3000])
@pytest.mark.parametrize("lna,pnp", [(9, 300), (24, 1500), (70, 6100)])
def test_small_calls(ctx, n, lna, pnp):
    cx = synth.make_complex(synth.ComplexSpec(pnp=pnp, lna=lna), seed=96)
    poses = synth.random_poses(np.random.default_rng(n), n, box=5.0)
    d = lib.DeviceComplex(ctx, cx)
    terms, raw = d.energy_poses(poses)
    _check(cx, poses, terms, raw, np.arange(n)[-60:])
