"""The far form of the pair terms (points beyond every atom of a warp by the
type pairs' far distance) against the CPU oracle: protein sizes at the edges of
chunks and tiles, ligands moved so that none, some or all of the points are
far, and force fields whose terms reach further than the packaged one's."""
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


def _complex(pnp, lna, shift, ff_edit=None, n_lig=3):
    cx = synth.make_complex(synth.ComplexSpec(pnp=pnp, lna=lna, n_lig=n_lig,
                                            n_psp=32 if pnp >= 100 else 0), seed=300 + pnp)
    cx.lig_center = (cx.lig_center + np.float32([shift, 0.0, 0.0])).astype(np.float32)
    if ff_edit:
        tab = abi.enepara_to_arrays(cx.ff)
        ff_edit(tab)
        cx.ff = abi.enepara_from_arrays(tab)
    cx._struct = None
    return cx


def _long_electrostatics(tab):
    tab["el1"] = np.float32(0.03)  # near-field up to 33 A


def _long_pmf(tab):
    tab["pmf0"] = tab["pmf0"] + np.float32(9.0)


def _wide_hbond(tab):
    tab["hdb1"] = np.where(np.isfinite(tab["hdb1"]), tab["hdb1"] * np.float32(0.2), tab["hdb1"])


def _check(cx, terms, poses, conf):
    terms_r, raw_r, asum = orc.energy_poses(cx, poses, 0, conf)
    bad, rel = tol.check_terms(terms, terms_r, raw_r, asum, cx.ff)
    assert not bad.any(), (np.argwhere(bad)[:5], np.nanmax(rel, axis=0))


@pytest.mark.parametrize("pnp", [1, 31, 32, 33, 127, 128, 129, 700, 2500])
@pytest.mark.parametrize("shift", [0.0, 21.0, 300.0])
def test_far_sizes(ctx, pnp, shift):
    """The start energies of a run (3 ligand conformations x 7 temperatures,
    lanes without a replica among them)."""
    cx = _complex(pnp, 23, shift)
    d = lib.DeviceComplex(ctx, cx)
    _, mb = lib.set_temperature(7, 0.004, 0.04)
    r = lib.Remc(d, 10, 10, mb)
    r.init()
    e = r.read().energy.reshape(7, 3, abi.NTERM)
    for conf in range(3):
        _check(cx, e[:, conf], np.zeros((7, 6), np.float32), conf)


@pytest.mark.parametrize("edit", [_long_electrostatics, _long_pmf, _wide_hbond])
@pytest.mark.parametrize("lna", [5, 40])
def test_far_other_force_fields(ctx, edit, lna):
    cx = _complex(2500, lna, 12.0, edit, n_lig=1)
    d = lib.DeviceComplex(ctx, cx)
    _, mb = lib.set_temperature(8, 0.004, 0.04)
    r = lib.Remc(d, 10, 10, mb)
    r.init()
    _check(cx, r.read().energy, np.zeros((8, 6), np.float32), 0)
