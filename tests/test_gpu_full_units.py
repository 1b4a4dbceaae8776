"""Full units of a complex whose last unit is small: the same bits as without
the small one (the ordered kernel), unsplit and on clusters, and the launch
rule behind it."""
import numpy as np
import pytest

from gpudock_b200 import abi, lib, synth
from tests import native


def test_rule(tmp_path):
    native.run(tmp_path, r"""
  auto packed = [](int nl, int nt) { return gd::all_packed_units(nl, nt); };
  // units of at most 16 replicas only
  CHECK(packed(1, 1) && packed(1, 8) && packed(2, 8) && packed(1, 16) && packed(2, 5) &&
        packed(16, 1) && packed(3, 5));
  // a full unit, alone or beside small ones; 17 .. 31 replicas
  CHECK(!packed(2, 16) && !packed(51, 16) && !packed(9, 4) && !packed(7, 8) && !packed(33, 1) &&
        !packed(7, 6) && !packed(1, 24) && !packed(3, 8) && !packed(1, 32) && !packed(1, 48));
""")


@pytest.mark.gpu
@pytest.mark.parametrize("lna", [9, 37, 70])
@pytest.mark.parametrize("n_lig,n_tmp", [(10, 16), (12, 8), (32, 2)])
@pytest.mark.parametrize("split", [1, 4])
def test_full_units_beside_a_small_one(lna, n_lig, n_tmp, split):
    """The start energies of the conformations in full units, with one more
    conformation (a unit of n_tmp replicas) and without."""
    ctx = lib.Context(0)
    ctx.set_split(split)
    cx = synth.make_complex(synth.ComplexSpec(pnp=1900, lna=lna, n_lig=n_lig + 1), seed=104)
    _, mb = lib.set_temperature(n_tmp, 0.004, 0.04)
    xyz, got = cx.lig_xyz, []
    for n in (n_lig, n_lig + 1):
        cx.lig_xyz = np.ascontiguousarray(xyz[:n])
        cx._struct = None
        d = lib.DeviceComplex(ctx, cx)
        r = lib.Remc(d, 10, 10, mb)
        r.init()
        got.append(r.read().energy.reshape(n_tmp, n, abi.NTERM)[:, :n_lig])
        r.close()
        d.close()
    assert np.array_equal(got[0], got[1])
    ctx.close()
