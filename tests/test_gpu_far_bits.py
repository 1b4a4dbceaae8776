"""MC units of more than 16 replicas: a replica's energies are the same bits
wherever the unit's other replicas are, although that decides which points take
the far form.  Two ligand conformations share each unit; the second is a copy of
the first (most points far), lies in the protein (most points near) or far
outside.  The H-bond term counts without its offset, so that its smallest values
show."""
import numpy as np
import pytest

from gpudock_b200 import abi, lib, synth

pytestmark = pytest.mark.gpu

FLAGS = abi.MC_EXCHANGE | abi.MC_RECORD
FORCE_FIELDS = {"packaged": 1.0, "wide": 0.2, "narrow": 4.0}


@pytest.fixture(scope="module")
def ctx():
    c = lib.Context(0)
    yield c
    c.close()


def _run(ctx, cx, steps=20):
    d = lib.DeviceComplex(ctx, cx)
    _, mb = lib.set_temperature(16, 0.004, 0.04)
    r = lib.Remc(d, steps, 10, mb, seed=8, flags=FLAGS)
    r.init()
    first = r.read().energy.reshape(16, 2, abi.NTERM)[:, 0]
    r.run(steps)
    out = r.read()
    r.close()
    d.close()
    return first, out.record.reshape(16, 2, steps)[:, 0]


@pytest.mark.parametrize("ff", FORCE_FIELDS)
@pytest.mark.parametrize("shift", [0.0, 26.0, 33.0, 38.0, 44.0, 60.0, 90.0])
@pytest.mark.parametrize("lna,split", [(37, 1), (8, 2), (96, 1)])
def test_bits_do_not_depend_on_other_replicas(ctx, ff, shift, lna, split):
    cx = synth.make_complex(synth.ComplexSpec(pnp=1900, lna=lna, n_lig=2), seed=71)
    tab = abi.enepara_to_arrays(cx.ff)
    tab["hdb1"] = np.where(np.isfinite(tab["hdb1"]), tab["hdb1"] * np.float32(FORCE_FIELDS[ff]),
                           tab["hdb1"])
    tab["b_para"][abi.E_HDB] = 0.0
    cx.ff = abi.enepara_from_arrays(tab)
    cx.lig_center = (cx.lig_center + np.float32([shift, 0.0, 0.0])).astype(np.float32)
    ctx.set_split(split)
    got = []
    for off in (0.0, -shift, 70.0):
        cx.lig_xyz[1] = cx.lig_xyz[0] + np.float32([off, 0.0, 0.0])
        cx._struct = None
        got.append(_run(ctx, cx))
    ctx.set_split(0)
    for first, rec in got[1:]:
        assert np.array_equal(first, got[0][0])
        assert np.array_equal(rec, got[0][1])
