"""Similarity matrices bit for bit against the oracle at the edges of the
kernels' tiles: conformation counts about the 64 x 64 tile, protein sizes
about a word and a round of 2,048 points, unions of few and of many contacts
(maps kept in shared memory and in global memory), thresholds that no
distance or every distance meets."""
import numpy as np
import pytest

from gpudock_b200 import abi, lib, synth
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = lib.Context(0)
    yield c
    c.close()


def _confs(cx, n, spread, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    c = np.zeros((n, 8), np.float32)
    c[:, 0] = rng.integers(0, cx.n_prt, n)
    c[:, 1] = rng.integers(0, cx.n_lig, n)
    c[:, 2:5] = rng.normal(0.0, spread, (n, 3))
    c[:, 5:8] = rng.normal(0.0, 1.0, (n, 3))
    return c


@pytest.mark.parametrize("n,lna,pnp,spread", [
    (1, 5, 130, 1.0), (2, 33, 2048, 2.0), (63, 8, 2049, 2.0), (64, 31, 500, 3.0),
    (65, 32, 4100, 0.1), (129, 40, 1000, 30.0), (200, 110, 5000, 18.0)])
def test_sizes(ctx, n, lna, pnp, spread):
    cx = synth.make_complex(synth.ComplexSpec(pnp=pnp, lna=lna, n_prt=2, n_lig=3), seed=97)
    confs = _confs(cx, n, spread, n)
    d = lib.DeviceComplex(ctx, cx)
    assert np.array_equal(d.similarity_matrix(confs), orc.similarity_matrix(cx, confs))


@pytest.mark.parametrize("pmf0", [-1.0, 0.0, 60.0])
def test_thresholds(ctx, pmf0):
    """No pair, (almost) no pair, and nearly every pair is a contact: the last
    needs maps longer than shared memory holds."""
    cx = synth.make_complex(synth.ComplexSpec(pnp=3000, lna=100), seed=98)
    tab = abi.enepara_to_arrays(cx.ff)
    tab["pmf0"] = np.full_like(tab["pmf0"], pmf0)
    cx.ff = abi.enepara_from_arrays(tab)
    cx._struct = None
    confs = _confs(cx, 70, 2.0, 5)
    d = lib.DeviceComplex(ctx, cx)
    assert np.array_equal(d.similarity_matrix(confs), orc.similarity_matrix(cx, confs))
