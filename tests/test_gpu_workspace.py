"""The memory that a context keeps for its calls' workspaces: calls that grow it
and calls that need less, several threads on one context, a captured call
replayed beside others, and many contexts one after another."""
import threading
import time

import numpy as np
import pytest

from gpudock_b200 import abi, lib, synth

pytestmark = pytest.mark.gpu


def _complex(pnp=2500, lna=50):
    return synth.make_complex(synth.ComplexSpec(pnp=pnp, lna=lna, n_lig=2), seed=95)


def _confs(n, seed=3):
    rng = np.random.default_rng(seed)
    confs = np.zeros((n, 8), np.float32)
    confs[:, 1] = rng.integers(0, 2, n)
    confs[:, 2:] = rng.normal(0.0, 1.0, (n, 6))
    return confs


def _poses(n, seed=1):
    return synth.random_poses(np.random.default_rng(seed), n, box=6.0)


def _fresh(cx, call):
    ctx = lib.Context(0)
    d = lib.DeviceComplex(ctx, cx)
    out = call(d)
    d.close()
    ctx.close()
    return out


CALLS = [lambda d, n=n: d.energy_poses(_poses(n))[0] for n in (4100, 60000, 5000)] + \
        [lambda d, n=n: d.similarity_matrix(_confs(n)) for n in (40, 1500, 300)]


def test_calls_of_all_sizes_in_turn():
    cx = _complex()
    want = [_fresh(cx, c) for c in CALLS]
    ctx = lib.Context(0)
    d = lib.DeviceComplex(ctx, cx)
    for k in (0, 3, 1, 4, 2, 5, 0, 4, 1, 3):
        assert np.array_equal(CALLS[k](d), want[k])
    d.close()
    ctx.close()


def test_threads_on_one_context():
    cx = _complex()
    want = [_fresh(cx, c) for c in CALLS]
    ctx = lib.Context(0)
    d = lib.DeviceComplex(ctx, cx)
    bad = []

    def work(t):
        for i in range(8):
            k = (t + i * (t + 1)) % len(CALLS)
            if not np.array_equal(CALLS[k](d), want[k]):
                bad.append((t, i, k))

    threads = [threading.Thread(target=work, args=(t,)) for t in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
    d.close()
    ctx.close()


@pytest.mark.parametrize("n", [40, 4100, 20000])  # without cells, dealt in one launch, in four
def test_captured_call_beside_others(n):
    torch = pytest.importorskip("torch")
    stream = torch.cuda.Stream()
    ctx = lib.Context(0, stream.cuda_stream)
    cx = _complex()
    d = lib.DeviceComplex(ctx, cx)
    poses = [torch.from_numpy(_poses(n, seed)).cuda() for seed in range(3)]
    x, out = poses[0].clone(), torch.empty((n, abi.NTERM), device="cuda")
    want = []
    for p in poses:
        t = torch.empty_like(out)
        d.energy_poses_dev(n, p.data_ptr(), t.data_ptr())
        torch.cuda.synchronize()
        want.append(t)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.stream(stream):
        g.capture_begin(capture_error_mode="thread_local")
        d.energy_poses_dev(n, x.data_ptr(), out.data_ptr())
        g.capture_end()
    other, t = torch.cuda.Stream(), torch.empty_like(out)
    for k in range(3):
        x.copy_(poses[k])
        torch.cuda.synchronize()
        with torch.cuda.stream(other):  # the graph runs beside a call of another size
            g.replay()
        d.energy_poses_dev(n, poses[k - 1].data_ptr(), t.data_ptr())
        torch.cuda.synchronize()
        assert torch.equal(out, want[k]) and torch.equal(t, want[k - 1])
    del g
    d.close()
    ctx.close()


def test_calls_do_not_slow_down_with_the_contexts_before():
    cx = _complex(pnp=500, lna=8)
    confs = _confs(10)
    ctxs, best = [], []
    for _ in range(24):
        ctx = lib.Context(0)
        d = lib.DeviceComplex(ctx, cx)
        ts = []
        for _ in range(30):
            t = time.perf_counter()
            d.similarity_matrix(confs)
            ts.append(time.perf_counter() - t)
        best.append(min(ts))
        ctxs.append((ctx, d))
    assert min(best[-4:]) < 2.0 * min(best[:4]), best
    for ctx, d in ctxs:
        d.close()
        ctx.close()
