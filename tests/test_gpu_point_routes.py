"""The three ways of a sampling call's points to the kernel (through the
library's pinned memory up to 8192 points, read where they lie beyond, copied
where neither can be): the same results bit for bit at sizes around the line,
with results over points, with arrays at odd addresses, in device memory and
from several threads."""
import ctypes as C
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

AXES = (np.linspace(-10.0, 20.0, 31), np.linspace(-0.3, 9.7, 11), np.linspace(-1 / 3, 5.1, 24))
SIZES = [1, 33, 8191, 8192, 8193, 20000]


@pytest.fixture(scope="module")
def spaces(birp):
    v = np.random.default_rng(2).uniform(0.5, 2.0, tuple(len(a) for a in AXES[::-1])).astype(np.float32)
    cube, model = birp.Cube(*AXES, v), birp.Cmem()
    L = birp.lib()
    yield {"nearest": lambda x, n, o: L.birp_cube_sample(cube.h, 0, C.c_void_p(x), n, C.c_void_p(o)),
           "trilinear": lambda x, n, o: L.birp_cube_sample(cube.h, 1, C.c_void_p(x), n, C.c_void_p(o)),
           "cmem": lambda x, n, o: L.birp_cmem_sample(model.h, C.c_void_p(x), n, C.c_void_p(o))}
    cube.close()
    model.close()


def points(n, seed=3):
    return np.random.default_rng(seed).uniform((-11, -1, -1), (21, 10, 6), (n, 3)).astype(np.float32)


def call(f, p):
    out = np.full(len(p), np.nan, np.float32)
    assert f(p.ctypes.data, len(p), out.ctypes.data) == 0
    return out


@pytest.mark.parametrize("kind", ["nearest", "trilinear", "cmem"])
@pytest.mark.parametrize("n", SIZES)
def test_routes_agree(spaces, monkeypatch, kind, n):
    f, p = spaces[kind], points(n)
    got = call(f, p)
    assert np.isfinite(got).all()
    monkeypatch.setenv("BIRP_HOST_DIRECT", "0")
    want = call(f, p)
    monkeypatch.delenv("BIRP_HOST_DIRECT")
    assert np.array_equal(got, want)
    for first in (0, 2 * n):  # results over the points
        q = p.copy().reshape(-1)
        assert f(q.ctypes.data, n, q.ctypes.data + 4 * first) == 0
        assert np.array_equal(q[first:first + n], want)
    raw = np.zeros(16 * n + 64, np.uint8)  # addresses that are no multiple of 4
    a = raw.ctypes.data
    raw[1:1 + 12 * n] = p.view(np.uint8).reshape(-1)
    assert f(a + 1, n, a + 12 * n + 7) == 0
    assert np.array_equal(np.frombuffer(raw[12 * n + 7:16 * n + 7].tobytes(), np.float32), want)


@pytest.mark.parametrize("n", [10, 8192, 20000])
def test_device_pointers(spaces, n):
    """Points or results in device memory: copied from and to there."""
    import torch
    for f in spaces.values():
        p = points(n)
        want, got = call(f, p), np.zeros(n, np.float32)
        d, r = torch.from_numpy(p).cuda(), torch.zeros(n, device="cuda")
        torch.cuda.synchronize()
        assert f(d.data_ptr(), n, got.ctypes.data) == 0 and np.array_equal(got, want)
        assert f(p.ctypes.data, n, r.data_ptr()) == 0 and np.array_equal(r.cpu().numpy(), want)
        assert f(d.data_ptr(), n, r.data_ptr()) == 0 and np.array_equal(r.cpu().numpy(), want)


def test_threads(spaces):
    want = {(k, n): call(f, points(n, n)) for k, f in spaces.items() for n in SIZES}
    bad = []

    def work(t):
        for i in range(60):
            k, n = list(want)[(7 * t + i) % len(want)]
            if not np.array_equal(call(spaces[k], points(n, n)), want[k, n]):
                bad.append((t, k, n))

    th = [threading.Thread(target=work, args=(t,)) for t in range(4)]
    for t in th:
        t.start()
    for t in th:
        t.join()
    assert not bad, bad[:4]
