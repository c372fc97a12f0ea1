"""Cubes whose values go through the library's pinned memory (up to 32768 nodes)
and just larger ones: the same cube, sign flag and images bit for bit as by the
copies, from pageable, pinned and oddly placed values, with a negative value at
either end; and many threads building small cubes at a time."""
import ctypes as C
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(2, 2, 2), (5, 4, 3), (32, 32, 31), (32, 32, 32), (32, 32, 33), (181, 181, 2)]


def axes(shape):
    return [np.linspace(-9.0, 9.0 + k, n) for k, n in enumerate(shape)]


def field(shape, seed, negative):
    v = np.random.default_rng(seed).uniform(0.5, 2.0, shape[::-1]).astype(np.float32)
    if negative is not None:
        v.reshape(-1)[negative] = -0.25
    return v


def make(birp, shape, address, layout):
    xs, ys, zs = axes(shape)
    h = C.c_void_p()
    birp.check(birp.lib().birp_cube_create_layout(
        *[a for ax in (xs, ys, zs) for a in (C.c_void_p(ax.ctypes.data), len(ax))], C.c_void_p(address), layout,
        C.byref(h)))
    return h


def images(birp, h):
    got = []
    for tri in (False, True):
        for pos in ((-8.5, -1.0, 2.0), (-20.0, 3.0, 1.0)):
            cam = birp.camera(pos, (10, 0, 0), 60.0, 50.0, 31, 23, n_samples=300, ray_length=44.0, trilinear=tri,
                              march=birp.CLIP)
            img = np.empty((23, 31), np.float32)
            birp.check(birp.lib().birp_render(h, None, C.byref(cam), C.c_void_p(img.ctypes.data), None))
            got.append(img)
    birp.lib().birp_cube_destroy(h)
    return got


@pytest.mark.parametrize("layout", [0, 1, 2])
@pytest.mark.parametrize("shape", SHAPES, ids=str)
@pytest.mark.parametrize("negative", [None, 0, -1])
def test_same_cube(birp, monkeypatch, layout, shape, negative):
    import torch
    v = field(shape, 5, negative)
    monkeypatch.setenv("BIRP_HOST_DIRECT", "0")
    want = images(birp, make(birp, shape, v.ctypes.data, layout))
    monkeypatch.delenv("BIRP_HOST_DIRECT")
    pinned = torch.from_numpy(v).pin_memory()
    odd = np.zeros(v.nbytes + 8, np.uint8)
    odd[3:3 + v.nbytes] = v.view(np.uint8).reshape(-1)
    for address in (v.ctypes.data, pinned.data_ptr(), odd.ctypes.data + 3):
        for a, b in zip(images(birp, make(birp, shape, address, layout)), want):
            assert np.array_equal(a, b)


def test_threads(birp):
    cases = [(s, seed, n) for s in SHAPES[:5] for seed, n in ((1, None), (2, 0))]
    fields = [field(*c) for c in cases]
    want = [images(birp, make(birp, c[0], v.ctypes.data, 1)) for c, v in zip(cases, fields)]
    bad = []

    def work(t):
        for i in range(40):
            k = (3 * t + i) % len(cases)
            got = images(birp, make(birp, cases[k][0], fields[k].ctypes.data, 1))
            if not all(np.array_equal(a, b) for a, b in zip(got, want[k])):
                bad.append((t, cases[k]))

    th = [threading.Thread(target=work, args=(t,)) for t in range(4)]
    for t in th:
        t.start()
    for t in th:
        t.join()
    assert not bad, bad[:4]
