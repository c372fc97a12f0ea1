"""Cubes built from values the device reads where they lie, against the copied
ones bit for bit: odd sizes and every start of the array relative to 16 bytes,
a negative value in each of the places where the copy's loads change (found or
not found), and values at the ends of FP32's range in the records layout."""
import ctypes
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(2, 2, 2), (3, 2, 5), (5, 4, 3), (17, 9, 13), (64, 33, 7), (131, 66, 45)]


class Copied:
    """Builds inside take the copies."""

    def __enter__(self):
        os.environ["BIRP_HOST_DIRECT"] = "0"

    def __exit__(self, *a):
        del os.environ["BIRP_HOST_DIRECT"]


def axes(shape):
    return [np.linspace(-4.0 - k, 5.0 + 0.3 * k, n) for k, n in enumerate(shape)]


def make(birp, shape, values, layout):
    """A cube from a raw pointer (the array may start anywhere)."""
    h = ctypes.c_void_p()
    ax = axes(shape)
    birp.check(birp.lib().birp_cube_create_layout(*[x for a in ax for x in (a.ctypes.data, len(a))],
                                                  values.ctypes.data, layout, ctypes.byref(h)))
    c = birp.Cube.__new__(birp.Cube)
    c.h, c.shape = h, shape[::-1]
    return c


def look(birp, cube):
    p = np.random.default_rng(1).uniform(-6, 7, (2000, 3)).astype(np.float32)
    cam = birp.camera((0.1, -0.2, 0.3), (3.0, 0, 0), 60.0, 50.0, 24, 17, n_samples=150, ray_length=12.0)
    return [cube.sample(p), cube.sample(p, trilinear=False), birp.render(cube, cam)], cube.info().device_bytes


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("layout", [0, 1, 2])
@pytest.mark.parametrize("start", [0, 1, 2, 3, "byte"])
def test_build_in_place(birp, shape, layout, start):
    n = int(np.prod(shape))
    rng = np.random.default_rng(n)
    raw = np.zeros(4 * n + 64, np.uint8)
    at = -raw.ctypes.data % 16 + (13 if start == "byte" else 4 * start)
    v = raw[at:at + 4 * n].view(np.float32) if start != "byte" else np.frombuffer(raw, np.float32, n, at)
    v[:] = rng.uniform(0.5, 2.0, n)
    places = [None, 0, 1, min(5, n - 1), n // 2, n - 2, n - 1]
    base = None
    for place in places:
        if place is not None:
            v[place] = -v[place]
        cube = make(birp, shape, v, layout)
        got, size = look(birp, cube)
        cube.close()
        with Copied():
            other = make(birp, shape, v, layout)
        want, want_size = look(birp, other)
        other.close()
        assert all(np.array_equal(a, b) for a, b in zip(got, want)), place
        assert size == want_size
        if base is None:
            base = size
        assert size - base == (n if place is not None else 0)
        if place is not None:
            v[place] = -v[place]


@pytest.mark.parametrize("scale", [1e-42, 1e-30, 1e-19, 1.0, 1e29, 1e37])
def test_records_range(birp, scale):
    """Coefficients of a record against FP64 through the field they give, at
    the middle of every cell: 8 roundings of the values around it."""
    shape = (9, 8, 7)
    ax = axes(shape)
    v = (np.random.default_rng(3).uniform(0.5, 2.0, shape[::-1]) * scale).astype(np.float32)
    v[2:4, 2:5, 3:6] = 0.0
    cube = birp.Cube(*ax, v)
    mid = [(a[1:] + a[:-1]) / 2 for a in ax]
    p = np.stack(np.meshgrid(*mid, indexing="ij"), -1).reshape(-1, 3).astype(np.float32)
    got = cube.sample(p).astype(np.float64)
    i = [np.searchsorted(a, p[:, k].astype(np.float64), "right") - 1 for k, a in enumerate(ax)]
    f = [(p[:, k] - a[i[k]]) / (a[i[k] + 1] - a[i[k]]) for k, a in enumerate(ax)]
    d = v.astype(np.float64)
    want, size = np.zeros(len(p)), np.zeros(len(p))
    for q in range(8):
        w = np.prod([f[k] if q >> k & 1 else 1 - f[k] for k in range(3)], axis=0)
        c = d[i[2] + (q >> 2), i[1] + ((q >> 1) & 1), i[0] + (q & 1)]
        want += w * c
        size = np.maximum(size, np.abs(c))
    assert np.all(np.abs(got - want) <= 1e-6 * size + 2e-44)
    cube.close()
