"""DataCube::GetSample where the exact float-pair cell choice and the
float-float interpolation can go wrong: points on and one FP32 step either
side of every node (nodes FP32 cannot hold among them), on the box's faces,
non-finite points and values, values at the ends of FP32's range; each layout,
both ways the call reaches its arrays (in place, and copied where results
overlap points). Cells bit for bit through nearest mode; trilinear values
against FP64 within 1e-6 of the values around the point (an FP32 record's
8 coefficients: 8 roundings of 6e-8, and the result's)."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

AXES = {
    "uniform": (np.linspace(-10.0, 20.0, 31), np.linspace(-0.3, 0.7, 11), np.linspace(-1 / 3, 5.1, 24)),
    "far": (1000.0 + np.linspace(0, 3, 13) ** 1.5, np.linspace(-1e-3, 1e-3, 9), np.linspace(-7.7, 4.4, 12) ** 3),
    "small": (np.array([0.1, 0.2]), np.array([-1.0, 0.0, 1e-4]), np.array([-0.7, 0.1, 3.3])),
}


def points(axes, seed):
    rng = np.random.default_rng(seed)
    lo, hi = np.array([a[0] for a in axes]), np.array([a[-1] for a in axes])
    p = [rng.uniform(lo - 0.05 * (hi - lo), hi + 0.05 * (hi - lo), (4000, 3)).astype(np.float32)]
    for k, a in enumerate(axes):
        c = a.astype(np.float32)
        for x in (c, np.nextafter(c, np.float32(np.inf)), np.nextafter(c, np.float32(-np.inf))):
            q = rng.uniform(lo, hi, (len(a), 3)).astype(np.float32)
            q[:, k] = x
            p.append(q)
    corners = np.stack(np.meshgrid(*[a[[0, -1]] for a in axes]), -1).reshape(-1, 3).astype(np.float32)
    bad = np.tile(p[0][:1], (4, 1))
    bad[0, 0], bad[1, 1], bad[2, 2], bad[3, 0] = np.nan, np.inf, -np.inf, 3e38
    return np.concatenate(p + [corners, bad])


def exact(axes, v, p):
    """FP64 cell, value and largest neighbour of each point; in-box mask."""
    x = p.astype(np.float64)
    inside = np.all([(x[:, k] >= a[0]) & (x[:, k] < a[-1]) for k, a in enumerate(axes)], axis=0)
    i, f = [], []
    for k, a in enumerate(axes):
        j = np.clip(np.searchsorted(a, np.where(inside, x[:, k], a[0]), "right") - 1, 0, len(a) - 2)
        i.append(j)
        f.append((np.where(inside, x[:, k], a[0]) - a[j]) / (a[j + 1] - a[j]))
    d = v.astype(np.float64)
    c = [d[i[2] + (q >> 2), i[1] + ((q >> 1) & 1), i[0] + (q & 1)] for q in range(8)]
    with np.errstate(all="ignore"):
        y = [c[2 * q] + f[0] * (c[2 * q + 1] - c[2 * q]) for q in range(4)]
        z = [y[2 * q] + f[1] * (y[2 * q + 1] - y[2 * q]) for q in range(2)]
        t = z[0] + f[2] * (z[1] - z[0])
    return inside, c[0], t, np.max(np.abs(c), axis=0)


@pytest.mark.parametrize("layout", [0, 1, 2])
@pytest.mark.parametrize("name", list(AXES))
def test_cells_and_values(birp, layout, name):
    axes = AXES[name]
    rng = np.random.default_rng(7)
    v = rng.uniform(0.5, 2.0, tuple(len(a) for a in axes[::-1])).astype(np.float32)
    p = points(axes, 11)
    cube = birp.Cube(*axes, v, layout=layout)
    inside, low, tri, size = exact(axes, v, p)
    near = cube.sample(p, trilinear=False)
    assert np.array_equal(near, np.where(inside, low, -1.0).astype(np.float32))
    got = cube.sample(p).astype(np.float64)
    assert np.array_equal(got == -1, ~inside)
    assert np.all(np.abs(got - tri)[inside] <= 1e-6 * size[inside])
    cube.close()


@pytest.mark.parametrize("layout", [1, 2])
@pytest.mark.parametrize("scale", [1e-42, 1e-30, 1e-19, 1e29, 1e38])
def test_range_of_values(birp, layout, scale):
    """Node-value layouts: FP64 takes over where float-float has no room."""
    axes = AXES["uniform"]
    rng = np.random.default_rng(8)
    v = (rng.uniform(0.5, 2.0, tuple(len(a) for a in axes[::-1])) * scale).astype(np.float32)
    v[5, 4, 6] = np.inf
    v[9, 3, 20] = np.nan
    v[12:16, 2:6, 8:14] = 0.0
    p = points(axes, 12)
    cube = birp.Cube(*axes, v, layout=layout)
    inside, low, tri, size = exact(axes, v, p)
    got = cube.sample(p)
    want = np.where(inside, tri, -1.0).astype(np.float32)
    fine = np.isfinite(want)
    assert np.array_equal(fine, np.isfinite(got))
    err = np.abs(got.astype(np.float64) - want)[fine]
    assert np.all(err <= 1e-6 * np.where(inside, size, 1.0)[fine] + 1.5e-45)
    cube.close()


@pytest.mark.parametrize("n", [1, 31, 257, 5000])
def test_results_over_points(birp, n):
    """out inside xyz: results as from separate arrays."""
    axes = AXES["uniform"]
    v = np.random.default_rng(9).uniform(0.5, 2.0, tuple(len(a) for a in axes[::-1])).astype(np.float32)
    cube, model = birp.Cube(*axes, v), birp.Cmem()
    p = np.resize(points(axes, 13), (n, 3)).astype(np.float32)
    want, want_m = cube.sample(p), model.sample(p)
    L = birp.lib()
    for shift in (0, n):
        buf = p.copy().reshape(-1)
        birp.check(L.birp_cube_sample(cube.h, 1, ctypes.c_void_p(buf.ctypes.data), n,
                                      ctypes.c_void_p(buf.ctypes.data + 4 * shift)))
        assert np.array_equal(buf[shift:shift + n], want)
        buf = p.copy().reshape(-1)
        birp.check(L.birp_cmem_sample(model.h, ctypes.c_void_p(buf.ctypes.data), n,
                                      ctypes.c_void_p(buf.ctypes.data + 4 * shift)))
        assert np.array_equal(buf[shift:shift + n], want_m, equal_nan=True)
    cube.close()
    model.close()
