"""Cubes in other units than Earth radii: coordinates from 1e-9 to 1e13, values
from 1e-10 to 1e10. The records' coefficients (products of up to three inverse
cell widths) keep FP32's precision: GetSample against FP64 within 1e-6 of the
values around a point (8 roundings of 6e-8 and the result's), as long as FP32
holds them, each layout."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("unit", [1e-9, 1e-3, 1e3, 6.378e6, 1e9, 3e11, 3e12, 1e13])
@pytest.mark.parametrize("value", [1e-10, 1.0, 1e10])
@pytest.mark.parametrize("layout", [0, 1, 2])
def test_sample(birp, unit, value, layout):
    rng = np.random.default_rng(3)
    axes = [np.cumsum(rng.uniform(0.7, 1.3, n)) * unit for n in (13, 11, 12)]
    v = (rng.uniform(0.5, 2.0, (12, 11, 13)) * value).astype(np.float32)
    with np.errstate(all="ignore"):
        c7 = np.abs(np.diff(np.diff(np.diff(v.astype(np.float64), axis=0), axis=1), axis=2)).max() / unit ** 3
    if layout == 0 and not (1e-30 < c7 < 1e30):
        pytest.skip("FP32 does not hold the coefficients")
    lo, hi = np.array([a[0] for a in axes]), np.array([a[-1] for a in axes])
    p = (lo + (hi - lo) * rng.uniform(0.001, 0.999, (4000, 3))).astype(np.float32)
    x = p.astype(np.float64)
    k = [np.clip(np.searchsorted(a, x[:, i], "right") - 1, 0, len(a) - 2) for i, a in enumerate(axes)]
    f = [(x[:, i] - a[k[i]]) / (a[k[i] + 1] - a[k[i]]) for i, a in enumerate(axes)]
    d = v.astype(np.float64)
    c = [d[k[2] + (q >> 2), k[1] + ((q >> 1) & 1), k[0] + (q & 1)] for q in range(8)]
    y = [c[2 * q] + f[0] * (c[2 * q + 1] - c[2 * q]) for q in range(4)]
    z = [y[2 * q] + f[1] * (y[2 * q + 1] - y[2 * q]) for q in range(2)]
    want = z[0] + f[2] * (z[1] - z[0])
    cube = birp.Cube(*axes, v, layout=layout)
    got = cube.sample(p).astype(np.float64)
    cube.close()
    err = np.abs(got - want) / np.max(np.abs(c), axis=0)
    assert err.max() <= 1e-6, err.max()
