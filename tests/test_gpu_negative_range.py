"""Cubes with negative values whose values lie at the lower end of FP32's range,
where float pairs have no room for their low parts: a run ends at its first
negative sample, so one sign taken wrongly drops the rest of a ray. A cube's
signs do not change when its values are multiplied by a power of two, and
neither then do the samples of any ray: the number of samples summed is the
same, exactly, as with the same values far from the end of the range."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

AXES = (np.linspace(-9.0, 9.0, 31), np.linspace(-8.0, 10.0, 28), np.linspace(-9.5, 9.0, 33))


@pytest.mark.parametrize("units", [8, 100, 3000, 1 << 20])
@pytest.mark.parametrize("layout", [0, 1, 2])
def test_runs_of_tiny_values(birp, layout, units):
    """Values up to 4 x units of FP32's smallest step, 2^-149 (the last ones are normal numbers)."""
    rng = np.random.default_rng(units)
    shape = tuple(len(a) for a in AXES[::-1])
    v = np.where(rng.random(shape) < 0.06, -rng.integers(1, units + 1, shape), rng.integers(1, 4 * units, shape))
    v[8:12, 10:20, 5:25] = 0
    counts = []
    for shift in (-149, -30):
        w = np.ldexp(v.astype(np.float64), shift).astype(np.float32)
        assert np.array_equal(np.ldexp(w.astype(np.float64), -shift), v)
        cube = birp.Cube(*AXES, w, layout=layout)
        got = []
        for march in (birp.PREFIX, birp.CLIP):
            for pos in ((-8.5, -1.0, 2.0), (3.0, 4.0, -2.0), (-12.0, 9.0, 11.0)):
                cam = birp.camera(pos, (10, 0, 0), 70.0, 60.0, 161, 127, n_samples=613, ray_length=24.0, trilinear=True,
                                  march=march)
                birp.kernel_stats(reset=True)
                birp.render(cube, cam)
                got.append(birp.kernel_stats()["samples"])
        counts.append(got)
        cube.close()
    assert counts[0] == counts[1]
