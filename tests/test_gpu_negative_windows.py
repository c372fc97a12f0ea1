"""Rays of cubes with many negative values are gone over in windows: no lane of
a ray walks far past the run's end (the cells summed stay near the run's own
number), and images and run lengths are those of the FP64 oracle whatever the
window a run starts, pauses or ends in, by every way to render."""
import os

import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu

TOL = 1e-5
THREADS = os.cpu_count() or 4
AXES = (np.linspace(-9.0, 9.0, 49), np.linspace(-8.0, 10.0, 44), np.linspace(-9.5, 9.0, 51))
Z, Y, X = np.meshgrid(*AXES[::-1], indexing="ij")


def field(name):
    rng = np.random.default_rng(4)
    if name == "ball":
        return (np.sqrt(X * X + Y * Y + Z * Z) - 5.0).astype(np.float32)
    if name == "smooth":
        return (np.sin(X) * np.cos(Y / 1.5) + np.sin(Z / 2) + 0.3).astype(np.float32)
    share = float(name)
    v = rng.uniform(0.5, 2.0, X.shape)
    return np.where(rng.random(X.shape) < share, -rng.uniform(0.1, 1.0, X.shape), v).astype(np.float32)


def o_cam(oracle, cam):
    return oracle.camera64(tuple(cam.pos), tuple(cam.aim), cam.fov_w_deg, cam.fov_h_deg, cam.nx, cam.ny,
                           cam.n_samples, cam.ray_length, cam.march)


@pytest.mark.parametrize("name,pos", [("ball", (1.0, 0.5, -0.5)), ("0.95", (0.3, -0.7, 0.4)), ("0.5", (0.3, -0.7, 0.4)),
                                      ("smooth", (1.0, -5.2, -3.1))])
@pytest.mark.parametrize("samples", [880, 20000])
def test_no_walk_past_a_short_run(birp, name, pos, samples):
    cube = birp.Cube(*AXES, field(name))
    cam = birp.camera(pos, (10, 0, 0), 40.0, 30.0, 40, 30, n_samples=samples, ray_length=44.0, trilinear=True, segments=8)
    birp.kernel_stats(reset=True)
    birp.render(cube, cam)
    s = birp.kernel_stats()
    cell = 18.0 / 48 / (44.0 / samples)  # samples across a cell
    # the run's own cells, and per lane those of its last window (up to 3 times the run) and a cell begun
    assert s["cells"] <= 4 * (3 * s["samples"] / cell) + 2 * 8 * 40 * 30 + 4 * s["samples"] / min(cell, 1.0)
    cube.close()


@pytest.mark.parametrize("name", ["ball", "smooth", "0.02", "0.2", "0.6"])
@pytest.mark.parametrize("layout", [0, 1, 2])
def test_against_the_oracle(birp, oracle, name, layout):
    v = field(name)
    cube = birp.Cube(*AXES, v, layout=layout)
    batch = birp.Batch(64, 1 << 17)
    items, refs = [], []
    for tri in (True, False):
        w = v if tri else np.sign(v)
        oc = oracle.Cube64(*AXES, w.astype(np.float64), int(tri))
        space = cube if tri else birp.Cube(*AXES, w, layout=layout)
        for march in (birp.PREFIX, birp.CLIP):
            for pos in ((1.0, 0.5, -0.5), (-8.5, -1.0, 2.0), (-20.0, -3.0, 1.0)):
                for segments, samples in ((1, 613), (8, 613), (4, 5), (0, 3000)):
                    cam = birp.camera(pos, (10, 0, 0), 50.0, 40.0, 33, 29, n_samples=samples, ray_length=44.0,
                                      trilinear=tri, march=march, segments=segments)
                    items.append((space, cam))
                    refs.append(oracle.render64(oc, o_cam(oracle, cam), threads=THREADS))
    for start in range(0, len(items), 24):
        part = items[start:start + 24]
        for (space, cam), img, ref in zip(part, batch.render(part), refs[start:start + 24]):
            for got in (img, birp.render(space, cam)):
                assert np.array_equal(got == 0, ref == 0), (tuple(cam.pos), cam.n_samples, cam.march)
                if cam.trilinear:
                    assert rel_err(got, ref)[0] <= TOL
                else:
                    assert np.array_equal(got, ref.astype(np.float32))
    batch.close()
