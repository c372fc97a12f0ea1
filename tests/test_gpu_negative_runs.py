"""Runs that start and end at negative samples in the middle of the walk: a
ray split over 1 to 8 lanes whose parts begin in, skip to, or end at negative
samples, and cells next to a negative node that hold infinities, NaN or
near-overflow values. Against the FP64 oracle: nearest mode bit for bit (each
pixel is its run's length), trilinear within the path's 1e-5 with the same
dark and non-finite pixels."""
import os

import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu

TOL = 1e-5
THREADS = os.cpu_count() or 4
AXES = (np.linspace(-9.0, 9.0, 31), np.linspace(-8.0, 10.0, 28), np.linspace(-9.5, 9.0, 33))


def o_cam(oracle, cam):
    return oracle.camera64(tuple(cam.pos), tuple(cam.aim), cam.fov_w_deg, cam.fov_h_deg, cam.nx, cam.ny,
                           cam.n_samples, cam.ray_length, cam.march)


def slabs(period, width):
    """Positive values with negative slabs across the line of sight (x and y)."""
    rng = np.random.default_rng(period)
    v = rng.uniform(0.5, 2.0, tuple(len(a) for a in AXES[::-1])).astype(np.float32)
    i = np.arange(len(AXES[0]))
    j = np.arange(len(AXES[1]))
    v[:, :, (i + 3) % period < width] *= -1
    v[:, (j % (2 * period)) == 1, :] *= -1
    return v


@pytest.mark.parametrize("segments", [1, 2, 4, 8])
@pytest.mark.parametrize("period,width", [(6, 1), (9, 4), (30, 20)])
@pytest.mark.parametrize("layout", [0, 1, 2])
def test_runs_across_lanes(birp, oracle, segments, period, width, layout):
    v = slabs(period, width)
    for tri in (False, True):
        w = v if tri else np.sign(v)
        cube = birp.Cube(*AXES, w, layout=layout)
        oc = oracle.Cube64(*AXES, w.astype(np.float64), int(tri))
        for march in (birp.PREFIX, birp.CLIP):
            for pos in ((-8.5, -1.0, 2.0), (-20.0, -3.0, 1.0), (4.0, 6.0, 8.0)):
                cam = birp.camera(pos, (10, 0, 0), 40.0, 30.0, 33, 29, n_samples=613, ray_length=44.0, trilinear=tri,
                                  march=march, segments=segments)
                img = birp.render(cube, cam)
                ref = oracle.render64(oc, o_cam(oracle, cam), threads=THREADS)
                if tri:
                    mx, rms, n = rel_err(img, ref)
                    assert mx <= TOL and np.array_equal(img == 0, ref == 0), (pos, march, mx)
                else:
                    assert np.array_equal(img, ref.astype(np.float32)), (pos, march)
        cube.close()


@pytest.mark.parametrize("layout", [0, 1, 2])
def test_special_values_next_to_negative_nodes(birp, oracle, layout):
    v = slabs(40, 0)
    rng = np.random.default_rng(3)
    for special in (np.inf, np.nan, 2e38):
        for _ in range(6):
            z, y, x = (int(rng.integers(2, n - 3)) for n in v.shape)
            v[z, y, x] = special
            v[z, y, x + 1] = -1.0
    cube = birp.Cube(*AXES, v, layout=layout)
    oc = oracle.Cube64(*AXES, v.astype(np.float64), 1)
    for march in (birp.PREFIX, birp.CLIP):
        cam = birp.camera((-8.5, -1.0, 2.0), (10, 0, 0), 60.0, 50.0, 61, 47, n_samples=800, ray_length=44.0, march=march)
        img = birp.render(cube, cam)
        with np.errstate(all="ignore"):
            ref = oracle.render64(oc, o_cam(oracle, cam), threads=THREADS)
            ref32 = ref.astype(np.float32)
        fine = np.isfinite(ref32)
        assert np.array_equal(fine, np.isfinite(img)) and (~fine).sum() > 0
        small = fine & (ref < 1e30)  # rays past a 2e38 node apart: relative errors against their own size
        for m in (small, fine & ~small):
            if m.any():
                err = np.abs(img[m].astype(np.float64) - ref[m]) / np.abs(ref[m]).max()
                assert err.max() <= TOL
        assert np.array_equal(img == 0, ref32 == 0)
    cube.close()
