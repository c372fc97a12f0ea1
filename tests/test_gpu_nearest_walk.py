"""The nearest walk's crossings where they can go wrong, bit for bit against
the FP64 oracle: samples exactly on node planes (rays along an axis whose step
divides the cells), rays almost parallel to the planes, steps longer than
several cells, one sample, very many samples, and every split over lanes. The
field takes distinct powers of two per node, so a sample in another cell than
the oracle's changes the sum."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

THREADS = os.cpu_count() or 4


def o_cam(oracle, cam):
    return oracle.camera64(tuple(cam.pos), tuple(cam.aim), cam.fov_w_deg, cam.fov_h_deg, cam.nx, cam.ny,
                           cam.n_samples, cam.ray_length, cam.march)


def cube(birp, n, layout, seed):
    rng = np.random.default_rng(seed)
    axes = [np.linspace(-8.0, 8.0, n), np.linspace(-4.0, 12.0, n), np.linspace(-10.0, 6.0, n)]
    v = np.exp2(rng.integers(-3, 4, (n, n, n))).astype(np.float32)
    return axes, v, birp.Cube(*axes, v, layout=layout)


# pose, aim: in general position; on node planes looking along x; nearly along x
VIEWS = [((1.0, -3.0, 4.0), (6.0, 0, 0)), ((-7.5, 0.0, 0.0), (6.0, 0, 0)), ((-7.5, 1e-3, 2e-3), (6.0, 0, 0)),
         ((0.0, 0.0, 5.0), (0.0, 0, 0)), ((-30.0, 2.0, -2.0), (6.0, 0, 0))]


@pytest.mark.parametrize("layout", [0, 1, 2])
@pytest.mark.parametrize("nodes,samples,length", [(17, 320, 16.0), (33, 640, 32.0), (65, 9, 30.0), (9, 1, 3.0),
                                                  (5, 60000, 25.0), (33, 1001, 29.7)])
@pytest.mark.parametrize("segments", [1, 4, 8])
def test_walk_bitwise(birp, oracle, layout, nodes, samples, length, segments):
    axes, v, g = cube(birp, nodes, layout, nodes + samples)
    oc = oracle.Cube64(*axes, v.astype(np.float64), 0)
    for pos, aim in VIEWS:
        for fov in (30.0, 0.01):
            for march in (birp.PREFIX, birp.CLIP):
                cam = birp.camera(pos, aim, fov, fov, 13, 11, n_samples=samples, ray_length=length, trilinear=False,
                                  march=march, segments=segments)
                img = birp.render(g, cam)
                ref = oracle.render64(oc, o_cam(oracle, cam), threads=THREADS).astype(np.float32)
                assert np.array_equal(img, ref), (pos, fov, march, np.abs(img - ref).max())
    g.close()


# Rays tilted against an axis by less and less, down to 1e-13: the walk's crossing index of a plane has 1 / (d dt) up
# to 1e14 in it, and each of its estimates ends somewhere on the way.
@pytest.mark.parametrize("tilt", [1e-4, 1e-6, 1e-8, 1e-9, 1e-10, 1e-11, 1e-13])
@pytest.mark.parametrize("nodes,samples", [(17, 321), (33, 2000)])
def test_walk_nearly_parallel(birp, oracle, tilt, nodes, samples):
    axes, v, g = cube(birp, nodes, 1, nodes)
    oc = oracle.Cube64(*axes, v.astype(np.float64), 0)
    for fov in (1e-3, 1e3 * tilt):
        for march in (birp.PREFIX, birp.CLIP):
            cam = birp.camera((-7.5, tilt, -2 * tilt), (6.0, 0, 0), fov, fov, 9, 7, n_samples=samples, ray_length=17.0,
                              trilinear=False, march=march)
            img = birp.render(g, cam)
            ref = oracle.render64(oc, o_cam(oracle, cam), threads=THREADS).astype(np.float32)
            assert np.array_equal(img, ref), (fov, march, np.abs(img - ref).max())
    g.close()
