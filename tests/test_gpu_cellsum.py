"""The closed-form cell sum of the trilinear march where it can go wrong: cells
that hold no sample (several planes between two samples), exactly one, or
thousands, a ray of one sample, odd splits over lanes, and cells without a
sample that hold an infinity. Each layout against the FP64 oracle within the
path's 1e-5."""
import os

import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu

TOL = 1e-5
THREADS = os.cpu_count() or 4
LENGTH = 44.0


def field(n, seed):
    rng = np.random.default_rng(seed)
    axes = [np.linspace(-9.0, 9.0, n), np.linspace(-8.0, 10.0, n + 1), np.linspace(-9.5, 9.0, n + 2)]
    return (*axes, rng.uniform(0.5, 2.0, (n + 2, n + 1, n)).astype(np.float32))


def camera(birp, samples, segments=0):
    return birp.camera((1.0, -5.0, 4.0), (10, 0, 0), 40.0, 30.0, 35, 27, n_samples=samples, ray_length=LENGTH,
                       segments=segments)


def o_cam(oracle, cam):
    return oracle.camera64(tuple(cam.pos), tuple(cam.aim), cam.fov_w_deg, cam.fov_h_deg, cam.nx, cam.ny,
                           cam.n_samples, cam.ray_length, cam.march)


# nodes per axis, samples per ray: 9 planes between samples; about one a cell; thousands in one cell
@pytest.mark.parametrize("nodes,samples", [(72, 20), (72, 1), (72, 176), (24, 61), (2, 20000), (3, 4099)])
@pytest.mark.parametrize("layout", [0, 1, 2])
@pytest.mark.parametrize("segments", [1, 8])
def test_samples_per_cell(birp, oracle, nodes, samples, layout, segments):
    xs, ys, zs, v = field(nodes, nodes + samples)
    cube = birp.Cube(xs, ys, zs, v, layout=layout)
    cam = camera(birp, samples, segments)
    img = birp.render(cube, cam)
    ref = oracle.render64(oracle.Cube64(xs, ys, zs, v.astype(np.float64), 1), o_cam(oracle, cam), threads=THREADS)
    mx, rms, n = rel_err(img, ref)
    assert mx <= TOL, (mx, n)
    cube.close()


@pytest.mark.parametrize("layout", [0, 1, 2])
def test_infinity_in_a_cell_without_samples(birp, oracle, layout):
    """Rays cross cells next to infinite nodes, no sample lies within two
    cells of one: the image is that of the field without them."""
    xs, ys, zs, v = field(72, 5)
    cam = camera(birp, 20)
    fr = birp.camera_frame(cam)
    R = fr["rinv"]
    sx = (2 * (np.arange(cam.nx) + 0.5) / cam.nx - 1) * fr["tfx"] * fr["aspect"]
    sy = (1 - 2 * (np.arange(cam.ny) + 0.5) / cam.ny) * fr["tfy"]
    d = (sx[None, :, None] * R[:, 0] - R[:, 2]) + sy[:, None, None] * R[:, 1]
    d /= np.linalg.norm(d, axis=2, keepdims=True)
    t = (np.arange(cam.n_samples) + 0.5) * fr["dt"]
    p = np.array(cam.pos) + d[:, :, None, :] * t[:, None]
    taken = np.zeros(v.shape, bool)
    k = [np.searchsorted(a, p[..., i], "right") - 1 for i, a in enumerate((xs, ys, zs))]
    inside = np.all([(q >= 0) & (q < len(a) - 1) for q, a in zip(k, (xs, ys, zs))], axis=0)
    for x, y, z in zip(*(q[inside] for q in k)):
        taken[max(z - 2, 0):z + 4, max(y - 2, 0):y + 4, max(x - 2, 0):x + 4] = True
    # nodes that a ray passes between two samples: along the rays at other distances
    t2 = np.linspace(0.0, LENGTH, 4000)
    hit = np.zeros(v.shape, bool)
    q = np.array(cam.pos) + d[::3, ::3, None, :] * t2[:, None]
    k = [np.searchsorted(a, q[..., i], "right") - 1 for i, a in enumerate((xs, ys, zs))]
    inside = np.all([(q_ >= 0) & (q_ < len(a) - 1) for q_, a in zip(k, (xs, ys, zs))], axis=0)
    hit[k[2][inside], k[1][inside], k[0][inside]] = True
    spots = hit & ~taken
    assert spots.sum() > 20
    w = v.copy()
    w[spots] = np.inf
    cube = birp.Cube(xs, ys, zs, w, layout=layout)
    img = birp.render(cube, cam)
    ref = oracle.render64(oracle.Cube64(xs, ys, zs, v.astype(np.float64), 1), o_cam(oracle, cam), threads=THREADS)
    assert np.isfinite(img).all()
    mx, rms, n = rel_err(img, ref)
    assert mx <= TOL, (mx, n)
    cube.close()
