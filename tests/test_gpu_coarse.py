"""Trilinear requests whose samples lie several cells apart take a march that
skips the cells between them: images on both sides of the rule (3 cell faces
between two samples) and far beyond it against the FP64 oracle, each layout,
march mode and number of lanes per ray, alone, in a batch and without
allocations; and a narrow cube of many thin cells."""
import ctypes as C
import os

import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu

TOL = 1e-5
THREADS = os.cpu_count() or 4
N = 81
CUBES = {"uniform": [np.linspace(-9.0, 9.0, N), np.linspace(-8.0, 10.0, N - 4), np.linspace(-9.5, 9.0, N + 2)],
         "uneven": [np.sign(t) * np.abs(t) ** 1.3 for t in (np.linspace(-5.5, 5.5, N),) * 3],
         "thin": [np.linspace(-9.0, 9.0, 900), np.linspace(-8.0, 10.0, 6), np.linspace(-9.5, 9.0, 5)]}
POSES = ((-8.5, -1.0, 2.0), (-20.0, -3.0, 1.0), (4.0, 6.0, 8.0))


def requests(birp, march):
    # a face every 0.225 Re along an axis: 2 to 4 between samples at 44 Re / 65 to 130, 40 at 8 samples
    for pos in POSES:
        for samples, segments in ((300, 0), (130, 1), (96, 2), (80, 8), (65, 0), (30, 4), (8, 1), (8, 8), (1, 0)):
            yield birp.camera(pos, (10, 0, 0), 60.0, 50.0, 37, 29, n_samples=samples, ray_length=44.0, trilinear=True,
                              march=march, segments=segments)


@pytest.mark.parametrize("name", list(CUBES))
@pytest.mark.parametrize("layout", [0, 1, 2])
def test_against_the_oracle(birp, oracle, name, layout):
    import torch
    axes = CUBES[name]
    v = np.random.default_rng(6).uniform(1.0, 1.4, tuple(len(a) for a in axes[::-1])).astype(np.float32)
    if name == "thin":  # smooth along the thin cells: a sample's FP32 position is worth 1e-6 Re
        v = (1.2 + 0.2 * np.sin(axes[0])[None, None, :] * np.ones_like(v)).astype(np.float32)
    cube = birp.Cube(*axes, v, layout=layout)
    oc = oracle.Cube64(*axes, v.astype(np.float64), 1)
    cams = [cam for march in (birp.PREFIX, birp.CLIP) for cam in requests(birp, march)]
    refs = [oracle.render64(oc, oracle.camera64(tuple(c.pos), tuple(c.aim), c.fov_w_deg, c.fov_h_deg, c.nx, c.ny,
                                                c.n_samples, c.ray_length, c.march), threads=THREADS) for c in cams]
    items = [(cube, cam) for cam in cams]
    batch = birp.Batch(len(items), len(items) * 37 * 29)
    got = [batch.render(items), [birp.render(cube, cam) for cam in cams]]
    fn = birp.lib().birp_batch_render_noalloc
    fn.argtypes, fn.restype = [C.c_void_p, C.c_int, C.c_void_p, C.c_void_p], C.c_int
    dev = torch.zeros(16, 29, 37, device="cuda")
    torch.cuda.synchronize()
    birp.check(fn(birp.Batch._reqs(items[:16]), 16, (C.c_void_p * 16)(*[d.data_ptr() for d in dev]), None))
    torch.cuda.synchronize()
    got.append(list(dev.cpu().numpy()))
    for images in got:
        for img, ref, cam in zip(images, refs, cams):
            assert np.array_equal(img == 0, ref == 0), (cam.n_samples, cam.march)
            assert rel_err(img, ref)[0] <= TOL, (cam.n_samples, cam.march, rel_err(img, ref))
    batch.close()
    cube.close()
