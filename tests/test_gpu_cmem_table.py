"""CMEM samples decided by the model's table of surface bounds, by the radii,
and in FP64: every way in against the FP64 oracle, over models whose surfaces
differ (dipole tilt, wind and field, flaring per axis, exponent, a field large
enough that the sheath needs its angle), points in every direction and shell,
on the planes and axes the reference treats apart, far out and not finite; and
renders with more open samples than a thread keeps."""
import os

import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu

TOL = 1e-5
THREADS = os.cpu_count() or 4
MODELS = [dict(), dict(dipole=0.3), dict(dipole=-0.4, v=(700, 10, 5)), dict(b=(50, 0, 40), v=(300, 0, 0)),
          dict(ay_bs=0.45, az_bs=0.8), dict(p0=0.9, p1=2), dict(density=1.0, v=(250, 0, 0)), dict(b=(20000, 0, 5)),
          dict(b=(0, 0, -20), density=30.0, bs=9.0, alpha=1.5, beta=0.4)]


def points(n, seed):
    rng = np.random.default_rng(seed)
    d = rng.normal(size=(n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    p = d * np.exp(rng.uniform(np.log(0.05), np.log(80.0), n))[:, None]
    k = n // 20
    p[:k, 0] = 0.0           # x = 0: theta = 0
    p[k:2 * k, 1] = 0.0      # y = 0: phi = 0
    p[2 * k:3 * k, 2] = 0.0
    p[3 * k:4 * k, 1:] *= 1e-4  # next to the Earth-Sun line
    p[4 * k:4 * k + 4] = [(12.0, 0, 0), (-30.0, 0, 0), (0, 11.0, 0), (0, 0, 9.0)]
    return p.astype(np.float32)


@pytest.mark.parametrize("kw", MODELS, ids=str)
def test_samples(birp, oracle, kw):
    p = points(120000, len(str(kw)))
    got = birp.Cmem(birp.cmem_params(**kw)).sample(p).astype(np.float64)
    om = oracle.Cmem64(oracle.cmem_args(**kw))
    p64 = p.astype(np.float64)
    with np.errstate(all="ignore"):
        ref, lo, hi = (om.sample(p64 * s) for s in (1.0, 1.0 - 3e-5, 1.0 + 3e-5))
    fine = np.isfinite(ref)
    assert np.array_equal(fine, np.isfinite(got))
    assert np.array_equal(got[fine] == 0, ref[fine] == 0)
    # values away from the surfaces' ramps and steps (there they move with the surface: covered by the renders)
    calm = fine & (ref != 0) & (np.abs(hi - lo) <= 1e-3 * np.abs(ref))
    assert calm.sum() > 0.9 * (ref != 0).sum() > 0.1 * len(p)
    err = np.abs(got[calm] - ref[calm]) / np.abs(ref[calm])
    assert err.max() <= TOL, (err.max(), p[calm][err.argmax()])


def test_points_out_of_range(birp):
    """Far points take the outer profile, points that are not finite neither
    fault nor hang nor disturb the others, whatever the call's length."""
    m = birp.Cmem()
    p = points(1000, 3)
    want = m.sample(p)
    for n in (1, 31, 33, 257, 1000):
        assert np.array_equal(m.sample(p[:n]), want[:n])
    q = p.copy()
    for k, bad in enumerate((np.nan, np.inf, -np.inf, 3e38, 1e15, -1e16)):
        for axis in range(3):
            q[100 + 3 * k + axis, axis] = bad
    got = m.sample(q)
    keep = np.ones(len(p), bool)
    keep[100:118] = False
    assert np.array_equal(got[keep], want[keep])


@pytest.mark.parametrize("kw", [MODELS[0], MODELS[2], MODELS[4], MODELS[7]], ids=str)
@pytest.mark.parametrize("segments,samples", [(1, 150000), (8, 150000), (2, 997), (4, 1)])
def test_renders(birp, oracle, kw, segments, samples):
    """150000 samples along 44 Re: up to dozens of open samples a lane."""
    m = birp.Cmem(birp.cmem_params(**kw))
    om = oracle.Cmem64(oracle.cmem_args(**kw))
    for pos in ((3.49, 0.0746, 0.244), (-2, -12, 16)):
        cam = birp.camera(pos, (9, 0, 0), 40.0, 30.0, 9, 7, n_samples=samples, segments=segments)
        img = birp.render(m, cam)
        ref = oracle.render64(om, oracle.camera64(tuple(cam.pos), tuple(cam.aim), cam.fov_w_deg, cam.fov_h_deg, cam.nx,
                                                  cam.ny, cam.n_samples, cam.ray_length, cam.march), threads=THREADS)
        mx, rms, n = rel_err(img, ref)
        assert mx <= TOL, (pos, mx)
    m.close()
