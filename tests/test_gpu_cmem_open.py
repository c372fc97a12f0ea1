"""CMEM samples that FP32 leaves open, of different kinds in one warp: eight
lanes work on a sample, so a warp's four groups hold points on the planes the
reference treats apart (x = 0: theta = 0; y = 0: phi = 0) beside ordinary ones.
Every point within a few FP32 steps of the magnetopause's or the bow shock's
outer edge; each against the FP64 oracle (which side of the edge, and the value
there within the path's 1e-5) and, bit for bit, against a call with that point
alone."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 1e-5
MODELS = [dict(), dict(dipole=0.3), dict(b=(0, 0, -20), density=30.0, bs=9.0, alpha=1.5, beta=0.4)]


def edge_points(om, kinds, seed):
    """A point per entry of kinds (0: x = 0, 1: y = 0, 2: neither) at an outer edge of a surface's ramp: where the
    oracle's value jumps along a ray from the Earth (the first such place for even entries, the last for odd ones), by
    bisection in FP64."""
    rng = np.random.default_rng(seed)
    r = np.linspace(0.5, 60.0, 20000)
    out = np.empty((len(kinds), 3), np.float32)
    for i, kind in enumerate(kinds):
        jumps = []
        while not len(jumps):
            u = rng.normal(size=3)
            if kind < 2:
                u[kind] = 0.0
            u /= np.linalg.norm(u)
            v = om.sample(u * r[:, None])
            with np.errstate(all="ignore"):
                jumps = np.flatnonzero((v[:-1] > 0) & (np.abs(np.log(v[1:] / v[:-1])) > 0.2) & (v[:-1] > 1e-9))
            jumps = [k for k in jumps if v[max(k - 8, 0)] > 0]  # past the ramp's first steps from 0
        k = jumps[0 if i % 2 == 0 else -1]
        lo, hi, mid, up = r[k], r[k + 1], 0.5 * (v[k] + v[k + 1]), v[k + 1] > v[k]
        for _ in range(40):
            m = 0.5 * (lo + hi)
            if (om.sample(u * m)[0] > mid) == up:
                hi = m
            else:
                lo = m
        out[i] = (u * (hi * (1.0 + 1e-6 * rng.uniform(-1, 1)))).astype(np.float32)
    return out


@pytest.mark.parametrize("kw", MODELS, ids=str)
def test_groups_of_a_warp(birp, oracle, kw):
    om = oracle.Cmem64(oracle.cmem_args(**kw))
    rng = np.random.default_rng(5)
    kinds = np.concatenate([np.arange(64) % 2 * 2, np.arange(64) % 3, rng.integers(0, 3, 131)])
    p = edge_points(om, kinds, 17)
    model = birp.Cmem(birp.cmem_params(**kw))
    got = model.sample(p)
    ref = om.sample(p.astype(np.float64))
    assert np.array_equal(got == 0, ref == 0)
    m = ref != 0
    assert m.all()
    assert np.max(np.abs(got[m] - ref[m]) / ref[m]) <= TOL
    alone = np.array([model.sample(q[None])[0] for q in p], np.float32)
    assert np.array_equal(got, alone)
    model.close()


@pytest.mark.parametrize("count", [1, 4, 5, 12, 13, 31, 32])
def test_open_samples_in_a_warp(birp, oracle, count):
    """Up to 12 open samples of a warp share its lanes, more take a lane each: the same values."""
    om = oracle.Cmem64()
    rng = np.random.default_rng(count)
    p = np.full((32, 3), 3.0, np.float32)  # inside the magnetopause: decided without them
    p[:, 0] = np.linspace(-3, 3, 32)
    at = rng.permutation(32)[:count]
    p[at] = edge_points(om, rng.integers(0, 3, count), count)
    model = birp.Cmem()
    got = model.sample(p)
    assert np.array_equal(got, np.array([model.sample(q[None])[0] for q in p], np.float32))
    ref = om.sample(p.astype(np.float64))
    assert np.array_equal(got == 0, ref == 0)
    assert np.max(np.abs(got - ref)[ref != 0] / ref[ref != 0]) <= TOL
    model.close()


def test_radii_that_are_not_numbers(birp, oracle):
    """A model whose radii are NaN leaves every sample open: the oracle's outer values, in calls and in renders."""
    kw = dict(density=-5.0)
    om, model = oracle.Cmem64(oracle.cmem_args(**kw)), birp.Cmem(birp.cmem_params(**kw))
    p = np.random.default_rng(2).uniform(-20, 20, (3000, 3)).astype(np.float32)
    with np.errstate(all="ignore"):
        ref = om.sample(p.astype(np.float64))
        assert np.max(np.abs(model.sample(p) - ref) / ref) <= TOL
        cam = birp.camera((5.9, 6.7, 17.7), (9, 0, 0), 40.0, 30.0, 19, 13, n_samples=120)
        img = birp.render(model, cam)
        want = oracle.render64(om, oracle.camera64(tuple(cam.pos), tuple(cam.aim), 40.0, 30.0, 19, 13, 120), threads=4)
    assert np.max(np.abs(img - want) / want) <= TOL
    model.close()
