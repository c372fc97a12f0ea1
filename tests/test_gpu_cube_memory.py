"""Device memory kept from destroyed cubes: no more than the stated 1 GiB
whatever sizes come and go, all of it back at birp_trim, and cubes in kept
blocks (an eighth larger than asked for at most, with another cube's values in
them) render as those in new memory."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# record arrays of 132 to 420 MB, each more than an eighth from the next: 1.6 GB in all
SIZES = [160, 175, 190, 205, 220, 235]
SLACK = 48 << 20  # of the driver's own granularity


def build(birp, n, layout):
    axes = [np.linspace(-9.0, 9.0, n), np.linspace(-8.0, 9.0, n), np.linspace(-9.0, 7.0, n)]
    v = np.random.default_rng(n).uniform(0.5, 2.0, (n, n, n)).astype(np.float32)
    return birp.Cube(*axes, v, layout=layout)


def test_bound_and_trim(birp):
    import torch

    def free():
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]

    cam = birp.camera((1.0, -5.0, 4.0), (10, 0, 0), 40.0, 30.0, 40, 30, n_samples=150, ray_length=20.0)
    c = build(birp, 40, 0)
    birp.render(c, cam)
    c.close()
    birp.trim()
    free0, want, most = free(), {}, 0
    for n in SIZES:  # in new memory
        for layout in (0, 2):
            c = build(birp, n, layout)
            want[n, layout] = birp.render(c, cam)
            c.close()
            birp.trim()
            assert abs(free() - free0) <= SLACK, n
    for turn in range(2):
        for n in SIZES + SIZES[::-1]:
            for layout in (0, 2):
                c = build(birp, n - turn, layout) if turn else build(birp, n, layout)
                img = birp.render(c, cam)
                c.close()
                assert turn or np.array_equal(img, want[n, layout]), (n, layout)
                most = max(most, free0 - free())
                assert free0 - free() <= (1 << 30) + SLACK, (n, layout)
    assert most > 512 << 20  # the blocks were kept
    birp.trim()
    assert abs(free() - free0) <= SLACK
    for n in SIZES[::-1]:
        c = build(birp, n, 0)
        assert np.array_equal(birp.render(c, cam), want[n, 0])
        c.close()
    birp.trim()
