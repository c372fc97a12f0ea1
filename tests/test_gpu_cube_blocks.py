"""Device memory that destroyed cubes leave for the next: a cube built in it
renders as one built in new memory, also while other threads build, render on
their own streams and release, and no more than the stated 1 GiB stays."""
import ctypes
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def field(shape, seed):
    return np.random.default_rng(seed).uniform(0.5, 2.0, shape[::-1]).astype(np.float32)


def axes(shape):
    return [np.linspace(-9.0, 9.0, n) for n in shape]


# sizes on both sides of the smallest kept block (8 MB), of an eighth, of the bound (1 GiB)
SHAPES = [(40, 40, 40), (66, 64, 63), (90, 80, 70), (92, 80, 70), (130, 120, 110), (128, 120, 110), (340, 330, 310)]


def view(birp, k):
    return birp.camera((1.0 + 0.1 * k, -5.0, 4.0), (10, 0, 0), 40.0, 30.0, 40, 30, n_samples=150, ray_length=20.0)


@pytest.mark.parametrize("layout", [0, 1, 2])
def test_reused_memory(birp, layout):
    import torch
    want = {}
    free0 = None
    for turn in range(3):
        for k, shape in enumerate(SHAPES if turn % 2 == 0 else SHAPES[::-1]):
            seed = int(np.prod(shape)) % 1000
            cube = birp.Cube(*axes(shape), field(shape, seed), layout=layout)
            img = birp.render(cube, view(birp, seed % 7))
            cube.close()
            assert np.array_equal(img, want.setdefault(shape, img)), (turn, shape)
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        free0 = free if free0 is None else free0
        assert abs(free - free0) <= (1 << 30) + (64 << 20)


def test_threads(birp):
    import torch
    shapes = SHAPES[1:6]
    want = {}
    for k, shape in enumerate(shapes):
        cube = birp.Cube(*axes(shape), field(shape, k))
        want[shape] = birp.render(cube, view(birp, k))
        cube.close()
    bad = []

    def work(t):
        try:
            stream = torch.cuda.Stream()
            out = torch.empty(30, 40, device="cuda")
            for turn in range(12):
                k = (t + turn) % len(shapes)
                cube = birp.Cube(*axes(shapes[k]), field(shapes[k], k))
                birp.check(birp.lib().birp_render_device(cube.h, None, ctypes.byref(view(birp, k)),
                                                         ctypes.c_void_p(out.data_ptr()),
                                                         ctypes.c_void_p(stream.cuda_stream)))
                cube.close()  # waits for the render before its memory can go to another cube
                stream.synchronize()
                if not np.array_equal(out.cpu().numpy(), want[shapes[k]]):
                    bad.append((t, turn))
        except Exception as e:  # noqa: BLE001
            bad.append(repr(e))

    threads = [threading.Thread(target=work, args=(t,)) for t in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad, bad
