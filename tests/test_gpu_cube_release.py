"""Releasing cubes beside other work: a stream another thread is capturing goes
on being captured (birp_cube_destroy waits for no more than it has to), and the
memory of a cube whose render is still in flight, on a caller's stream or in a
submitted batch, goes to no other cube before that render is done."""
import ctypes as C
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPE = (96, 90, 84)  # 8 MB and more in every layout's largest array
AXES = [np.linspace(-9.0, 9.0, n) for n in SHAPE]


def cube(birp, value, layout=0):
    return birp.Cube(*AXES, np.full(SHAPE[::-1], value, np.float32), layout=layout)


def view(birp, w=40, h=30, n=150, **kw):
    return birp.camera((1.0, -5.0, 4.0), (10, 0, 0), 40.0, 30.0, w, h, n_samples=n, ray_length=20.0, **kw)


@pytest.mark.parametrize("mode", [1, 2], ids=["thread_local", "relaxed"])
def test_capture_in_another_thread(birp, mode):
    import torch
    rt = C.CDLL("libcudart.so.13")
    cam, keep, victim = view(birp), cube(birp, 1.0), cube(birp, 2.0)
    want = birp.render(keep, cam)
    birp.render(victim, cam)
    out = torch.zeros(30, 40, device="cuda")
    torch.cuda.synchronize()
    stream, graph, run = C.c_void_p(), C.c_void_p(), C.c_void_p()
    assert rt.cudaStreamCreateWithFlags(C.byref(stream), 1) == 0
    got, go, done = {}, threading.Event(), threading.Event()

    def record():
        def render():
            return birp.lib().birp_render_device(keep.h, None, C.byref(cam), C.c_void_p(out.data_ptr()), stream)
        got["begin"] = rt.cudaStreamBeginCapture(stream, mode)
        got["first"] = render()
        go.set()
        done.wait(60)
        got["second"] = render()
        got["end"] = rt.cudaStreamEndCapture(stream, C.byref(graph))

    t = threading.Thread(target=record)
    t.start()
    assert go.wait(60)
    victim.close()
    done.set()
    t.join()
    assert got == {"begin": 0, "first": 0, "second": 0, "end": 0}, got
    assert rt.cudaGraphInstantiate(C.byref(run), graph, C.c_ulonglong(0)) == 0
    assert rt.cudaGraphLaunch(run, stream) == 0 and rt.cudaStreamSynchronize(stream) == 0
    assert np.array_equal(out.cpu().numpy(), want)
    rt.cudaGraphExecDestroy(run)
    rt.cudaGraphDestroy(graph)
    rt.cudaStreamDestroy(stream)
    keep.close()


def test_batches_made_while_cubes_are_released(birp):
    """birp_batch_create captures its graph; cubes come and go in another thread meanwhile."""
    cam, keep = view(birp), cube(birp, 1.0)
    want = birp.render(keep, view(birp, segments=1))
    bad, stop = [], threading.Event()

    def batches():
        while not stop.is_set():
            try:
                b = birp.Batch(2, 1 << 12)
                if not np.allclose(b.render([(keep, cam)])[0], want, rtol=1e-5):
                    bad.append("image")
                b.close()
            except Exception as e:  # noqa: BLE001
                bad.append(repr(e))

    t = threading.Thread(target=batches)
    t.start()
    for _ in range(60):
        c = cube(birp, 3.0)
        birp.render(c, cam)
        c.close()
    stop.set()
    t.join()
    assert not bad, bad[:3]
    keep.close()


@pytest.mark.parametrize("layout", [0, 1, 2])
@pytest.mark.parametrize("route", ["stream", "batch", "noalloc"])
def test_release_with_a_render_in_flight(birp, layout, route):
    import torch
    cam = view(birp, 512, 384, 60000, segments=1)  # a few ms
    a = cube(birp, 1.0, layout)
    stream = torch.cuda.Stream()
    out = torch.zeros(384, 512, device="cuda")
    batch = birp.Batch(1, 512 * 384)
    want = batch.render([(a, cam)])[0]
    torch.cuda.synchronize()
    for _ in range(3):
        out.zero_()
        torch.cuda.synchronize()
        s = C.c_void_p(stream.cuda_stream)
        if route == "stream":
            birp.check(birp.lib().birp_render_device(a.h, None, C.byref(cam), C.c_void_p(out.data_ptr()), s))
        elif route == "batch":
            batch.submit([(a, cam)])
        else:
            fn = birp.lib().birp_batch_render_noalloc
            fn.argtypes, fn.restype = [C.c_void_p, C.c_int, C.c_void_p, C.c_void_p], C.c_int
            birp.check(fn(birp.Batch._reqs([(a, cam)]), 1, (C.c_void_p * 1)(out.data_ptr()), s))
        a.close()
        b = cube(birp, 7.0, layout)  # would take a's memory and overwrite it under the render
        if route == "batch":
            batch.wait()
            img = np.ctypeslib.as_array(birp.lib().birp_batch_image(batch.h, 0), (384, 512))
        else:
            stream.synchronize()
            img = out.cpu().numpy()
        assert np.allclose(img, want, rtol=1e-6, atol=0)
        b.close()
        a = cube(birp, 1.0, layout)
    a.close()
    batch.close()
