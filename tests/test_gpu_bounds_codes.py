"""The bounds-checking build checks each kind of table access: a few renders in
a child process reach every code (birp_debug_bounds_codes) and none is out of
range."""
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_every_code_is_checked():
    from birp_cpp_gb300 import build
    env = dict(os.environ, BIRP_LIB=build.build_debug_bounds())
    r = subprocess.run([sys.executable, os.path.abspath(__file__)], env=env, cwd=ROOT, capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-2000:]
    assert r.stdout.split() == ["status", "0x0", "codes"] + [str(c) for c in range(1, 13)]


def main():
    sys.path.insert(0, ROOT)
    import birp_cpp_gb300 as B
    from birp_cpp_gb300 import synth
    B.init(0)
    B.debug_bounds(reset=True)
    node = np.arange(-8.0, 9.0)
    stretched = synth.stretched_axis(-20, 25, 41)
    rng = np.random.default_rng(1)
    for axes in ((node, node, node), (stretched, node, node)):
        for negatives in (False, True):
            v = rng.uniform(0.5, 2.0, tuple(len(a) for a in axes[::-1]))
            if negatives:
                v[rng.random(v.shape) < 0.02] *= -1
            for layout in (B.CUBE_RECORDS, B.CUBE_COMPACT, B.CUBE_PAIRS):
                cube = B.Cube(*axes, v.astype(np.float32), layout=layout)
                for tri in (True, False):
                    # along x, samples 1/4 apart from -7.25 on: many on planes; rays start on a plane and skim others
                    for pos, fov in (((-7.375, 0.25, 0.25), 0.5), ((-20.0, -3.0, 2.0), 60.0), ((-7.5, 0.0, 0.0), 2.0)):
                        cam = B.camera(pos, (5.0, 0, 0) if pos[0] == -7.5 else (10.0, 0, 0), fov, fov, 17, 17,
                                       n_samples=64, ray_length=16.0, trilinear=tri, march=B.CLIP)
                        B.render(cube, cam)
                cube.close()
    # uniform axes, nearest, one ray along x exactly: its samples lie on the nodes
    cube = B.Cube(node, node, node, np.ones((17, 17, 17), np.float32))
    B.render(cube, B.camera((-7.375, 0.0, 0.0), (5.0, 0, 0), 1.0, 1.0, 1, 1, n_samples=64, ray_length=16.0,
                            trilinear=False, march=B.CLIP))
    cube.close()
    B.render(B.Cmem(), B.camera((5.9, 6.7, 17.7), (7.8, 0, 0), 36.0, 36.0, 24, 24, n_samples=200))
    status, codes = B.debug_bounds(reset=False), B.debug_bounds_codes()
    print("status", hex(status), "codes", *[c for c in range(64) if codes >> c & 1])


if __name__ == "__main__":
    main()
